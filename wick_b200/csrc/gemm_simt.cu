// C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores with float32 multiply-adds
// (never a reduced-precision tensor mode).  This is the matrix product of the
// 32-bit path and the plain twin of the tensor-core kernels of the bfloat16
// path.
//
// GATED: W holds 2N rows, gate rows first and up rows after them; the output is
// silu(A*gate^T) * (A*up^T)  (wick src/model.rs:493-501, src/kernels.rs:374-378).
//
// float32 (K a multiple of four, rows that start at multiples of 16 bytes): K is cut into at most
// eight slices of slice_len(K) numbers; an output is the sum, in slice order, of the slices' dot
// products, each accumulated along k in index order.  That order depends on K alone, and all forms
// below follow it, so a row's result depends neither on the other rows nor on M:
//   * gemm_f32_few_kernel, up to 32 rows of A: the weights stream through shared memory, once per 16 rows;
//   * gemm_f32_tile_kernel, more rows: tiles of 128 x 128, 64 x 128 or 64 x 64 outputs;
//   * gemm_nt_kernel, some sizes of up to 256 inputs, see few_inputs_form.
// Everything else goes through gemm_nt_kernel as well, one dot product along K in index order.
#include <type_traits>

#include "common.cuh"

namespace wick {

inline __host__ __device__ int slice_len(int K) { return (K + 1023) / 1024 * 128; }

__device__ __forceinline__ void cp16(void* dst, const void* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 16 : 0;                // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A block makes RB = 8 RPL outputs for MB rows of A.  Warp w takes slice w of K: its RB rows of W and its MB rows of A
// come in stages of KST numbers through a ring of its own (cp.async, the first stages of W before the kernel before this
// one has finished).  Lane l holds rows l % 8 (and l % 8 + 8) of W and the rows l / 8, l / 8 + 4, ... of A, and walks along
// k four numbers at a time; 16-byte pieces are XOR-swizzled by the row so that eight rows' pieces come from shared memory at
// once.  The slices' sums meet in shared memory and are added in slice order.
// What bounds it is the stream of weights.  Four rows of A, times us (GB/s): 2,048 x 2,048 weights 174 -> 5.8 (2,890), gated
// 2 x 5,120 x 2,048 239 -> 20.3 (4,140), 32,768 x 2,048 345 -> 54 (4,940); before, 64 x 64 outputs a block and one load after the other.
constexpr int FEW_WARPS = 8, FEW_STAGES = 2;

template <int MB, int RPL, bool GATED>
struct Few {
    static constexpr int RB = 8 * RPL, KST = RPL == 1 ? 128 : 64, CH = KST / 4;      // CH: 16-byte pieces of a stage's row
    static constexpr int AM = (MB + 3) / 4;                                          // rows of A a lane holds
    static constexpr int STAGE = (RB + MB) * KST;                                    // floats
    static constexpr size_t SMEM = sizeof(float) * (size_t)FEW_WARPS * FEW_STAGES * STAGE;
    static constexpr int NB = GATED ? RB / 2 : RB;                                   // outputs of a block
};

template <int MB, int RPL, bool GATED>
__global__ void __launch_bounds__(32 * FEW_WARPS, 2)
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, int w_static) {
    typedef Few<MB, RPL, GATED> F;
    extern __shared__ __align__(16) float few_smem[];
    __shared__ float sums[2][FEW_WARPS][F::RB][MB];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.x * MB;
    const int len = slice_len(K), k_begin = warp * len, k_end = min(K, k_begin + len);
    const int n_st = k_end > k_begin ? (k_end - k_begin + F::KST - 1) / F::KST : 0;
    // the block's groups of outputs: blockIdx.y, blockIdx.y + gridDim.y, ...; the warp's ring runs on from one to the next
    const int n_groups = ((N + F::NB - 1) / F::NB - (int)blockIdx.y + (int)gridDim.y - 1) / (int)gridDim.y;
    float* ring = few_smem + (size_t)warp * FEW_STAGES * F::STAGE;
    int wg = 0, wi = 0, ag = 0, ai = 0;                  // group and stage that are fetched next, of W and of A
    // row r of a group's rows of W (gated: the first half gate rows, the second half their up rows)
    auto load_w = [&](int slot) {
        if (wg >= n_groups) return;
        float* dst = ring + slot * F::STAGE;
        const int k0 = k_begin + wi * F::KST, n0 = ((int)blockIdx.y + wg * (int)gridDim.y) * F::NB;
#pragma unroll
        for (int x = lane; x < F::RB * F::CH; x += 32) {
            const int r = x / F::CH, c = x % F::CH, k = k0 + 4 * c, n = min(n0 + (GATED ? r % F::NB : r), N - 1);
            const float* row = W + (int64_t)(GATED && r >= F::NB ? N + n : n) * K;
            cp16(dst + r * F::KST + (c ^ (r & 7)) * 4, row + min(k, K - 4), k < k_end);
        }
        if (++wi == n_st) wi = 0, ++wg;
    };
    auto load_a = [&](int slot) {
        if (ag >= n_groups) return;
        float* dst = ring + slot * F::STAGE + F::RB * F::KST;
        const int k0 = k_begin + ai * F::KST;
#pragma unroll
        for (int x = lane; x < MB * F::CH; x += 32) {
            const int m = x / F::CH, c = x % F::CH, k = k0 + 4 * c;
            cp16(dst + m * F::KST + (c ^ (m & 7)) * 4, A + (int64_t)min(m0 + m, M - 1) * K + min(k, K - 4), k < k_end);
        }
        if (++ai == n_st) ai = 0, ++ag;
    };
    if (!w_static) pdl_wait();
    if (n_st > 0) {
#pragma unroll
        for (int i = 0; i < FEW_STAGES; ++i) load_w(i);
    }
    if (w_static) pdl_wait();
#pragma unroll
    for (int i = 0; i < FEW_STAGES; ++i) {               // (a group of copies per stage, empty beyond the last)
        if (n_st > 0) load_a(i);
        cp_commit();
    }
    const int row = lane & 7, mq = lane >> 3;
    const int used = (K + len - 1) / len;                // slices that hold numbers
    int slot = 0;
    for (int g = 0; g < n_groups; ++g) {
        float acc[RPL][F::AM];
#pragma unroll
        for (int r = 0; r < RPL; ++r)
#pragma unroll
            for (int a = 0; a < F::AM; ++a) acc[r][a] = 0.f;
        for (int i = 0; i < n_st; ++i) {
            cp_wait<FEW_STAGES - 1>();
            __syncwarp();
            const float* ws = ring + slot * F::STAGE;
            const float* as = ws + F::RB * F::KST;
#pragma unroll 8
            for (int c = 0; c < F::CH; ++c) {
                float4 w[RPL], a[F::AM];
#pragma unroll
                for (int r = 0; r < RPL; ++r) w[r] = *reinterpret_cast<const float4*>(ws + (row + 8 * r) * F::KST + (c ^ row) * 4);
#pragma unroll
                for (int j = 0; j < F::AM; ++j) {
                    const int m = MB >= 4 ? mq + 4 * j : mq % MB;
                    a[j] = *reinterpret_cast<const float4*>(as + m * F::KST + (c ^ (m & 7)) * 4);
                }
#pragma unroll
                for (int r = 0; r < RPL; ++r)
#pragma unroll
                    for (int j = 0; j < F::AM; ++j) {
                        acc[r][j] = fmaf(a[j].x, w[r].x, acc[r][j]);
                        acc[r][j] = fmaf(a[j].y, w[r].y, acc[r][j]);
                        acc[r][j] = fmaf(a[j].z, w[r].z, acc[r][j]);
                        acc[r][j] = fmaf(a[j].w, w[r].w, acc[r][j]);
                    }
            }
            __syncwarp();                                // every lane is done with the stage
            load_w(slot);
            load_a(slot);
            cp_commit();
            slot = slot + 1 == FEW_STAGES ? 0 : slot + 1;
        }
        float (*out)[F::RB][MB] = sums[g & 1];           // (a warp writes one of the two again only after everyone has read the other)
#pragma unroll
        for (int r = 0; r < RPL; ++r)
#pragma unroll
            for (int j = 0; j < F::AM; ++j)
                if (MB >= 4 || mq < MB) out[warp][row + 8 * r][MB >= 4 ? mq + 4 * j : mq] = acc[r][j];
        __syncthreads();
        const int n0 = ((int)blockIdx.y + g * (int)gridDim.y) * F::NB;
        for (int x = tid; x < F::NB * MB; x += 32 * FEW_WARPS) {
            const int r = x % F::NB, m = x / F::NB;
            if (m0 + m >= M || n0 + r >= N) continue;
            float v = out[0][r][m], u = GATED ? out[0][F::NB + r][m] : 0.f;
            for (int s = 1; s < used; ++s) {
                v += out[s][r][m];
                if (GATED) u += out[s][F::NB + r][m];
            }
            if (GATED) v = v / (1.0f + expf(-v)) * u;
            C[(int64_t)(m0 + m) * N + n0 + r] = v;
        }
    }
}

// A block makes BM x BN outputs, a thread 8 x TN: steps of 16 numbers of K through two buffers in shared memory, both
// operands k-major there, the next step's loads in flight during this one's arithmetic.  GATED: the tile's columns are
// BN / 2 gate rows, then their up rows, and a thread holds both of each of its outputs.  Bound by the rate of
// float32 multiply-adds.  SLICED: for products with few of the large tiles (300 x 2,048 outputs are 48 of 128 x 128): the blocks of
// a cluster take a slice of K each, and the slices' tiles meet over distributed shared memory, a share of the rows in each block.
// 300 rows of A, us (TFLOP/s): 2,048 x 2,048 223 -> 77 (33), gated 2 x 5,120 x 2,048 476 -> 317 (40); 1,024 rows x 32,768 x 2,048
// in tiles of 128 x 128 5,290 -> 2,950 (47).
constexpr int TILE_BK = 16;

template <int BM, int BN, int TN, bool GATED, bool SLICED, bool W_STATIC>
__global__ void __launch_bounds__((BM / 8) * (BN / TN))
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K) {
    constexpr int THREADS = (BM / 8) * (BN / TN), TX = BN / TN, NB = GATED ? BN / 2 : BN;
    constexpr int LA = BM * 4 / THREADS, LB = BN * 4 / THREADS;          // 16-byte pieces a thread brings per step
    static_assert(!GATED || TN == 8, "a gated thread holds four gate and four up columns");
    constexpr int A_STEP = TILE_BK * (BM + 4), B_STEP = TILE_BK * (BN + 4), OPERANDS = 2 * (A_STEP + B_STEP);
    __shared__ __align__(16) float tile_smem[SLICED && BM * BN > OPERANDS ? BM * BN : OPERANDS];
    float (*As)[TILE_BK][BM + 4] = reinterpret_cast<float (*)[TILE_BK][BM + 4]>(tile_smem);
    float (*Bs)[TILE_BK][BN + 4] = reinterpret_cast<float (*)[TILE_BK][BN + 4]>(tile_smem + 2 * A_STEP);
    pdl_trigger();
    pdl_wait();
    A = fresh(A);
    if (!W_STATIC) W = fresh(W);                         // (300 rows, gated 2 x 2,048 x 512: 47.6 us with it, 43.6 without)
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * NB;
    const float* arow[LA];
    const float* brow[LB];
#pragma unroll
    for (int i = 0; i < LA; ++i) arow[i] = A + (int64_t)min(m0 + (tid + i * THREADS) / 4, M - 1) * K;
#pragma unroll
    for (int i = 0; i < LB; ++i) {
        const int r = (tid + i * THREADS) / 4, n = min(n0 + (GATED ? r % NB : r), N - 1);
        brow[i] = W + (int64_t)(GATED && r >= NB ? N + n : n) * K;
    }
    const int kc = (tid & 3) * 4;
    float4 ra[LA], rb[LB];
    auto fetch = [&](int k0) {
        const int k = k0 + kc;
#pragma unroll
        for (int i = 0; i < LA; ++i) ra[i] = k < K ? *reinterpret_cast<const float4*>(arow[i] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < LB; ++i) rb[i] = k < K ? *reinterpret_cast<const float4*>(brow[i] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int r = (tid + i * THREADS) / 4;
            As[buf][kc][r] = ra[i].x; As[buf][kc + 1][r] = ra[i].y; As[buf][kc + 2][r] = ra[i].z; As[buf][kc + 3][r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int r = (tid + i * THREADS) / 4;
            Bs[buf][kc][r] = rb[i].x; Bs[buf][kc + 1][r] = rb[i].y; Bs[buf][kc + 2][r] = rb[i].z; Bs[buf][kc + 3][r] = rb[i].w;
        }
    };
    float acc[8][TN], total[SLICED ? 1 : 8][TN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    const int len = slice_len(K);
    const int s_begin = SLICED ? (int)blockIdx.z * (len / TILE_BK) : 0;
    const int s_end = (min(K, SLICED ? ((int)blockIdx.z + 1) * len : K) + TILE_BK - 1) / TILE_BK;
    int until = len;                                     // where the slice at hand ends
    fetch(s_begin * TILE_BK);
    put(s_begin & 1);
    __syncthreads();
    for (int s = s_begin; s < s_end; ++s) {
        const int buf = s & 1;
        if (s + 1 < s_end) fetch((s + 1) * TILE_BK);
#pragma unroll
        for (int kk = 0; kk < TILE_BK; ++kk) {
            float a[8], b[TN];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8]);
            *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8 + 4]);
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
            if (TN == 8) *reinterpret_cast<float4*>(b + TN - 4) = *reinterpret_cast<const float4*>(&Bs[buf][kk][BN / 2 + tx * 4]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (!SLICED && ((s + 1) * TILE_BK == until || s + 1 == s_end)) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    total[SLICED ? 0 : i][j] = until == len ? acc[i][j] : total[SLICED ? 0 : i][j] + acc[i][j];
                    acc[i][j] = 0.f;
                }
            until += len;
        }
        if (s + 1 < s_end) put(buf ^ 1);
        __syncthreads();
    }
    if constexpr (SLICED) {
        // the block's sums into its shared memory (row by row), then rows of everybody's, added in slice order
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            *reinterpret_cast<float4*>(tile_smem + (ty * 8 + i) * BN + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            if (TN == 8) *reinterpret_cast<float4*>(tile_smem + (ty * 8 + i) * BN + BN / 2 + tx * 4) =
                make_float4(acc[i][TN - 4], acc[i][TN - 3], acc[i][TN - 2], acc[i][TN - 1]);
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int slices = (int)gridDim.z;
        const uint32_t here = (uint32_t)__cvta_generic_to_shared(tile_smem);
        auto sum4 = [&](int at) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int z = 0; z < slices; ++z) {
                uint32_t there;
                float4 d;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here + 4u * (uint32_t)at), "r"(z));
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w) : "r"(there) : "memory");
                v = z == 0 ? d : make_float4(v.x + d.x, v.y + d.y, v.z + d.z, v.w + d.w);
            }
            return v;
        };
        for (int x = (int)blockIdx.z * THREADS + tid; x < BM * (NB / 4); x += slices * THREADS) {
            const int r = x / (NB / 4), c = x % (NB / 4) * 4;
            if (m0 + r >= M) continue;
            const float4 v4 = sum4(r * BN + c), u4 = GATED ? sum4(r * BN + NB + c) : v4;
            const float v[4] = {v4.x, v4.y, v4.z, v4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n0 + c + j < N) C[(int64_t)(m0 + r) * N + n0 + c + j] = GATED ? v[j] / (1.0f + expf(-v[j])) * u[j] : v[j];
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // (nobody's shared memory goes while it is read)
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + ty * 8 + i;
        if (m >= M) continue;
        float* c = C + (int64_t)m * N + n0;
#pragma unroll
        for (int j = 0; j < (GATED ? 4 : TN); ++j) {
            const int n = (j < 4 ? 0 : BN / 2) + tx * 4 + (j & 3);
            if (n0 + n >= N) continue;
            float v = total[SLICED ? 0 : i][j];
            if (GATED) v = v / (1.0f + expf(-v)) * total[SLICED ? 0 : i][TN - 4 + j];
            c[n] = v;
        }
    }
}

// Up to this many rows of A the weights are streamed once per 16 rows.  Beyond, tiles are better on wide matrices (64 rows, gated
// 2 x 5,120 x 2,048: 131 us streamed, 78 as tiles) and little worse on narrow ones (2,048 x 2,048: 29 and 39).
constexpr int FEW_MAX = 32;

template <int MB, int RPL, bool GATED>
int gemm_f32_few(const float* A, const float* W, float* C, int M, int N, int K, int w_static, cudaStream_t s) {
    typedef Few<MB, RPL, GATED> F;
    const int rows = ceil_div(N, F::NB);
    static bool raised = false;
    if (!raised) {
        WICK_CUDA(cudaFuncSetAttribute(gemm_f32_few_kernel<MB, RPL, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::SMEM));
        raised = true;
    }
    const int chunks = ceil_div(M, MB), resident = sm_count() * (F::SMEM <= 104 * 1024 ? 2 : 1);
    WICK_CUDA(launch(gemm_f32_few_kernel<MB, RPL, GATED>, dim3(chunks, max(1, min(rows, resident / chunks))), dim3(32 * FEW_WARPS), F::SMEM, s, A, W, C, M, N, K, w_static));
    return check_launch("gemm_f32_few");
}

template <int BM, int BN, int TN, bool GATED, bool SLICED>
int gemm_f32_tiles(const float* A, const float* W, float* C, int M, int N, int K, int w_static, cudaStream_t s) {
    const int slices = SLICED ? ceil_div(K, slice_len(K)) : 1;                // at most eight: a cluster
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(N, GATED ? BN / 2 : BN), ceil_div(M, BM), slices);
    cfg.blockDim = dim3((BM / 8) * (BN / TN));
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = slices;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    if (w_static) WICK_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<BM, BN, TN, GATED, SLICED, true>, A, W, C, M, N, K));
    else WICK_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<BM, BN, TN, GATED, SLICED, false>, A, W, C, M, N, K));
    return check_launch("gemm_f32_tile");
}

// Few inputs (up to 256, one or two slices): only one or two of the streaming form's eight warps work, each through whole stages of 64 or 128
// numbers whatever K is, and a second slice of a few numbers costs the tiles that a cluster joins as much as a full one.  Where
// the general form's blocks of 64 x 64 outputs fill much of the device once and little more, it is the fastest then; with more blocks than
// one or two an SM tiles of 64 rows that take both slices one after the other are.  All add in the same order.  us, the
// streaming form or joined tiles / the general form / tiles of 64 rows: K = 132, gated x 8,192 24 rows 29.3 / 15.6 / 19.5, 64 rows 31.6 /
// 16.0 / 19.7, 100 rows 33.8 / 25.5 / 20.7, 200 rows 58.4 / 49.4 / 39.8; x 2,048 200 rows 31.6 / 16.0 / 19.5; not gated x 8,192 64 rows
// 18.6 / 11.3, 100 rows 23.0 / 16.0 / 18.6, x 32,768 24 rows 33.3 / 34.9 / 19.2; K = 192 gated x 8,192 64 rows 31.6 / 23.4 / 24.6, 100 rows 33.8 / 34.1 / 25.4; K = 100 not gated x 8,192 100
// rows 16.8 / 12.2, gated x 8,192 12 rows 15.9 / 13.7; K = 48 gated x 32,768 4 rows 24.4 / 16.3.
enum { AS_MANY_INPUTS = 0, GENERAL_FORM = 1, TILES_OF_64 = 2 };
inline int few_inputs_form(int M, int N, int K, bool gated) {
    const int64_t blocks = (int64_t)ceil_div(M, 64) * ceil_div(N, 64), sms = sm_count();
    if (K > 256) return AS_MANY_INPUTS;
    if (M <= 8) return K < 64 && blocks > sms ? GENERAL_FORM : AS_MANY_INPUTS;
    if (M <= 16) {
        const bool whole_stages = K % 64 == 0 || K % 64 > 40;           // (or nearly)
        return K <= 144 && (blocks > sms || (blocks >= 128 && (K < 64 || !whole_stages))) ? GENERAL_FORM : AS_MANY_INPUTS;
    }
    if (K <= slice_len(K)) {
        if (M <= FEW_MAX) return N > (K <= 100 ? 2048 : 4096) ? GENERAL_FORM : AS_MANY_INPUTS;
        if (gated) return K < 64 || (blocks > 64 && (K <= 100 || (int64_t)ceil_div(M, 128) * ceil_div(N, 64) < 2 * sms)) ? GENERAL_FORM : AS_MANY_INPUTS;
        return (blocks > 100 && blocks <= 3 * sms) || (K < 64 && blocks > 64 && blocks <= 4 * sms) ? GENERAL_FORM : AS_MANY_INPUTS;
    }
    if (blocks < 64 || (blocks == 64 && K > (gated ? 176 : 144)) || (blocks <= (K > 240 ? 100 : 90) && K > 200)) return AS_MANY_INPUTS;
    if (gated) {
        if (blocks <= sms) return GENERAL_FORM;
        return blocks <= 2 * sms || (blocks < 4 * sms && (K <= 144 || (blocks > 3 * sms && K <= 192))) ? TILES_OF_64 : AS_MANY_INPUTS;
    }
    if (blocks <= (K <= 176 ? 2 : 1) * sms) return K <= 240 ? GENERAL_FORM : AS_MANY_INPUTS;
    return K <= 176 && blocks <= 8 * sms ? TILES_OF_64 : AS_MANY_INPUTS;
}

template <bool GATED>
int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int w_static, int form, cudaStream_t s) {
    if (form == TILES_OF_64) return gemm_f32_tiles<64, GATED ? 128 : 64, GATED ? 8 : 4, GATED, false>(A, W, C, M, N, K, w_static, s);
    // (few slices leave most warps of the streaming form without work: then tiles, which bring the weights once, from 17 rows on.
    // us streamed / as tiles, 17 rows, K = 256 x 4,096 10.4 / 9.0, x 32,768 70 / 33, gated x 4,096 17.2 / 14.7; K = 384 x 8,192 18.1 / 20.5,
    // x 32,768 66 / 47, gated x 16,384 67 / 52, x 32,768 135 / 89)
    const bool wide = M > 16 && ((K <= 256 && N >= 4096) || (K <= 384 && N >= (GATED ? 16384 : 32768)));
    if (M <= FEW_MAX && !wide) {
        // (16 outputs a block halve the trips of A's rows; with few outputs 8 a block fill the device)
        if (M <= 2) return gemm_f32_few<2, 1, GATED>(A, W, C, M, N, K, w_static, s);
        if (M <= 4) return gemm_f32_few<4, 1, GATED>(A, W, C, M, N, K, w_static, s);
        if (M <= 8 && ceil_div(N, GATED ? 8 : 16) <= sm_count()) return gemm_f32_few<8, 1, GATED>(A, W, C, M, N, K, w_static, s);
        if (M <= 8) return gemm_f32_few<8, 2, GATED>(A, W, C, M, N, K, w_static, s);
        return gemm_f32_few<16, 2, GATED>(A, W, C, M, N, K, w_static, s);
    }
    // (up to 64 rows of a gated product: half of a tile of 128 rows would be empty.  33 rows, gated 2 x 32,768 x 1,024: 439 us in tiles of
    // 128 x 128, 224 in tiles of 64 x 128.)
    if constexpr (GATED)
        if (M <= 64 && ceil_div(N, 64) >= 2 * sm_count()) return gemm_f32_tiles<64, 128, 8, true, false>(A, W, C, M, N, K, w_static, s);
    if ((int64_t)ceil_div(M, 128) * ceil_div(N, GATED ? 64 : 128) >= 2 * sm_count()) return gemm_f32_tiles<128, 128, 8, GATED, false>(A, W, C, M, N, K, w_static, s);
    if constexpr (GATED) return gemm_f32_tiles<64, 128, 8, true, true>(A, W, C, M, N, K, w_static, s);
    else return gemm_f32_tiles<64, 64, 4, false, true>(A, W, C, M, N, K, w_static, s);
}

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// SLICED: the inner dimension's slices are added up as the forms above add them.
template <typename T, typename TOut, bool GATED, bool SLICED>
__global__ void __launch_bounds__(256)
gemm_nt_kernel(const T* __restrict__ A, const T* __restrict__ W, TOut* __restrict__ C, int M, int N, int K) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ float Us[GATED ? BK : 1][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lrow = tid / 4, lk = (tid % 4) * 4;

    float acc[TM][TN] = {};
    float accu[GATED ? TM : 1][TN] = {};
    float total[SLICED ? TM : 1][TN], totalu[SLICED && GATED ? TM : 1][TN];
    const int len = SLICED ? slice_len(K) : 0;
    int until = len;                                     // where the slice at hand ends

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            const int m = m0 + lrow, n = n0 + lrow;
            As[lk + i][lrow] = (m < M && k < K) ? ld(A + (int64_t)m * K + k) : 0.f;
            Ws[lk + i][lrow] = (n < N && k < K) ? ld(W + (int64_t)n * K + k) : 0.f;
            if (GATED) Us[lk + i][lrow] = (n < N && k < K) ? ld(W + ((int64_t)N + n) * K + k) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN], u[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
            if (GATED) {
#pragma unroll
                for (int j = 0; j < TN; ++j) u[j] = Us[kk][tx * TN + j];
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
                    if (GATED) accu[i][j] = fmaf(a[i], u[j], accu[i][j]);
                }
        }
        if constexpr (SLICED) {
            if (k0 + BK == until || k0 + BK >= K) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        total[i][j] = until == len ? acc[i][j] : total[i][j] + acc[i][j];
                        acc[i][j] = 0.f;
                        if constexpr (GATED) {
                            totalu[i][j] = until == len ? accu[i][j] : totalu[i][j] + accu[i][j];
                            accu[i][j] = 0.f;
                        }
                    }
                until += len;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            float v = SLICED ? total[SLICED ? i : 0][j] : acc[i][j];
            if (GATED) v = v / (1.0f + expf(-v)) * (SLICED ? totalu[SLICED && GATED ? i : 0][j] : accu[GATED ? i : 0][j]);
            st(C + (int64_t)m * N + n, v);
        }
    }
}

template <typename T, typename TOut, bool GATED>
int gemm_nt(const void* A, const void* W, void* C, int M, int N, int K, int w_static, cudaStream_t s) {
    WICK_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return 0;
    if constexpr (std::is_same<T, float>::value && std::is_same<TOut, float>::value) {
        if (K % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && M <= 65535 * 64) {
            const int form = few_inputs_form(M, N, K, GATED);
            if (form != GENERAL_FORM) return gemm_f32<GATED>((const float*)A, (const float*)W, (float*)C, M, N, K, w_static, form, s);
            const dim3 grid(ceil_div(N, BN), ceil_div(M, BM));
            if (K <= slice_len(K)) gemm_nt_kernel<float, float, GATED, false><<<grid, 256, 0, s>>>((const float*)A, (const float*)W, (float*)C, M, N, K);
            else gemm_nt_kernel<float, float, GATED, true><<<grid, 256, 0, s>>>((const float*)A, (const float*)W, (float*)C, M, N, K);
            return check_launch("gemm_simt");
        }
    }
    dim3 grid(ceil_div(N, BN), ceil_div(M, BM));
    WICK_REQUIRE(grid.y <= 65535, "gemm: M=%d is beyond the grid limit", M);
    gemm_nt_kernel<T, TOut, GATED, false><<<grid, 256, 0, s>>>((const T*)A, (const T*)W, (TOut*)C, M, N, K);
    return check_launch("gemm_simt");
}

}  // namespace wick

using namespace wick;
typedef __nv_bfloat16 bf16;

// Names: wick_gemm_simt_<in>_<out>[_gated].  A [M,K], W [N,K] ([2N,K] gated), C [M,N].
// w_static: no kernel ever writes W (weights), so it may be fetched before the kernel launched before has finished.
WICK_API int wick_gemm_simt_bf16_bf16(const void* A, const void* W, void* C, int M, int N, int K, int w_static, void* s) {
    return gemm_nt<bf16, bf16, false>(A, W, C, M, N, K, w_static, (cudaStream_t)s);
}
WICK_API int wick_gemm_simt_bf16_f32(const void* A, const void* W, void* C, int M, int N, int K, int w_static, void* s) {
    return gemm_nt<bf16, float, false>(A, W, C, M, N, K, w_static, (cudaStream_t)s);
}
WICK_API int wick_gemm_simt_f32_f32(const void* A, const void* W, void* C, int M, int N, int K, int w_static, void* s) {
    return gemm_nt<float, float, false>(A, W, C, M, N, K, w_static, (cudaStream_t)s);
}
WICK_API int wick_gemm_simt_bf16_bf16_gated(const void* A, const void* W, void* C, int M, int N, int K, int w_static, void* s) {
    return gemm_nt<bf16, bf16, true>(A, W, C, M, N, K, w_static, (cudaStream_t)s);
}
WICK_API int wick_gemm_simt_f32_f32_gated(const void* A, const void* W, void* C, int M, int N, int K, int w_static, void* s) {
    return gemm_nt<float, float, true>(A, W, C, M, N, K, w_static, (cudaStream_t)s);
}
