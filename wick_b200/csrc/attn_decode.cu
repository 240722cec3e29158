// Decode attention (one new token per sequence) over the paged cache, fast form.
//
// grid = (splits, kv_heads, sequences).  A block handles W pages (64 positions each) of one
// sequence and kv head, for all query heads of that kv head, four at a time: a warp takes one
// page for one head, or for all four.  With one warp for a page's four heads a block of one
// or two pages was one or two warps that walked 64 KB of shared memory alone (4 sequences of 100
// positions, 4 kv heads of 128, float32 14.6 us, now 6.2; bfloat16, 8 sequences of 500, 13.4 us,
// now 11.9).  A block of four pages (heads of up to 64 numbers in bfloat16, 32 in float32) has
// four warps anyway: there a warp per head is better only while few blocks run, since a
// page is read from shared memory once per warp (64 sequences of 3,000 positions, 8 kv heads
// of 32, bfloat16, 32 heads: 122 us, a warp for four heads 70; heads of 64, 16 sequences of 250: 8.3 us and 9.9).
// Both give the same bits.
// One thread starts bulk copies (cp.async.bulk, completion on an mbarrier) of the pages'
// key and value tiles — each tile is one contiguous [64][head_dim] block of the cache —
// so that everything the block needs is in flight at once; scores, softmax statistics
// and the weighted sum of values are then computed from shared memory in float32.  A second kernel merges the
// splits of a sequence in index order.  The plain form of the same computation
// (global loads, no shared-memory staging) is attn_decode_kernel in attn.cu.
//
// Formulas: wick src/model.rs:520-553 (see attn.cu).  The split size is fixed by
// the head size and the element type, the order of every sum is fixed, so a
// sequence's result does not depend on what else is in the batch.
#include "common.cuh"
#include "sm100.cuh"

#ifndef WICK_HD
#error "compile with -DWICK_HD=<head_dim>"
#endif

namespace wick {
namespace fastdecode {

constexpr int HD = WICK_HD;
constexpr int GT = 4;                                  // query heads handled per pass

// First key that the query at position p sees: mask 0 every earlier key, 1 those of p's own block of `size`
// positions (blocks counted from position 0), 2 the last `size` positions.
__device__ __forceinline__ int first_visible_key(int p, int mask, int size) {
    return mask == 1 ? p / size * size : (mask == 2 ? max(0, p - size + 1) : 0);
}

template <typename T> struct Shape {
    static constexpr int EPC = Vec16<T>::N;                      // elements per 16-byte chunk
    static constexpr int CHUNKS = HD / EPC;                      // chunks per row
    static constexpr int TILE_BYTES = kPage * HD * (int)sizeof(T);
    static constexpr int W_RAW = 65536 / (2 * TILE_BYTES);
    static constexpr int WARPS = W_RAW >= 4 ? 4 : (W_RAW >= 2 ? 2 : 1);
    static constexpr int SPLIT = WARPS * kPage;
    static constexpr int pow2ceil(int v) { int p = 1; while (p < v) p <<= 1; return p; }
    static constexpr int TS = CHUNKS >= 32 ? 32 : pow2ceil(CHUNKS);   // lanes that share a key in the value pass
    static constexpr int CPL = (CHUNKS + TS - 1) / TS;
    static constexpr int KPI = 32 / TS;
    static constexpr bool SWZ = CHUNKS % 8 == 0;                 // visit chunks in a per-lane order that avoids bank conflicts
    static constexpr size_t SMEM = (size_t)2 * WARPS * TILE_BYTES + (size_t)(GT * HD + GT * SPLIT + WARPS * GT * HD) * sizeof(float);
};

// HPW: heads that a warp takes of its page.
template <typename T, int HPW>
__global__ void __launch_bounds__(Shape<T>::WARPS * (GT / HPW) * 32)
attn_decode_fast_kernel(const T* __restrict__ q, const T* __restrict__ kv, float* __restrict__ part_o,
                        float* __restrict__ part_ml, const int* __restrict__ kv_len_arr,
                        const int* __restrict__ page_table, int table_width, int n_heads, int n_kv, int max_splits,
                        float scale, int* status, int mask, int mask_size) {
    using S = Shape<T>;
    constexpr int EPC = S::EPC, CHUNKS = S::CHUNKS, WARPS = S::WARPS, SPLIT = S::SPLIT, PER_PAGE = GT / HPW, THREADS = WARPS * PER_PAGE * 32;
    constexpr int TS = S::TS, CPL = S::CPL, KPI = S::KPI;
    pdl_trigger();
    pdl_wait();
    q = fresh(q);
    kv = fresh(kv);
    const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    // A length beyond what the page table or the scratch (max_splits) holds is cut back to it
    // and reported: nothing outside the table or the scratch is touched.
    const int most = min(table_width * kPage, max_splits * SPLIT);
    int kv_len = kv_len_arr[b];
    if (kv_len > most) {
        if (split == 0 && kvh == 0 && threadIdx.x == 0 && status) atomicCAS(status, 0, 10);
        kv_len = most;
    }
    const int key_begin = split * SPLIT;
    if (key_begin >= kv_len) return;
    // the new token (position kv_len - 1) sees the keys from key_lo on; a split that lies before them has no part
    const int key_lo = first_visible_key(kv_len - 1, mask, mask_size);
    if (key_begin + SPLIT <= key_lo) return;
    const int group = n_heads / n_kv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    extern __shared__ __align__(128) uint8_t smem_raw[];
    T* k_s = reinterpret_cast<T*>(smem_raw);                               // [WARPS][64][HD]
    T* v_s = k_s + (size_t)WARPS * kPage * HD;                             // [WARPS][64][HD]
    float* q_s = reinterpret_cast<float*>(v_s + (size_t)WARPS * kPage * HD);   // [GT][HD]
    float* sc = q_s + GT * HD;                                             // [GT][SPLIT]
    float* red = sc + GT * SPLIT;                                          // [WARPS][GT][HD]
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    __shared__ float stat[2][GT][WARPS];                         // maxima, sums of a head's pages

    const int n_pages = min(WARPS, (kv_len - key_begin + kPage - 1) / kPage);
    if (tid == 0) {
        abort_flag = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
        const int64_t page_elems = (int64_t)2 * n_kv * kPage * HD;
        mbar_expect_tx(&bar, (uint32_t)(2 * n_pages * S::TILE_BYTES));
        for (int i = 0; i < n_pages; ++i) {
            const int page = page_table[(int64_t)b * table_width + key_begin / kPage + i];
            const T* kp = kv + page * page_elems + ((int64_t)kvh * kPage) * HD;
            bulk_load(k_s + (size_t)i * kPage * HD, kp, S::TILE_BYTES, &bar);
            bulk_load(v_s + (size_t)i * kPage * HD, kp + (int64_t)n_kv * kPage * HD, S::TILE_BYTES, &bar);
        }
    }
    const int w = warp / PER_PAGE, hh = warp % PER_PAGE * HPW;   // this warp's page and (first) head
    const T* kw = k_s + (size_t)w * kPage * HD;
    const T* vw = v_s + (size_t)w * kPage * HD;
    float* mine = sc + hh * SPLIT + w * kPage;                   // the warp's weights (its next head's SPLIT on)
    bool waited = false;

    for (int h0 = 0; h0 < group; h0 += GT) {
        const int nh = min(GT, group - h0);
        const bool warp_live = w < n_pages && hh < nh;
        __syncthreads();
        for (int i = tid; i < GT * HD; i += THREADS) {
            const int h = i / HD, d = i % HD;
            q_s[i] = h < nh ? ld(q + ((int64_t)b * n_heads + kvh * group + h0 + h) * HD + d) : 0.f;
        }
        __syncthreads();
        if (!waited) {
            mbar_wait(&bar, 0, &abort_flag, status, 4);
            waited = true;
            __syncthreads();
            if (abort_flag) break;          // the same decision in every thread
        }

        // ---- scores: lane = key (two keys per lane), chunks of the row in turn ----
        float s0[HPW], s1[HPW];
#pragma unroll
        for (int h = 0; h < HPW; ++h) s0[h] = s1[h] = 0.f;
        if (warp_live) {
#pragma unroll (HPW == 1 ? 4 : 2)
            for (int c = 0; c < CHUNKS; ++c) {
                const int cc = S::SWZ ? (c ^ (lane & 7)) : c;
                Vec16<T> k0, k1;
                k0.load(kw + (size_t)lane * HD + cc * EPC);
                k1.load(kw + (size_t)(lane + 32) * HD + cc * EPC);
#pragma unroll
                for (int h = 0; h < HPW; ++h) {
                    const float* qh = q_s + (hh + h) * HD + cc * EPC;
#pragma unroll
                    for (int e = 0; e < EPC; e += 4) {
                        const float4 q4 = *reinterpret_cast<const float4*>(qh + e);
                        s0[h] = fmaf(q4.x, k0.v[e], s0[h]); s0[h] = fmaf(q4.y, k0.v[e + 1], s0[h]);
                        s0[h] = fmaf(q4.z, k0.v[e + 2], s0[h]); s0[h] = fmaf(q4.w, k0.v[e + 3], s0[h]);
                        s1[h] = fmaf(q4.x, k1.v[e], s1[h]); s1[h] = fmaf(q4.y, k1.v[e + 1], s1[h]);
                        s1[h] = fmaf(q4.z, k1.v[e + 2], s1[h]); s1[h] = fmaf(q4.w, k1.v[e + 3], s1[h]);
                    }
                }
            }
        }
        const int at = key_begin + w * kPage + lane;
        const bool sees0 = warp_live && at < kv_len && at >= key_lo, sees1 = warp_live && at + 32 < kv_len && at + 32 >= key_lo;

        // ---- softmax statistics of the split, per head ----
#pragma unroll
        for (int h = 0; h < HPW; ++h) {
            s0[h] = sees0 ? __fmul_rn(s0[h], scale) : -INFINITY;
            s1[h] = sees1 ? __fmul_rn(s1[h], scale) : -INFINITY;
            const float m = warp_max(fmaxf(s0[h], s1[h]));
            if (lane == 0) stat[0][hh + h][w] = m;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < HPW; ++h) {
            float m = stat[0][hh + h][0];
#pragma unroll
            for (int i = 1; i < WARPS; ++i) m = fmaxf(m, stat[0][hh + h][i]);    // (finite: the split holds a visible key)
            const float p0 = expf(s0[h] - m), p1 = expf(s1[h] - m);
            mine[h * SPLIT + lane] = p0;
            mine[h * SPLIT + lane + 32] = p1;
            const float l = warp_sum(p0 + p1);
            if (lane == 0) stat[1][hh + h][w] = l;
        }
        __syncwarp();

        // ---- weighted sum of values: TS lanes share a key, each owns 16-byte chunks of the row ----
        const int tl = lane % TS, team = lane / TS;
        float acc[HPW][CPL][EPC];
#pragma unroll
        for (int h = 0; h < HPW; ++h)
#pragma unroll
            for (int c = 0; c < CPL; ++c)
#pragma unroll
                for (int e = 0; e < EPC; ++e) acc[h][c][e] = 0.f;
        if (warp_live) {
            const int keys_here = min(kPage, kv_len - key_begin - w * kPage);
#pragma unroll (HPW == 1 ? 8 : 4)
            for (int it = 0; it < kPage / KPI; ++it) {
                const int key = it * KPI + team;
                if (key < keys_here) {
#pragma unroll
                    for (int c = 0; c < CPL; ++c) {
                        const int chunk = tl + c * TS;
                        if (chunk < CHUNKS) {
                            Vec16<T> vv;
                            vv.load(vw + (size_t)key * HD + chunk * EPC);
#pragma unroll
                            for (int h = 0; h < HPW; ++h) {
                                const float p = mine[h * SPLIT + key];
#pragma unroll
                                for (int e = 0; e < EPC; ++e) acc[h][c][e] = fmaf(p, vv.v[e], acc[h][c][e]);
                            }
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int h = 0; h < HPW; ++h)
#pragma unroll
            for (int c = 0; c < CPL; ++c)
#pragma unroll
                for (int e = 0; e < EPC; ++e) {
                    float v = acc[h][c][e];
#pragma unroll
                    for (int o = TS; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    const int chunk = tl + c * TS;
                    if (team == 0 && chunk < CHUNKS) red[(w * GT + hh + h) * HD + chunk * EPC + e] = v;
                }
        __syncthreads();
        for (int i = tid; i < nh * HD; i += THREADS) {
            const int h = i / HD, d = i % HD;
            float v = red[h * HD + d];
#pragma unroll
            for (int j = 1; j < WARPS; ++j) v += red[(j * GT + h) * HD + d];
            const int64_t row = ((int64_t)b * n_heads + kvh * group + h0 + h) * max_splits + split;
            part_o[row * HD + d] = v;
            if (d == 0) {
                float most_of = stat[0][h][0], sum = stat[1][h][0];
#pragma unroll
                for (int j = 1; j < WARPS; ++j) {
                    most_of = fmaxf(most_of, stat[0][h][j]);
                    sum += stat[1][h][j];
                }
                part_ml[row * 2] = most_of;
                part_ml[row * 2 + 1] = sum;
            }
        }
    }
    if (!waited) mbar_wait(&bar, 0, &abort_flag, status, 4);     // never leave with copies in flight
    if (abort_flag) {
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
}

template <typename T>
__global__ void attn_decode_fast_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                              const int* __restrict__ kv_len_arr, T* __restrict__ out, int n_heads,
                                              int max_splits, int mask, int mask_size, const float* __restrict__ sink) {
    constexpr int SPLIT = Shape<T>::SPLIT;
    pdl_trigger();
    pdl_wait();
    part_o = fresh(part_o);
    part_ml = fresh(part_ml);
    const int head = blockIdx.x, b = blockIdx.y;
    const int n_splits = min((kv_len_arr[b] + SPLIT - 1) / SPLIT, max_splits);   // (a longer length was cut back and reported)
    const int64_t row0 = ((int64_t)b * n_heads + head) * max_splits;
    // (splits before the first visible key wrote nothing; a sink is a score without a value)
    const int s_first = kv_len_arr[b] > 0 ? min(first_visible_key(kv_len_arr[b] - 1, mask, mask_size) / SPLIT, n_splits) : 0;
    float m = sink ? sink[head] : -INFINITY;
    for (int s = s_first; s < n_splits; ++s) m = fmaxf(m, part_ml[(row0 + s) * 2]);
    float denom = sink ? expf(sink[head] - m) : 0.f;
    for (int s = s_first; s < n_splits; ++s) denom += expf(part_ml[(row0 + s) * 2] - m) * part_ml[(row0 + s) * 2 + 1];
    const float inv = n_splits > s_first ? 1.0f / denom : 0.f;
    for (int d = threadIdx.x; d < HD; d += blockDim.x) {
        float v = 0.f;
        for (int s = s_first; s < n_splits; ++s) v = fmaf(expf(part_ml[(row0 + s) * 2] - m), part_o[(row0 + s) * HD + d], v);
        st(out + ((int64_t)b * n_heads + head) * HD + d, v * inv);
    }
}

template <typename T>
int run(const void* q, const void* kv, void* out, float* scratch, int64_t scratch_floats, const int* kv_len, int n_seqs,
        int max_kv_len, const int* page_table, int table_width, int n_heads, int n_kv, float scale, int* status,
        cudaStream_t s, int mask = 0, int mask_size = 0, const float* sink = nullptr) {
    using S = Shape<T>;
    WICK_REQUIRE(mask == 0 || ((mask == 1 || mask == 2) && mask_size > 0), "attention decode: mask %d of size %d", mask, mask_size);
    WICK_REQUIRE(n_heads > 0 && n_kv > 0 && n_heads % n_kv == 0, "attention: %d heads over %d kv heads", n_heads, n_kv);
    WICK_REQUIRE(n_kv <= 65535 && n_seqs <= 65535, "attention: grid limit");
    if (n_seqs == 0) return 0;
    const int max_splits = ceil_div(max_kv_len > 0 ? max_kv_len : 1, S::SPLIT);
    const int64_t need = (int64_t)n_seqs * n_heads * max_splits * (HD + 2);
    WICK_REQUIRE(scratch_floats >= need, "attention decode: scratch of %lld floats, %lld needed",
                 (long long)scratch_floats, (long long)need);
    float* ml = scratch + (int64_t)n_seqs * n_heads * max_splits * HD;
#define WICK_DECODE(HPW)                                                                                                                                  \
    do {                                                                                                                                                  \
        static bool raised = false;                                                                                                                       \
        if (!raised) {                                                                                                                                    \
            WICK_CUDA(cudaFuncSetAttribute(attn_decode_fast_kernel<T, HPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));                  \
            raised = true;                                                                                                                                \
        }                                                                                                                                                 \
        WICK_CUDA(launch(attn_decode_fast_kernel<T, HPW>, dim3(max_splits, n_kv, n_seqs), dim3(S::WARPS * (GT / HPW) * 32), S::SMEM, s, (const T*)q,        \
                         (const T*)kv, scratch, ml, kv_len, page_table, table_width, n_heads, n_kv, max_splits, scale, status, mask, mask_size));          \
    } while (0)
    // (a warp takes one head up to a block for every SM, or every other one where pages are small, 16 or 32 numbers a head in bfloat16 and
    // 16 in float32: of 1,225 sizes measured none was slower by more than runs differ than the form before, a warp for four heads and
    // barriers for every head and sum)
    bool done = false;
    if constexpr (S::WARPS == 4) {
        if ((int64_t)max_splits * n_kv * n_seqs * (S::TILE_BYTES < 8192 ? 2 : 1) > sm_count()) {
            WICK_DECODE(GT);
            done = true;
        }
    }
    if (!done) WICK_DECODE(1);
#undef WICK_DECODE
    if (int e = check_launch("attn_decode")) return e;
    WICK_CUDA(launch(attn_decode_fast_merge_kernel<T>, dim3(n_heads, n_seqs), dim3(HD >= 128 ? 128 : 64), 0, s,
                     (const float*)scratch, (const float*)ml, kv_len, (T*)out, n_heads, max_splits, mask, mask_size, sink));
    return check_launch("attn_decode_merge");
}

}  // namespace fastdecode
}  // namespace wick

using namespace wick;
typedef __nv_bfloat16 bf16;

// Positions per split of the fast decode kernels (the scratch holds, per
// sequence and head, ceil(max_kv_len / split) partial results of HD + 2 floats).
// The arguments of wick_attn_decode_bf16 / _f32 below, then the mask (0, or 1 / 2 with its size) and the sinks
// (float32 [n_heads] or null).
WICK_API int wick_attn_decode_masked_bf16(const void* q, const void* kv, void* out, float* scratch, long long scratch_floats,
                                          const int* kv_len, int n_seqs, int max_kv_len, const int* page_table,
                                          int table_width, int n_heads, int n_kv, float scale, int* status, int mask,
                                          int mask_size, const float* sink, void* s) {
    return fastdecode::run<bf16>(q, kv, out, scratch, scratch_floats, kv_len, n_seqs, max_kv_len, page_table, table_width,
                                 n_heads, n_kv, scale, status, (cudaStream_t)s, mask, mask_size, sink);
}
WICK_API int wick_attn_decode_masked_f32(const void* q, const void* kv, void* out, float* scratch, long long scratch_floats,
                                         const int* kv_len, int n_seqs, int max_kv_len, const int* page_table,
                                         int table_width, int n_heads, int n_kv, float scale, int* status, int mask,
                                         int mask_size, const float* sink, void* s) {
    return fastdecode::run<float>(q, kv, out, scratch, scratch_floats, kv_len, n_seqs, max_kv_len, page_table, table_width,
                                  n_heads, n_kv, scale, status, (cudaStream_t)s, mask, mask_size, sink);
}

WICK_API int wick_attn_decode_split_bf16() { return fastdecode::Shape<bf16>::SPLIT; }
WICK_API int wick_attn_decode_split_f32() { return fastdecode::Shape<float>::SPLIT; }

// q, out: [n_seqs, n_heads, HD]; kv: one schedule entry's cache.  status: device
// int that receives 4 if a block gave up waiting for its copies, 10 if a length was beyond the
// page table or max_kv_len (it is then cut back to what they hold).
WICK_API int wick_attn_decode_bf16(const void* q, const void* kv, void* out, float* scratch, int64_t scratch_floats,
                                   const int* kv_len, int n_seqs, int max_kv_len, const int* page_table,
                                   int table_width, int n_heads, int n_kv, float scale, int* status, void* s) {
    return fastdecode::run<bf16>(q, kv, out, scratch, scratch_floats, kv_len, n_seqs, max_kv_len, page_table, table_width,
                                 n_heads, n_kv, scale, status, (cudaStream_t)s);
}
WICK_API int wick_attn_decode_f32(const void* q, const void* kv, void* out, float* scratch, int64_t scratch_floats,
                                  const int* kv_len, int n_seqs, int max_kv_len, const int* page_table,
                                  int table_width, int n_heads, int n_kv, float scale, int* status, void* s) {
    return fastdecode::run<float>(q, kv, out, scratch, scratch_floats, kv_len, n_seqs, max_kv_len, page_table, table_width,
                                  n_heads, n_kv, scale, status, (cudaStream_t)s);
}

// ---------------------------------------------------------------------------
// Decode attention for callers that cannot allocate device memory (declared in
// attn_decode_noalloc.h; wick has nothing like it).
//
// wick_attn_decode_bf16 above needs a scratch buffer from its caller for the
// per-split partial results.  A host that has no allocator to ask — a plug-in
// inside another runtime's memory pool, a real-time loop that may not block in
// cudaMalloc, a process whose memory budget is fixed at load time — can call
// this entry point instead: the partial results go to a fixed array that is part
// of this library's image on the device.
//
// * The array holds kNoAllocFloats float32 (8 MiB).  Every GPU that loads this
//   library carries it until the process exits.  A call that needs more
//   (n_seqs * n_heads * ceil(max_kv_len / split) * (head_dim + 2) floats) is
//   refused with an error; nothing is launched.
// * In host code the array's name is only a handle.  The device address is
//   looked up with cudaGetSymbolAddress, once per device, by the first call made
//   while that device is current; make that first call before capturing a stream.
// * All calls share the one array, and it keeps what the last call left.  Nothing
//   in it has to start at zero: every entry a call reads was written by that
//   call.  Two calls that overlap on the GPU (different streams) race on it; keep
//   calls that use this entry point on one stream or order them with events.
// * No cudaMalloc, cudaFree or other allocating routine is called, here or below.
namespace wick {
namespace fastdecode {

constexpr long long kNoAllocFloats = 2ll * 1024 * 1024;
static __device__ __align__(256) float g_noalloc_scratch[kNoAllocFloats];

static int noalloc_scratch(float** out) {
    // (No lock: two host threads may both look the symbol up on a device's first call; they
    // store the same address.)
    static float* per_device[64] = {};
    int dev = -1;
    WICK_CUDA(cudaGetDevice(&dev));
    WICK_REQUIRE(dev >= 0 && dev < 64, "attention decode (no allocation): device index %d is out of range", dev);
    if (per_device[dev] == nullptr) {
        float* p = nullptr;
        WICK_CUDA(cudaGetSymbolAddress((void**)&p, g_noalloc_scratch));
        WICK_REQUIRE(p != nullptr, "attention decode (no allocation): the scratch array has no device address");
        per_device[dev] = p;
    }
    *out = per_device[dev];
    return 0;
}

}  // namespace fastdecode
}  // namespace wick

WICK_API long long wick_attn_decode_noalloc_capacity() { return wick::fastdecode::kNoAllocFloats; }

WICK_API int wick_attn_decode_noalloc_bf16(const void* q, const void* kv, void* out, const int* kv_len, int n_seqs,
                                           int max_kv_len, const int* page_table, int table_width, int n_heads,
                                           int n_kv, float scale, int* status, void* s) {
    using namespace wick::fastdecode;
    WICK_REQUIRE(n_seqs >= 0 && n_heads > 0 && max_kv_len >= 0, "attention decode (no allocation): bad sizes");
    const long long splits = (max_kv_len > 0 ? max_kv_len : 1) / Shape<bf16>::SPLIT +
                             ((max_kv_len > 0 ? max_kv_len : 1) % Shape<bf16>::SPLIT != 0);
    const long long need = (long long)n_seqs * n_heads * splits * (HD + 2);
    WICK_REQUIRE(need <= kNoAllocFloats,
                 "attention decode (no allocation): %d sequences x %d heads x %lld splits need %lld floats of scratch, "
                 "the built-in array holds %lld", n_seqs, n_heads, splits, need, kNoAllocFloats);
    float* scratch = nullptr;
    if (int e = noalloc_scratch(&scratch)) return e;
    return run<bf16>(q, kv, out, scratch, kNoAllocFloats, kv_len, n_seqs, max_kv_len, page_table, table_width, n_heads,
                     n_kv, scale, status, (cudaStream_t)s);
}
