// D[m, n] = sum_k A[m, k] * B[n, k] for bfloat16 operands that are both
// contiguous along k, on the 5th-generation tensor cores of sm_100a:
//
//   * TMA (cp.async.bulk.tensor, 128-byte swizzle) stages 128 x 64 tiles of A and
//     bn x 64 tiles of B in a ring of shared-memory buffers;
//   * one elected thread issues tcgen05.mma (M = 128, N = bn, K = 16 per
//     instruction) with the float32 accumulator in tensor memory;
//   * four warps read the accumulator back with tcgen05.ld and write the result.
//
// The same kernel serves both shapes of work.  Prompts: A = activations
// [tokens, k], B = weights [out, k], D written row-major [tokens, out].  Decode
// (few tokens): A = weights, B = activations (bn = tokens rounded up to 16), D
// written transposed, so that the 128-row side of the instruction is always
// full and every CTA streams a 128-row slab of the weight matrix.  Options:
// a gated pair (two accumulators, silu(g) * u in the epilogue; wick
// src/model.rs:493-501), float32 or bfloat16 output, and a split of the k range
// over blockIdx.z into float32 partial sums that the consumer adds in index
// order.  Each output element is accumulated along k in index order within a
// split, whatever the tile it falls into, so a row's result does not depend on
// the other rows of the batch.
//
// Every wait on an mbarrier is bounded (about one second); when a wait gives up,
// the kernel records a code in *status, stops waiting anywhere, lets copies in
// flight land, frees its tensor memory and returns.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "sm100.cuh"
#include "tcgen05.cuh"

namespace wick {

constexpr int BM = 128;            // rows of the A tile = M of the instruction
constexpr int BK = 64;             // k per stage: 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int MAX_STAGES = 12;
constexpr int NUM_THREADS = 192;   // warp 0: TMA, warp 1: MMA + tensor memory, warps 2-5: epilogue

struct GemmParams {
    int a_rows;                    // valid rows of A (outputs beyond are not written)
    int b_rows;                    // valid rows of B
    int bn;                        // rows of a B tile = N of the instruction (multiple of 16, <= 256)
    int k_blocks;                  // ceil(k / 64)
    int k_blocks_per_split;
    int stages;
    int gated;                     // 0 none, 1 the pair lives in A (two tiles), 2 the pair lives in B (two tiles),
                                   // 3 the pair lives in A and shares one tile: rows 0-63 gate, rows 64-127 up
    int pair_offset;               // row offset of the second half of the pair
    int transposed;                // 0: out[m * ldo + n], 1: out[n * ldo + m]
    int out_f32;
    int total_tiles, grid_m, grid_n;   // tiles = grid_m * grid_n * splits, the m tile varying fastest
    int a_packed, b_packed;        // that operand is stored as tiles of 128 rows x 64 columns (see wick_gemm_tc)
    int a_static;                  // A is never written by a kernel (weights): it may be fetched before the
    int b_static;                  //   preceding kernel has finished; likewise B
    long long ldo;
    long long split_stride;        // elements between the partial results of two splits
    void* out;
    int* status;
};

// (A struct of its own: with these fields in GemmParams the kernels that do not use them came out with up to half as many registers
// again, and the decode products were 1 to 3 % slower.)
constexpr int NAMED_WORDS = 32;
struct GroupedParams : GemmParams {
    // Grouped (several matrices of A one after the other, see wick_gemm_tc_grouped): the m tiles of one matrix, its padded
    // rows, the rows of B it is multiplied with (0: all matrices with the same rows), elements of out between two matrices'
    // results; the step's token ids and the table that names each id's `top` matrices.
    int group_tiles, group_rows, group_b_rows, top, n_tokens;
    int n_groups;                                   // of matrices (ranked; at most 32 NAMED_WORDS)
    long long group_out;
    const int *tokens, *table;
    // A matrix that every token uses besides (the shared expert's; its m tiles follow the groups'), multiplied with rows of its own:
    // operands, sizes and result as for the groups.  shared_tiles 0: there is none.
    int groups_end, shared_tiles, shared_rows, shared_pair_offset, shared_k_blocks, shared_k_blocks_per_split;
    long long shared_split_stride;
    void* shared_out;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Persistent: block b works on tiles b, b + gridDim.x, ...  A tile is (m tile, n
// tile, split) with the m tile varying fastest, so that blocks running at the
// same time share B tiles through the L2 cache.  With two accumulators in tensor
// memory the epilogue of one tile overlaps the main loop of the next.
//
// Grouped: the m tiles run over several matrices (experts), all multiplied with the same few rows of B or each with rows of
// its own.  A block whose matrix no token of the step uses leaves at once, and of the others' results only those of tokens
// that use the matrix are written.
//
// Ranked: there are blocks for as many matrices as the step can name, the blocks of slot i taking the i-th that it names.  (With blocks
// for all of 256 experts of 512 x 1,024, eight a token, a layer of one token took 48 us, with the kernels that walk the rows 40; ranked 18.
// It costs half a microsecond, and the blocks of experts that are named late start late.)
//
// Joined (a gated pair that shares a tile, transposed bfloat16 result): the runs of the inner dimension along blockIdx.z are a
// cluster; every block leaves its accumulator in its shared memory (the ring is idle by then), and the blocks finish a share of the
// tokens each, adding the runs' sums in index order over distributed shared memory.  A pair cannot be left as partial sums, and
// without runs a narrow matrix fills a part of the device only: 5,120 + 5,120 rows of 2,048 at one token are 80 blocks,
// 16.5 us; as 240 blocks 11.7 us.  With up to four runs a block finishes many results: four neighbours a thread (one at a time, 128 tokens
// x 512 inputs, two runs took 15.9 us, 12.8 without runs; now 8.3); with more, one at a time (2,048 inputs, eight runs, 24 tokens 6.8 us
// against 7.7).
template <bool PERSIST, int GATED, bool TRANSPOSED, bool OUT_F32, bool GROUPED, bool JOINED, bool RANKED = false>
__device__ __forceinline__ void
gemm_tc_block(const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap* shared_a, const CUtensorMap* shared_b,
              const std::conditional_t<GROUPED, GroupedParams, GemmParams>& p) {
    // A gated pair that shares a tile leaves its accumulator in the ring, which is idle by then, and all six warps finish the results from
    // there, four neighbours a thread.  (Gate and up values lie in different warps' parts of tensor memory.  Crossing 16 columns at a time,
    // with two barriers each and the four epilogue warps at work, 64 / 100 tokens x 2 x 12,288 outputs of 4,096 took 39.5 / 46.0 us; now 37.4 / 42.9.)
    constexpr bool STAGED = GATED == 3 && !GROUPED && !OUT_F32 && !PERSIST;
    static_assert(!JOINED || STAGED, "runs are joined where the accumulator is staged");
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[MAX_STAGES];
    __shared__ uint64_t empty_bar[MAX_STAGES];
    __shared__ uint64_t acc_full[2];
    __shared__ uint64_t acc_empty[2];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    __shared__ int ok_w[4];
    __shared__ float xch[GATED == 3 && !STAGED ? 2 : 1][64][17];   // gated == 3: up values on their way to the warps that hold the gate values

    __shared__ unsigned uses[GROUPED ? 8 : 1];   // grouped: a bit per token that uses this block's matrix
    __shared__ unsigned named[RANKED ? NAMED_WORDS : 1];               // ranked: a bit per matrix that the step names

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int group = 0, bx = blockIdx.x;                          // this block's matrix, its m tile there
    if constexpr (GROUPED) {
        group = bx < p.groups_end ? bx / p.group_tiles : -1;       // (-1: the shared matrix)
        bx -= group < 0 ? p.groups_end : group * p.group_tiles;
        // (the step's description is the host's or step_prepare's: it may be read before griddepcontrol.wait)
        if (threadIdx.x < 8) uses[threadIdx.x] = group < 0 ? ~0u : 0u;
        if (RANKED && group >= 0) {
            const int words = (p.n_groups + 31) / 32;
            for (int i = threadIdx.x; i < words; i += NUM_THREADS) named[i] = 0u;
            __syncthreads();
            for (int i = threadIdx.x; i < p.n_tokens * p.top; i += NUM_THREADS) {
                const int e = p.table[(long long)p.tokens[i / p.top] * p.top + i % p.top];
                if (e >= 0 && e < p.n_groups) atomicOr(&named[e >> 5], 1u << (e & 31));
            }
            __syncthreads();
            int word = 0, rank = group;                      // (every thread finds the same one)
            while (word < words && rank >= __popc(named[word])) rank -= __popc(named[word++]);
            if (word == words) return;
            unsigned left = named[word];
            while (rank-- > 0) left &= left - 1;
            group = 32 * word + __ffs(left) - 1;
        }
        __syncthreads();
        bool mine = group < 0;
        for (int i = threadIdx.x; i < (group < 0 ? 0 : p.n_tokens * p.top); i += NUM_THREADS) {
            const int t = i / p.top;
            if (p.table[(long long)p.tokens[t] * p.top + (i - t * p.top)] == group) {
                mine = true;
                atomicOr(&uses[t >> 5], 1u << (t & 31));
            }
        }
        if (!__syncthreads_or(mine)) return;
    }
    const int tile_m = GATED == 3 ? BM / 2 : BM;
    const int a_tiles = GATED == 1 ? 2 : 1, b_tiles = GATED == 2 ? 2 : 1;
    const uint32_t a_bytes = BM * BK * 2, b_bytes = (uint32_t)p.bn * BK * 2;
    const uint32_t stage_bytes = a_tiles * a_bytes + b_tiles * b_bytes;
    uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int n_acc = (GATED == 1 || GATED == 2) ? 2 : 1;
    const int acc_cols = n_acc * p.bn;                       // columns of one tile's accumulators
    // PERSIST: block b runs tiles b, b + gridDim.x, ...; otherwise the grid is (m tiles, n tiles, splits).
    const int my_tiles = PERSIST ? (p.total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 1;
    const int w_first = PERSIST ? (int)blockIdx.x : 0, w_end = PERSIST ? p.total_tiles : 1;
    const int w_step = PERSIST ? (int)gridDim.x : 1;
    const int acc_bufs = (my_tiles > 1 && 2 * acc_cols <= 512) ? 2 : 1;
    uint32_t tmem_cols = 32;
    while (tmem_cols < (uint32_t)(acc_bufs * acc_cols)) tmem_cols <<= 1;

    auto tile_coords = [&](int w, int& m0, int& n0, int& kb_begin, int& n_kb, int& z) {
        int x, y;
        if (PERSIST) {
            x = w % p.grid_m;
            y = (w / p.grid_m) % p.grid_n;
            z = w / (p.grid_m * p.grid_n);
        } else {                                             // one tile per block: a three-dimensional grid
            x = GROUPED ? bx : (int)blockIdx.x;
            y = blockIdx.y;
            z = blockIdx.z;
        }
        m0 = x * tile_m;
        n0 = y * p.bn;
        if constexpr (GROUPED) {
            const int per = group < 0 ? p.shared_k_blocks_per_split : p.k_blocks_per_split;
            kb_begin = z * per;
            n_kb = min(group < 0 ? p.shared_k_blocks : p.k_blocks, kb_begin + per) - kb_begin;
        } else {
            kb_begin = z * p.k_blocks_per_split;
            n_kb = min(p.k_blocks, kb_begin + p.k_blocks_per_split) - kb_begin;
        }
    };
    // this block's operands and result
    const CUtensorMap *ma = &map_a, *mb = &map_b;
    int k_blocks = p.k_blocks, pair_offset = p.pair_offset, a_rows = p.a_rows;
    long long ldo = p.ldo;
    if constexpr (GROUPED) {
        if (group < 0) {
            ma = shared_a;
            mb = shared_b;
            k_blocks = p.shared_k_blocks;
            pair_offset = p.shared_pair_offset;
            ldo = a_rows = p.shared_rows;
        }
    }

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 4);                     // one arrival per epilogue warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    pdl_trigger();

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        // (Here and below the whole warp walks through the loop and one elected lane issues, where a branch of one lane did.  With that, loops
        // that stay loops and waits out of line a decode step of one sequence on a small model went from 334 to 319 us.)
        const bool one = elect_one();
        int s = 0;                                           // the ring's next stage, how often the ring has been gone through
        uint32_t round = 0;
        bool ok = true;
#pragma unroll 1
        for (int w = w_first; w < w_end && ok; w += w_step) {
            int m0, n0, kb_begin, n_kb, z;
            tile_coords(w, m0, n0, kb_begin, n_kb, z);
            if constexpr (GROUPED) {                         // (from here on rows of the operands, not of the result)
                m0 += max(group, 0) * p.group_rows;
                n0 += max(group, 0) * p.group_b_rows;
            }
            // Coordinates of the box that holds rows row.. of k-block kb: in a row-major
            // operand (kb * 64, row); in a packed one the tile (row / 128, kb) lies as
            // 128 contiguous lines of 128 bytes.
            auto load = [&](const CUtensorMap* map, int packed, int s, void* dst, int kb, int row) {
                tma_load_2d(map, &full_bar[s], dst, packed ? 0 : kb * BK, packed ? ((row >> 7) * k_blocks + kb) * 128 + (row & 127) : row);
            };
            auto load_a = [&](int i, int s) {
                uint8_t* st = tiles + (size_t)s * stage_bytes;
                const int kb = kb_begin + i;
                load(ma, p.a_packed, s, st, kb, m0);
                if (a_tiles == 2) load(ma, p.a_packed, s, st + a_bytes, kb, m0 + pair_offset);
                if (GATED == 3) load(ma, p.a_packed, s, st + a_bytes / 2, kb, m0 + pair_offset);   // 64-row boxes
            };
            auto load_b = [&](int i, int s) {
                uint8_t* sb = tiles + (size_t)s * stage_bytes + a_tiles * a_bytes;
                const int kb = kb_begin + i;
                load(mb, p.b_packed, s, sb, kb, n0);
                if (p.b_packed && p.bn > 128) load(mb, p.b_packed, s, sb + 128 * BK * 2, kb, n0 + 128);   // 256 rows: two tiles
                if (b_tiles == 2) load(mb, p.b_packed, s, sb + b_bytes, kb, n0 + pair_offset);
            };
            // The first ring of stages is free.  An operand that no kernel
            // writes (weights) is fetched before the preceding kernel has
            // finished; the other one only after pdl_wait.
            const int first = round == 0 && s == 0 ? min(n_kb, p.stages) : 0;
#pragma unroll 1
            for (int pass = first > 0 ? 0 : 2; pass < 3; ++pass) {
                if (pass == 1) pdl_wait();
                // pass 0: what is static of the first ring; 1: the rest of it; 2: everything behind it
#pragma unroll 1
                for (int i = pass == 2 ? first : 0; i < (pass == 2 ? n_kb : first); ++i) {
                    int at = i;
                    if (pass == 2) {
                        at = s;
                        if (round > 0) ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[s], (round & 1) ^ 1, &abort_flag, p.status, 1));
                        if (!ok) break;
                        if (++s == p.stages) s = 0, ++round;
                    }
                    if (one) {
                        if (pass != 1) mbar_expect_tx(&full_bar[at], stage_bytes);
                        if (pass == 2 || (p.a_static != 0) == (pass == 0)) load_a(i, at);
                        if (pass == 2 || (p.b_static != 0) == (pass == 0)) load_b(i, at);
                    }
                    __syncwarp();
                }
                if (pass == 1) {
                    s = first;
                    if (s == p.stages) s = 0, round = 1;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // kind::f16, A and B bfloat16 and k-major, float32 accumulator, M = 128, N = bn
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
        const bool one = elect_one();
        int s = 0;
        uint32_t round = 0;
        bool ok = true;
        int t = 0;
#pragma unroll 1
        for (int w = w_first; w < w_end && ok; w += w_step, ++t) {
            int m0, n0, kb_begin, n_kb, z;
            tile_coords(w, m0, n0, kb_begin, n_kb, z);
            const int buf = acc_bufs == 2 ? (t & 1) : 0;
            const uint32_t use = acc_bufs == 2 ? (uint32_t)(t >> 1) : (uint32_t)t;   // how often this buffer was used before
            if (t > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], (use & 1) ^ 1, &abort_flag, p.status, 5));  // the epilogue has drained it
                if (!ok) break;
                tc_fence_after();
            }
            const uint32_t d0 = tmem_base + buf * acc_cols;
#pragma unroll 1
            for (int i = 0; i < n_kb; ++i) {
                ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], round & 1, &abort_flag, p.status, 2));
                if (!ok) break;
                tc_fence_after();
                const uint32_t sa = smem_u32(tiles + (size_t)s * stage_bytes);
                const uint32_t sb = sa + a_tiles * a_bytes;
                if (one) {
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        const uint32_t acc = (i > 0 || k > 0) ? 1u : 0u;
                        const uint64_t da = smem_desc(sa + k * UMMA_K * 2), db = smem_desc(sb + k * UMMA_K * 2);
                        tc_mma(d0, da, db, idesc, acc);
                        if (GATED == 1) tc_mma(d0 + p.bn, smem_desc(sa + a_bytes + k * UMMA_K * 2), db, idesc, acc);
                        if (GATED == 2) tc_mma(d0 + p.bn, da, smem_desc(sb + b_bytes + k * UMMA_K * 2), idesc, acc);
                    }
                    tc_commit(&empty_bar[s]);          // the stage is free once these instructions have read it
                    if (i + 1 == n_kb) tc_commit(&acc_full[buf]);   // this tile's accumulator is complete
                }
                __syncwarp();
                if (++s == p.stages) s = 0, ++round;
            }
            if (n_kb <= 0 && one) tc_commit(&acc_full[buf]);
        }
    } else {
        // ---------------- epilogue: tensor memory -> global ----------------
        const int q = warp & 3;                    // this warp reads lanes 32q .. 32q+31
        pdl_wait();                                // the output may alias memory an earlier kernel still reads
        int t = 0;
#pragma unroll 1
        for (int w = w_first; w < w_end; w += w_step, ++t) {
            int m0, n0, kb_begin, n_kb, z;
            tile_coords(w, m0, n0, kb_begin, n_kb, z);
            const int buf = acc_bufs == 2 ? (t & 1) : 0;
            const uint32_t use = acc_bufs == 2 ? (uint32_t)(t >> 1) : (uint32_t)t;
            const int m = m0 + q * 32 + lane;
            const uint32_t lane_addr = tmem_base + buf * acc_cols + ((uint32_t)(q * 32) << 16);
            char* out_base = (char*)p.out + (size_t)z * p.split_stride * (OUT_F32 ? 4 : 2);
            if constexpr (GROUPED) {
                if (group >= 0) out_base += (size_t)group * p.group_out * (OUT_F32 ? 4 : 2);
                else out_base = (char*)p.shared_out + (size_t)z * p.shared_split_stride * (OUT_F32 ? 4 : 2);
            }
            // One answer for the four epilogue warps, so that they leave the loop together.
            const bool ok_warp = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], use & 1, &abort_flag, p.status, 3));
            bool ok = ok_warp;
            if (my_tiles > 1 || (GATED == 3 && !STAGED)) {            // (a block with one plain tile has nothing left to agree on)
                if (lane == 0) ok_w[q] = ok_warp ? 1 : 0;
                asm volatile("bar.sync 1, 128;" ::: "memory");
                ok = ok_w[0] && ok_w[1] && ok_w[2] && ok_w[3];
                asm volatile("bar.sync 1, 128;" ::: "memory");
            }
            tc_fence_after();
            if constexpr (STAGED) {
                // column n of the accumulator at tiles[n][128 rows]
                float* acc = reinterpret_cast<float*>(tiles) + q * 32 + lane;
#pragma unroll 1
                for (int c0 = 0; c0 < p.bn; c0 += 32, acc += 32 * BM) {
                    float v[32];
                    tc_ld16_nowait(lane_addr + c0, v);
                    tc_ld16_nowait(lane_addr + c0 + 16, v + 16);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[j * BM] = v[j];
                    if (c0 + 16 < p.bn)
#pragma unroll
                        for (int j = 16; j < 32; ++j) acc[j * BM] = v[j];
                }
            } else if (GATED == 3) {
                // Lanes 0-63 of the accumulator hold gate rows, lanes 64-127 the up rows of the
                // same outputs (transposed output only).  Of every 16 columns the warps of the gate
                // rows finish and store the first 8, the warps of the up rows the last 8 (the
                // activation's exponential and division are the long part of a decode block's
                // end: all four warps share them); what each side lacks crosses through shared
                // memory.
                const int mg = m0 + (q & 1) * 32 + lane, xrow = (q & 1) * 32 + lane;
                const bool upper = q >= 2;
#pragma unroll 1
                for (int c0 = 0; c0 < p.bn; c0 += 16) {
                    float v[16];
                    if (ok && n_kb > 0) tc_ld16(lane_addr + c0, v);
                    float (*xb)[17] = xch[(c0 >> 4) & 1];
#pragma unroll
                    for (int j = 0; j < 8; ++j) xb[xrow][upper ? j : 8 + j] = upper ? v[j] : v[8 + j];
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (ok && n_kb > 0 && mg < a_rows) {
#pragma unroll
                        for (int jj = 0; jj < 8; ++jj) {
                            const int j = upper ? 8 + jj : jj;
                            const int n = n0 + c0 + j;
                            bool wanted = n < p.b_rows;
                            if constexpr (GROUPED) wanted = wanted && (uses[n >> 5] >> (n & 31) & 1u);
                            if (wanted) {
                                const float mine = upper ? v[8 + jj] : v[jj], other = xb[xrow][j];
                                const float g = upper ? other : mine, u = upper ? mine : other;
                                const float r = g / (1.0f + expf(-g)) * u;
                                const long long off = (long long)n * ldo + mg;
                                if (OUT_F32) ((float*)out_base)[off] = r;
                                else ((__nv_bfloat16*)out_base)[off] = __float2bfloat16_rn(r);
                            }
                        }
                    }
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");     // the exchange buffers are free for the next tile
            } else if (TRANSPOSED && GATED == 0 && !GROUPED) {
                // 32 columns' loads at a time, then a store a column whose address moves by one addition (64 tokens x 6,144 and 4,096 outputs of
                // 4,096, us: 16 at a time, an address and a test each 12.2 and 9.2, now 11.7 and 8.8)
                if (ok && n_kb > 0) {
                    typedef std::conditional_t<OUT_F32, float, __nv_bfloat16> Out;
                    Out* o = (Out*)out_base + (long long)n0 * ldo + m;
                    const int n_end = m < a_rows ? min(p.bn, p.b_rows - n0) : 0;   // (bn may be an odd multiple of 16: what lies behind is not this tile's)
#pragma unroll 1
                    for (int c0 = 0; c0 < p.bn; c0 += 32) {
                        float v[32];
                        tc_ld16_nowait(lane_addr + c0, v);              // (tensor memory is allocated in multiples of 32 columns)
                        tc_ld16_nowait(lane_addr + c0 + 16, v + 16);
                        tc_wait_ld();
#pragma unroll
                        for (int half = 0; half < 32; half += 16) {
                            if (c0 + half + 16 <= n_end) {
#pragma unroll
                                for (int j = 0; j < 16; ++j, o += ldo) st(o, v[half + j]);
                            } else if (c0 + half < n_end) {
#pragma unroll
                                for (int j = 0; j < 16; ++j, o += ldo)
                                    if (c0 + half + j < n_end) st(o, v[half + j]);
                            }
                        }
                    }
                }
            } else if (ok && n_kb > 0) {
#pragma unroll 1
                for (int c0 = 0; c0 < p.bn; c0 += 16) {
                    float v[16];
                    tc_ld16(lane_addr + c0, v);
                    if (GATED) {
                        float u[16];
                        tc_ld16(lane_addr + p.bn + c0, u);
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = v[j] / (1.0f + expf(-v[j])) * u[j];
                    }
                    if (m < a_rows) {
                        if (!TRANSPOSED) {
                            const int n_left = p.b_rows - (n0 + c0);
                            const long long off = (long long)m * ldo + n0 + c0;
                            if (OUT_F32) {
                                float* o = (float*)out_base + off;
                                if (n_left >= 16 && (off & 3) == 0) {
#pragma unroll
                                    for (int j = 0; j < 16; j += 4) *(float4*)(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                                } else {
                                    for (int j = 0; j < 16 && j < n_left; ++j) o[j] = v[j];
                                }
                            } else {
                                __nv_bfloat16* o = (__nv_bfloat16*)out_base + off;
                                if (n_left >= 16 && (off & 7) == 0) {
                                    uint4 wv[2];
                                    __nv_bfloat162* h = (__nv_bfloat162*)wv;
#pragma unroll
                                    for (int j = 0; j < 8; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                                    *(uint4*)o = wv[0];
                                    *(uint4*)(o + 8) = wv[1];
                                } else {
                                    for (int j = 0; j < 16 && j < n_left; ++j) o[j] = __float2bfloat16_rn(v[j]);
                                }
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const int n = n0 + c0 + j;
                                bool wanted = n < p.b_rows;
                                if constexpr (GROUPED) wanted = wanted && (uses[n >> 5] >> (n & 31) & 1u);
                                if (wanted) {
                                    const long long off = (long long)n * ldo + m;
                                    if (OUT_F32) ((float*)out_base)[off] = v[j];
                                    else ((__nv_bfloat16*)out_base)[off] = __float2bfloat16_rn(v[j]);
                                }
                            }
                        }
                    }
                }
            }
            // this warp has read what it needs of the accumulator: hand the buffer back
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
            if (!ok) break;
        }
    }

    if constexpr (STAGED) {
        if constexpr (JOINED) {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else {
            __syncthreads();
        }
        const int runs = JOINED ? (int)gridDim.z : 1, rank = JOINED ? (int)blockIdx.z : 0, m0 = (int)blockIdx.x * (BM / 2);
        const int n0 = blockIdx.y * p.bn;
        const uint32_t here = smem_u32(tiles);
        __nv_bfloat16* o = (__nv_bfloat16*)p.out;
        const int tokens = min(p.bn, p.b_rows - n0);
        const bool whole = m0 + BM / 2 <= p.a_rows && (p.ldo & 3) == 0 && (reinterpret_cast<size_t>(o) & 7) == 0;
        // V neighbours' gate and up sums a thread, the runs' added in index order
        auto finish = [&](auto neighbours) {
            constexpr int V = decltype(neighbours)::value;
            auto load = [](uint32_t at, float (&v)[V]) {
                if constexpr (V == 4)
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(at) : "memory");
                else
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[0]) : "r"(at) : "memory");
            };
            for (int x = rank * NUM_THREADS + (int)threadIdx.x; x < tokens * (BM / 2 / V); x += runs * NUM_THREADS) {
                const int n = x / (BM / 2 / V), m = x % (BM / 2 / V) * V;
                float g[V], u[V];
#pragma unroll 8
                for (int z = 0; z < runs; ++z) {
                    uint32_t there = here + 4u * (uint32_t)(n * BM + m);
                    float a[V], b[V];
                    if (JOINED) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here + 4u * (uint32_t)(n * BM + m)), "r"(z));
                    load(there, a);
                    load(there + 2u * BM, b);
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        g[i] = z == 0 ? a[i] : g[i] + a[i];
                        u[i] = z == 0 ? b[i] : u[i] + b[i];
                    }
                }
#pragma unroll
                for (int i = 0; i < V; ++i) g[i] = g[i] / (1.0f + expf(-g[i])) * u[i];
                __nv_bfloat16* at = o + (long long)(n0 + n) * p.ldo + m0 + m;
                if (V == 4 && whole) st4(at, g[0], g[V > 1 ? 1 : 0], g[V > 2 ? 2 : 0], g[V > 3 ? 3 : 0]);
                else
#pragma unroll
                    for (int i = 0; i < V; ++i)
                        if (m0 + m + i < p.a_rows) at[i] = __float2bfloat16_rn(g[i]);
            }
        };
        if (!JOINED || runs <= 4) finish(std::integral_constant<int, 4>());
        else finish(std::integral_constant<int, 1>());
        if constexpr (JOINED)
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // (nobody leaves while it is read)
    }

    tc_fence_before();
    __syncthreads();
    if (abort_flag) {
        // Copies that were already issued may still be in flight: give them time
        // to land before this block's shared memory is given up.
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols));
    }
}

template <bool PERSIST, int GATED, bool TRANSPOSED, bool OUT_F32, bool JOINED = false>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
    gemm_tc_block<PERSIST, GATED, TRANSPOSED, OUT_F32, false, JOINED>(map_a, map_b, nullptr, nullptr, p);
}

template <int GATED, bool OUT_F32, bool RANKED>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tc_grouped_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap shared_a, const __grid_constant__ CUtensorMap shared_b, const GroupedParams p) {
    gemm_tc_block<false, GATED, true, OUT_F32, true, false, RANKED>(map_a, map_b, &shared_a, &shared_b, p);
}

// ---- host side ---------------------------------------------------------------
// A [rows, k] bfloat16 matrix, row-major, as a TMA descriptor with boxes of box_rows x 64.
static int make_map(CUtensorMap* map, const void* ptr, int64_t rows, int64_t k, int box_rows) {
    return make_bf16_map(map, ptr, rows, k, box_rows, "gemm_tc");
}

}  // namespace wick

using namespace wick;

// a: [a_total_rows, k] bf16 (the 128-row side), b: [b_total_rows, k] bf16.
// a_rows / b_rows: rows that produce output (for a gated pair: rows of ONE half;
// the other half starts pair_offset rows further).
// gated: 0 none, 1 pair in a, 2 pair in b.  transposed: out[n * ldo + m].
// splits > 1 needs out_f32; partial s lies split_stride elements after s - 1.
// a_static / b_static: that operand is never written by any kernel (weights), so
// the kernel may fetch it before the kernel launched before it has finished.
// a_packed / b_packed: that operand is not row-major but stored as [rows / 128][ceil(k / 64)]
// tiles of 128 rows x 64 columns, each tile contiguous (16 KB), rows and columns padded
// with zeros (a gated pair: each half padded on its own, pair_offset counts padded rows);
// a_total_rows / b_total_rows then count padded rows.  A weight tile then comes from DRAM as
// one contiguous piece instead of 128 pieces of 128 bytes.
// status: device int that receives a non-zero code if a wait inside the kernel gave up.
struct Groups {
    int n, rows, b_rows, top, n_tokens;            // n: 0 where A is one matrix
    long long out;
    const int *tokens, *table;
    // the shared matrix (null: none): packed, with k_shared inner numbers; its rows of B; its result
    const void *shared_a, *shared_b;
    long long shared_a_rows, shared_b_rows;
    int shared_rows, shared_k, shared_pair_offset;
    void* shared_out;
};

// The blocks along z are a cluster.
static int launch_joined(dim3 grid, int smem, const CUtensorMap& map_a, const CUtensorMap& map_b, const GemmParams& p, cudaStream_t s) {
    static bool raised = false;
    if (!raised) {
        WICK_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<false, 3, true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 210 * 1024));
        raised = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = grid.z;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    WICK_CUDA(cudaLaunchKernelEx(&cfg, gemm_tc_kernel<false, 3, true, false, true>, map_a, map_b, p));
    return check_launch("gemm_tc_joined");
}

static int gemm_tc_host(const void* a, long long a_total_rows, int a_rows, const void* b, long long b_total_rows,
                        int b_rows, int k, int bn, int gated, int pair_offset, int transposed, int out_f32,
                        int a_static, int b_static, int a_packed, int b_packed, void* out, long long ldo, int splits, long long split_stride, int max_smem_bytes, int* status,
                        const Groups& G, void* stream) {
    WICK_REQUIRE(bn % 16 == 0 && bn >= 16 && bn <= 256, "gemm_tc: tile width %d must be a multiple of 16 in [16, 256]", bn);
    WICK_REQUIRE(!(gated == 2 && bn > 128) , "gemm_tc: a gated pair needs two accumulators: tile width <= 128");
    WICK_REQUIRE(gated >= 0 && gated <= 3 && splits >= 1, "gemm_tc: bad options");
    WICK_REQUIRE(gated != 3 || transposed, "gemm_tc: the shared-tile pair is built for the transposed output only");
    WICK_REQUIRE(gated != 1 || transposed, "gemm_tc: a pair in the 128-row operand goes with the transposed output");
    WICK_REQUIRE(gated != 2 || !transposed, "gemm_tc: a pair in the narrow operand goes with the row-major output");
    // (a gated pair that shares a tile: the runs of the inner dimension are joined inside the kernel, by a cluster)
    WICK_REQUIRE(splits == 1 || (out_f32 && !gated) || (gated == 3 && !out_f32 && splits <= 8), "gemm_tc: a split inner dimension needs plain float32 partial sums");
    WICK_REQUIRE(a_rows > 0 && b_rows >= 0 && k > 0, "gemm_tc: bad sizes");
    if (b_rows == 0) return 0;
    const int k_blocks = ceil_div(k, BK);
    WICK_REQUIRE(splits <= k_blocks, "gemm_tc: %d splits over %d blocks of the inner dimension", splits, k_blocks);
    const int per_split = ceil_div(k_blocks, splits);
    WICK_REQUIRE((long long)(splits - 1) * per_split < k_blocks, "gemm_tc: a split would be empty");
    CUtensorMap map_a, map_b;
    WICK_REQUIRE(!a_packed || a_total_rows % 128 == 0, "gemm_tc: a packed operand has a multiple of 128 rows");
    WICK_REQUIRE(!b_packed || (b_total_rows % 128 == 0 && (bn <= 128 || bn == 256)), "gemm_tc: a packed narrow operand comes in tiles of 128 rows");
    if (int e = a_packed ? make_map(&map_a, a, a_total_rows * k_blocks, 64, gated == 3 ? BM / 2 : BM)
                         : make_map(&map_a, a, a_total_rows, k, gated == 3 ? BM / 2 : BM)) return e;
    if (int e = b_packed ? make_map(&map_b, b, b_total_rows * k_blocks, 64, bn < 128 ? bn : 128)
                         : make_map(&map_b, b, b_total_rows, k, bn)) return e;
    const int stage_bytes = (gated == 1 ? 2 : 1) * BM * BK * 2 + (gated == 2 ? 2 : 1) * bn * BK * 2;
    int budget = max_smem_bytes > 0 ? max_smem_bytes : 200 * 1024;
    if (budget > 208 * 1024) budget = 208 * 1024;     // 227 KB per block minus the static arrays
    int stages = (budget - 1024) / stage_bytes;
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    if (stages > per_split) stages = per_split < 2 ? 2 : per_split;
    WICK_REQUIRE(stages >= 2, "gemm_tc: %d bytes of shared memory hold fewer than two stages of %d bytes", budget, stage_bytes);
    const bool joined = gated == 3 && splits > 1, staged = gated == 3 && !out_f32 && !G.n;
    if (staged && stages * stage_bytes < bn * BM * 4) stages = ceil_div(bn * BM * 4, stage_bytes);      // (the ring holds the accumulator at the end)
    WICK_REQUIRE(!staged || stages <= MAX_STAGES, "gemm_tc: the tile does not fit the ring");
    const int smem = stages * stage_bytes + 1024;
    GemmParams p;
    p.a_rows = a_rows; p.b_rows = b_rows; p.bn = bn; p.k_blocks = k_blocks; p.k_blocks_per_split = per_split;
    p.stages = stages; p.gated = gated; p.pair_offset = pair_offset; p.transposed = transposed; p.out_f32 = out_f32;
    p.ldo = ldo; p.split_stride = split_stride; p.out = out; p.status = status;
    p.a_static = a_static; p.b_static = b_static; p.a_packed = a_packed; p.b_packed = b_packed;
    p.grid_m = ceil_div(a_rows, gated == 3 ? BM / 2 : BM);
    p.grid_n = ceil_div(b_rows, bn);
    const long long total = (long long)p.grid_m * p.grid_n * splits;
    WICK_REQUIRE(total < (1ll << 30), "gemm_tc: too many tiles");
    p.total_tiles = (int)total;
    if (G.n) {
        GroupedParams g;
        static_cast<GemmParams&>(g) = p;
        g.group_tiles = p.grid_m; g.group_rows = G.rows; g.group_b_rows = G.b_rows; g.group_out = G.out;
        g.top = G.top; g.n_tokens = G.n_tokens; g.tokens = G.tokens; g.table = G.table;
        // Ranked where the blocks of all matrices are more than run at once and the step can name two in five of them at most.  (Layers of
        // 64 experts of 768 x 2,048, eight a token, us as all / ranked: 1 token 33 / 28, 3 52 / 50, 4 67 / 69; 128 experts 1 token
        // 49 / 29, 6 93 / 89, 8 113 / 115, 15 157 / 175; 8 experts of 1,536 x 2,048, two a token, 1 token 24.7 / 25.0.)
        const bool ranked = 5ll * G.n_tokens * G.top <= 2ll * G.n && G.n <= 32 * NAMED_WORDS && (long long)p.grid_m * G.n > 2 * sm_count();
        g.n_groups = G.n;
        g.groups_end = p.grid_m * (ranked ? G.n_tokens * G.top : G.n);
        CUtensorMap shared_a = map_a, shared_b = map_b;
        g.shared_tiles = 0;
        if (G.shared_a) {
            g.shared_k_blocks = ceil_div(G.shared_k, BK);
            g.shared_k_blocks_per_split = ceil_div(g.shared_k_blocks, splits);
            WICK_REQUIRE(G.shared_rows > 0 && G.shared_out && G.shared_a_rows % 128 == 0 && G.shared_b_rows >= G.n_tokens &&
                         (long long)(splits - 1) * g.shared_k_blocks_per_split < g.shared_k_blocks, "gemm_tc: bad shared matrix");
            g.shared_tiles = ceil_div(G.shared_rows, gated == 3 ? BM / 2 : BM);
            g.shared_rows = G.shared_rows; g.shared_pair_offset = G.shared_pair_offset; g.shared_out = G.shared_out;
            g.shared_split_stride = (long long)G.n_tokens * G.shared_rows;
            if (int e = make_map(&shared_a, G.shared_a, G.shared_a_rows * g.shared_k_blocks, 64, gated == 3 ? BM / 2 : BM)) return e;
            if (int e = make_map(&shared_b, G.shared_b, G.shared_b_rows, G.shared_k, bn)) return e;
        }
        WICK_REQUIRE(a_packed && transposed && (gated == 0 || gated == 3) && (out_f32 != 0) == (gated == 0) && !joined, "gemm_tc: grouped products are built for packed matrices, transposed results");
        WICK_REQUIRE((long long)G.n * G.rows <= a_total_rows && G.rows % 128 == 0 && G.n_tokens == b_rows && b_rows <= 256 && G.top > 0, "gemm_tc: bad groups");
        WICK_REQUIRE(total * G.n < (1ll << 30) && splits <= 65535 && p.grid_n <= 65535, "gemm_tc: too many tiles");
        const dim3 grid(g.groups_end + g.shared_tiles, p.grid_n, splits);
        static bool raised = false;
        if (!raised) {
            WICK_CUDA(cudaFuncSetAttribute(gemm_tc_grouped_kernel<3, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 210 * 1024));
            WICK_CUDA(cudaFuncSetAttribute(gemm_tc_grouped_kernel<0, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 210 * 1024));
            WICK_CUDA(cudaFuncSetAttribute(gemm_tc_grouped_kernel<3, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 210 * 1024));
            WICK_CUDA(cudaFuncSetAttribute(gemm_tc_grouped_kernel<0, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 210 * 1024));
            raised = true;
        }
#define WICK_GROUPED(P, F, R) WICK_CUDA(launch(gemm_tc_grouped_kernel<P, F, R>, grid, dim3(NUM_THREADS), (size_t)smem, (cudaStream_t)stream, map_a, map_b, shared_a, shared_b, g))
        if (gated && ranked) WICK_GROUPED(3, false, true);
        else if (gated) WICK_GROUPED(3, false, false);
        else if (ranked) WICK_GROUPED(0, true, true);
        else WICK_GROUPED(0, true, false);
#undef WICK_GROUPED
        return check_launch("gemm_tc_grouped");
    }
    // persistent blocks: as many as can be resident at once (one or two per SM by shared memory)
    const int resident = sm_count() * ((smem + 12 * 1024) * 2 <= 227 * 1024 ? 2 : 1);
    // Decode orientation (and anything that fits at once): one tile per block, so
    // that a block starting while others still stream overlaps their drain.
    // Prompt orientation with more tiles than resident blocks: persistent blocks.
    const bool persistent = !transposed && p.total_tiles > resident;
    WICK_REQUIRE(persistent || (p.grid_n <= 65535 && splits <= 65535), "gemm_tc: grid limit");
    const dim3 grid = persistent ? dim3(resident) : dim3(p.grid_m, p.grid_n, splits);
    if (joined) return launch_joined(dim3(p.grid_m, p.grid_n, splits), smem, map_a, map_b, p, (cudaStream_t)stream);
    // One instantiation per (persistent, pair mode, orientation, output type): a
    // block of a decode step runs for a few microseconds, so the kernel it loads
    // should hold nothing but its own path.
#define WICK_GEMM_CASE(P, G, T, F)                                                                              \
    if (persistent == P && gated == G && (transposed != 0) == T && (out_f32 != 0) == F) {                       \
        static bool raised_##P##G##T##F = false;                                                                 \
        if (!raised_##P##G##T##F) {                                                                              \
            WICK_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<P, G, T, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                           210 * 1024));                                                         \
            raised_##P##G##T##F = true;                                                                          \
        }                                                                                                        \
        WICK_CUDA(launch(gemm_tc_kernel<P, G, T, F>, grid, dim3(NUM_THREADS), (size_t)smem, (cudaStream_t)stream, \
                         map_a, map_b, p));                                                                      \
        return check_launch("gemm_tc");                                                                          \
    }
    WICK_GEMM_CASE(false, 0, true, true) WICK_GEMM_CASE(false, 0, true, false)
    WICK_GEMM_CASE(false, 1, true, true) WICK_GEMM_CASE(false, 1, true, false)
    WICK_GEMM_CASE(false, 3, true, true) WICK_GEMM_CASE(false, 3, true, false)
    WICK_GEMM_CASE(false, 0, false, true) WICK_GEMM_CASE(false, 0, false, false)
    WICK_GEMM_CASE(false, 2, false, true) WICK_GEMM_CASE(false, 2, false, false)
    WICK_GEMM_CASE(true, 0, false, true) WICK_GEMM_CASE(true, 0, false, false)
    WICK_GEMM_CASE(true, 2, false, true) WICK_GEMM_CASE(true, 2, false, false)
#undef WICK_GEMM_CASE
    return fail("gemm_tc: no kernel for pair mode %d with %s output", gated, transposed ? "transposed" : "row-major");
}

WICK_API int wick_gemm_tc(const void* a, long long a_total_rows, int a_rows, const void* b, long long b_total_rows,
                          int b_rows, int k, int bn, int gated, int pair_offset, int transposed, int out_f32,
                          int a_static, int b_static, int a_packed, int b_packed, void* out, long long ldo, int splits, long long split_stride, int max_smem_bytes, int* status,
                          void* stream) {
    const Groups none = {};
    return gemm_tc_host(a, a_total_rows, a_rows, b, b_total_rows, b_rows, k, bn, gated, pair_offset, transposed, out_f32, a_static, b_static,
                        a_packed, b_packed, out, ldo, splits, split_stride, max_smem_bytes, status, none, stream);
}

// Few tokens (at most 256) times the matrices of the experts that a table names for their ids: a holds n_groups packed matrices
// of group_rows padded rows one after the other; a gated pair (silu(g) * u, bfloat16 out) or plain (float32 out).  Matrix e's
// results lie at out + e * n_tokens * a_rows, token by token; only those of tokens whose id names e are written.  splits: runs of the
// inner dimension, left as partial sums n_groups * n_tokens * a_rows apart (not for gated pairs).
// shared_a (or null): a packed matrix (of a pair, the second half shared_pair_offset rows on) that every token uses, times the n_tokens rows
// of shared_b, in the same launch; result as for one group, at shared_out.
// per_group_b: matrix e is multiplied with rows e * n_tokens .. of b, otherwise all of them with the first n_tokens rows.
WICK_API int wick_gemm_tc_grouped(const void* a, int n_groups, int group_rows, int a_rows, const void* b, long long b_total_rows,
                                  int per_group_b, int n_tokens, int k, int bn, int gated, int pair_offset, void* out,
                                  const int* tokens, const int* table, int top, int splits, const void* shared_a, long long shared_a_rows,
                                  const void* shared_b, int shared_rows, int shared_k, int shared_pair_offset, void* shared_out,
                                  int max_smem_bytes, int* status, void* stream) {
    WICK_REQUIRE(n_groups > 0 && tokens && table, "gemm_tc: bad groups");
    WICK_REQUIRE(bn >= n_tokens, "gemm_tc: a grouped product takes its tokens in one tile");
    const Groups G = {n_groups, group_rows, per_group_b ? n_tokens : 0, top, n_tokens, (long long)n_tokens * a_rows, tokens, table,
                      shared_a, shared_b, shared_a_rows, n_tokens, shared_rows, shared_k, shared_pair_offset, shared_out};
    return gemm_tc_host(a, (long long)n_groups * group_rows, a_rows, b, b_total_rows, n_tokens, k, bn, gated ? 3 : 0, pair_offset, 1, gated ? 0 : 1,
                        1, 0, 1, 0, out, a_rows, splits, gated ? 0 : (long long)n_groups * n_tokens * a_rows, max_smem_bytes, status, G, stream);
}
