// Causal attention of a step's new tokens over the paged cache on the 5th-
// generation tensor cores (tcgen05), bfloat16, head sizes 64 and 128.
//
// The 128 rows of a tile are query heads of one key head times consecutive tokens: as many heads as fill it with whole
// tokens, i.e. the largest power of two that divides their number (4 heads to a key head: 4 x 32 tokens; 5 or 1: 1 x 128; one
// TMA box of heads x tokens either way).  A block runs two streams over blocks of 128 keys (two cache pages),
// each with its own scores and its own result in tensor memory and four softmax warps:
//   * two tiles of neighbouring tokens over all key blocks (a key or value tile is read twice), or
//   * where the step is too small for that to fill the device, or the second tile has no tokens,
//     ONE tile, even key blocks in one stream and odd ones in the other, joined at the end.
//   * a producer thread fetches the query rows once and the key and value pages
//     through a ring of five tiles (TMA, 64 x 64 boxes, 128-byte swizzle);
//   * an issuing thread alternates between the streams: O += P V of one (the values are the
//     MN-major operand: their rows are keys), the scores S = Q K^T of its next key block, then
//     the other stream's, so that one stream's softmax runs beside the other's products;
//   * a softmax thread owns a row of its stream: it reads 128 scores from tensor memory, scales,
//     masks (a key is visible up to the token's own position), and writes P as pairs of bfloat16
//     over the scores, where the second product takes it from.  The next scores overwrite P:
//     tensor-core instructions of one thread execute in order.  That a stream's scores of step t + 1
//     are complete therefore also says that its product of step t is.
// A block an SM works through its items one behind the other: the next item's tiles and scores are under way during the
// last one's epilogue.
// What bounds it: a tile and key block take the tensor core 1,024 clocks (16 instructions of 64) and the
// exponentials as many; a stream's chain of softmax (1,830 clocks), product, scores and the waits between them takes ~3,400 clocks for
// both streams' blocks.  Before (a tile of one head's rows a block, two threads a row, one lane issuing) / now, us alone, one behind the
// other: 2,048 tokens, 32 heads over 8 67 / 42, 8,192 tokens 654 / 517 (at the power cap); 16 prompts of 64 to 2,048 tokens, 40 over 8
// 472 / 355; 1,419 tokens behind 3,100 118 / 94; 8 x 1,024, 64 over 8 336 / 190.  Short prompts have a thread for 128 scores where they had
// two: 64 tokens, 32 over 8 5.8 / 6.2, 200 7.2 / 7.4, 400 9.8 / 9.4, 16 over 4 400 9.0 / 9.3, 1,000 14.4 / 14.9; a whole step of 64 tokens is 2 to 5 %
// shorter than before all the same, one of 200 or 400 0.3 to 0.7 % longer.
// O and the sum are scaled by a maximum that follows the true running maximum
// lazily: only when a block's maximum exceeds it by more than 8 (in units of
// log2 e) is O rescaled in tensor memory, so that after the first blocks of a row
// the rescaling is rare; probabilities stay below 2^8, which bfloat16 and
// float32 hold without loss of relative precision.
// Value rows beyond the cached length are zeroed in shared memory before they
// are multiplied (their weight is zero, but the row may hold anything).
// The EXTRA form also sees the blocks of `block` positions that lie wholly before a row's
// window, each as one key and value (tiles of 64 blocks a sequence, laid out like cache
// pages; their key blocks come before the window's), soft-caps the scores and multiplies
// the result by a number per token and head.
// Work items are dealt longest first (see Finder): neighbouring block indexes are the key heads of one item.  Steps of several
// sequences whose page table has up to eight pages deal them in index order.
// Every wait is bounded and reports through the status word.
// Formulas: wick src/model.rs:520-553.  The plain forms of this computation are
// attn_prompt_mma_kernel (attn_prompt_mma.cu) and attn_prompt_kernel (attn.cu).
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "sm100.cuh"
#include "tcgen05.cuh"

#ifndef WICK_HD
#error "compile with -DWICK_HD=<head_dim>"
#endif

namespace wick {
namespace prompttc {

constexpr bool SUPPORTED = WICK_HD == 64 || WICK_HD == 128;
constexpr int HD = SUPPORTED ? WICK_HD : 64;           // other head sizes: the entry point refuses, the kernel is never launched
constexpr int BQ = 128;                                // rows of a tile
constexpr int BK = 128;                                // keys of an inner step (two pages)
constexpr int PANELS = HD / 64;                        // 64-column panels of a head row
constexpr int PANEL_BYTES = 128 * 128;                 // 128 rows of 128 bytes
constexpr int TILE_BYTES = PANELS * PANEL_BYTES;       // a tile of Q, or one block of keys or of values
constexpr int LONG = 9;                                // key blocks of an item from which on its softmax is written out (8,192 tokens: 537 us looped, 453)
constexpr int P_FIRST = 64;                            // keys of a block whose probabilities the product begins with
constexpr int NSLOT = 5;                               // key / value tiles in flight
constexpr int MAX_ITEMS = 16;                          // work items of a block
// A work item: the sequence (-1: none), its place, new and cached tokens; the item's first token; the heads; key blocks.
struct Item {
    int b, tok0, q_len, start, q0, kvh, head0;
    int jb0, n_pool, n_blk;                            // first block of keys; of the item's n_blk, those of blocks of positions
    int split;                                         // one tile, its key blocks dealt to both streams
    // Tiles come through the ring in the order in which the issuing thread uses them: K0 V0 K1 V1 ..., or, split,
    // K0 K1 V0 K2 V1 K3 ... V(n-2) V(n-1): an item's 2 n_blk tiles, and the place of block j's values among them.
    __device__ __forceinline__ int place_v(int j) const { return split ? min(2 * j + 2, 2 * n_blk - 1) : 2 * j + 1; }
};
// The key blocks that a tile multiplies: those before `pool`, and those from `from` up to `to`.
struct Seen {
    int pool, from, to;
    __device__ __forceinline__ bool has(int j) const { return j < pool || (j >= from && j < to); }
    __device__ __forceinline__ int first() const { return pool > 0 ? 0 : from; }
};
constexpr int GUARDED = 4;                             // (of a form of the issuing loop, beside how far it is unrolled)
// Behind the tiles in shared memory (which begins on a multiple of 1,024 bytes, and has no room for a shift):
struct Shared {
    float ml[2][2][BQ];                                // the streams' maxima and sums, where they share rows
    uint64_t q_full, q_empty, full[NSLOT], empty[NSLOT], s_full[2], p_full[2][2], o_full[2], o_empty[2], join, joined;
    Item items[MAX_ITEMS];
    uint32_t tmem_slot;
    int abort_flag;
};
constexpr int SMEM_BYTES = (2 + NSLOT) * TILE_BYTES + (int)sizeof(Shared);
static_assert(SMEM_BYTES <= 227 * 1024, "a block's shared memory");
constexpr int THREADS = 320;                           // warp 0: TMA, warp 1: MMA + tensor memory, warps 2-5 and 6-9: softmax
constexpr uint32_t TMEM_COLS = 512;                    // S of both streams | O of both; P (bfloat16 pairs) takes the place of
constexpr uint32_t COL_S = 0, COL_O = 2 * BK;          // the first 64 columns of the S it was computed from
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_ld32_nowait(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tc_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The issuing thread is one thread: what it computes per instruction is what limits
// the rate of small products.  A shared-memory descriptor is therefore kept as two
// 32-bit halves: the high half is a constant, the low half (start address in 16-byte
// units, leading offset) moves by one addition per instruction.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo_bytes) {
    return ((addr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
// stride offset 1024 bytes (8 rows of 128 bytes), descriptor version 1 (bit 46), 128-byte swizzle (bits 61-63)
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);

// D (tensor memory) (+)= A (shared memory) * B (shared memory)
template <int ACC>
__device__ __forceinline__ void mma_ss(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(DESC_HI), "r"(idesc), "n"(ACC)
        : "memory");
}
// D (tensor memory) (+)= A (tensor memory: 128 lanes x 8 columns of bfloat16 pairs) * B (shared memory)
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc, int acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(DESC_HI), "r"(idesc), "r"(acc)
        : "memory");
}
template <int I, int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<I + 1, N>(f);
    }
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint64_t* bar, void* dst, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
// The softmax warps are bound by the number of instructions they issue: two products-and-sums,
// two sums, or a maximum of three per instruction where sm_100 has one.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {      // a * b + c, each half rounded once
    uint64_t ra, rb, rc, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t ra, rb, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
    return d;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t ra, rb, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
    return d;
}
// tanh(z) = z (c0 + c1 z^2 + c2 z^4 + c3 z^6 + c4 z^8) for |z| <= 0.75, off by at most 4.2e-7 (the interpolant of tanh(z) / z, as a
// function of z^2, at the Chebyshev points of the interval, fitted by least squares).
constexpr float TANH_SMALL = 0.75f, TANH_C0 = 0.99999945f, TANH_C1 = -0.33328349f, TANH_C2 = 0.13259838f, TANH_C3 = -0.050080256f,
                TANH_C4 = 0.012950745f;

// Descriptors.  A k-major operand (Q, K): rows of 128 bytes, eight-row groups 1024
// bytes apart, the leading offset unused (1).  The MN-major operand (V): rows are
// keys, a row holds 64 consecutive dims in 128 bytes, eight rows make a 1024-byte
// group, and the next 64 dims lie one panel (the leading offset) further.

// First key that the query at position p sees: mask 0 every earlier key, 1 those of p's own block of `size`
// positions (blocks counted from position 0), 2 the last `size` positions.
__device__ __forceinline__ int first_visible_key(int p, int mask, int size) {
    return mask == 1 ? p / size * size : (mask == 2 ? max(0, p - size + 1) : 0);
}

// What the EXTRA form does besides.
struct TcExtra {
    int pool_tiles, block;         // tile i of sequence b is page b * pool_tiles + i of the blocks' array; block 0: there are none
    float cap;                     // of the scores; 0: none
    const float* gate;             // float32 [n, heads] or null: a factor of the result
};
__device__ __forceinline__ int blocks_seen(int p, int window, int block) { return block > 0 && p + 1 > window ? (p + 1 - window) / block : 0; }
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Work items of R tokens, longest first: all items of the step in falling order of the key block that their first
// token lies in (items of one sequence that share it, and sequences, in index order); this finds the item at place `rank`.
// A warp takes the sequences 32 at a time (the first 32 are kept in registers); the key block is found by bisection over counts
// (9 steps for 40,960 positions; one sequence needs none).  Not ordered: all items in index order.
struct Finder {
    const int *cu_seqlens, *start_arr;
    int n_seqs, R, tok0, q_len, start, top;                        // (lane l: sequence l; top: no item lies in this key block or beyond)
    bool ordered;
    __device__ __forceinline__ Finder(const int* cu, const int* st, int n, int r, bool o) : cu_seqlens(cu), start_arr(st), n_seqs(n), R(r), ordered(o) {
        const int s = threadIdx.x & 31;
        tok0 = s < n ? cu[s] : 0;
        q_len = s < n ? cu[s + 1] - tok0 : 0;
        start = s < n ? st[s] : 0;
        if (!ordered) return;
        int t = (start + q_len) / BK + 1;
#pragma unroll 1
        for (int i = s + 32; i < n; i += 32) t = max(t, (st[i] + cu[i + 1] - cu[i]) / BK + 1);
        top = (int)__reduce_max_sync(0xffffffffu, t);
    }
    // items of this lane's sequence of the chunk at s0, and those of them whose first token lies in key block k or a later one
    __device__ __forceinline__ int items(int s0) const {
        const int s = s0 + (int)(threadIdx.x & 31), n = s0 == 0 ? q_len : (s < n_seqs ? cu_seqlens[s + 1] - cu_seqlens[s] : 0);
        return (n + R - 1) / R;
    }
    __device__ __forceinline__ int from(int s0, int n, int k) const {
        const int s = s0 + (int)(threadIdx.x & 31), before = k * BK - (s0 == 0 ? start : (s < n_seqs ? start_arr[s] : 0));
        return before > 0 ? max(0, n - (before + R - 1) / R) : n;
    }
    __device__ __forceinline__ int count(int k) const {
        int c = 0;
#pragma unroll 1
        for (int s0 = 0; s0 < n_seqs; s0 += 32) c += from(s0, items(s0), k);
        return (int)__reduce_add_sync(0xffffffffu, c);
    }
    // (every lane gets the item)
    __device__ __forceinline__ Item find(int rank) const {
        Item it;
        it.b = -1;
        int lo = 0, hi = top, above = 0;
        if (n_seqs == 1) {
            const int n = (__shfl_sync(0xffffffffu, q_len, 0) + R - 1) / R;
            if (rank < n) it.b = 0, it.q0 = (n - 1 - rank) * R;
        } else if (!ordered || count(0) > rank) {
#pragma unroll 1
            while (ordered && hi - lo > 1) {                       // count(lo) > rank >= count(hi) = above
                const int mid = (lo + hi) >> 1, c = count(mid);
                if (c > rank) lo = mid;
                else hi = mid, above = c;
            }
            int left = rank - above;                               // place among the items of key block lo
#pragma unroll 1
            for (int s0 = 0; s0 < n_seqs; s0 += 32) {
                const int all = items(s0), later = ordered ? from(s0, all, lo + 1) : 0, n = ordered ? from(s0, all, lo) - later : all;
                int upto = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, upto, o);
                    if ((int)(threadIdx.x & 31) >= o) upto += t;
                }
                const int total = __shfl_sync(0xffffffffu, upto, 31);
                if (left < total) {
                    const int l = __ffs(__ballot_sync(0xffffffffu, left < upto)) - 1;
                    it.b = s0 + l;                                 // (all - later - n: the sequence's first item in lo)
                    it.q0 = (__shfl_sync(0xffffffffu, all - later - upto, l) + left) * R;
                    break;
                }
                left -= total;
            }
        }
        if (it.b >= 0) {
            if (it.b < 32) {
                it.tok0 = __shfl_sync(0xffffffffu, tok0, it.b);
                it.q_len = __shfl_sync(0xffffffffu, q_len, it.b);
                it.start = __shfl_sync(0xffffffffu, start, it.b);
            } else {
                it.tok0 = cu_seqlens[it.b], it.q_len = cu_seqlens[it.b + 1] - it.tok0, it.start = start_arr[it.b];
            }
        }
        return it;
    }
};

// What follows from an item's place: `column` counts the step's tiles of heads.
__device__ __forceinline__ void complete(Item& it, int column, int per_kv, int gs, int T, int tiles, int mask, int mask_size, int block) {
    const int kv_len = it.start + it.q_len;
    it.kvh = per_kv == 1 ? column : column / per_kv;                // (a group of more than 128 heads: several tiles of heads)
    it.head0 = column * gs;
    it.split = tiles == 1 || it.q0 + T >= it.q_len;
    const int last_key = min(it.start + it.q0 + (it.split ? T : 2 * T) - 1, kv_len - 1);   // the last position any row of the item may see
    // With a mask the first block of keys is the one that holds the first row's first visible key (the first
    // visible key grows with the position); blocks are counted from there, j = 0 .. n_blk - 1, everywhere below.
    it.jb0 = first_visible_key(it.start + it.q0, mask, mask_size) / BK;
    // (EXTRA: the first n_pool key blocks hold blocks of positions; block j >= n_pool holds the keys from (j - n_pool + jb0) BK on)
    it.n_pool = block > 0 ? (blocks_seen(last_key, mask_size, block) + BK - 1) / BK : 0;
    it.n_blk = last_key / BK + 1 - it.jb0 + it.n_pool;
}

// GUARD: two tiles an item, of more tokens together than a key block has keys.  A tile then multiplies no block that none of its rows sees
// a key of: such a block weighs nothing, but a value that is infinite or no number would show in rows that do not see it.  (A kernel
// of its own: with this in one kernel a step of a short prompt, which meets the code once a layer, took 2 us longer a layer.)
// LONGS: there can be items of LONG key blocks and more.  (Without them the code is 51 KB instead of 69: 400 tokens, 32 heads over 8
// 9.9 us, now 9.5; 200 tokens 7.9 and 7.5; a step of 200 tokens on 6 8B layers 1,238 and 1,227, of 400 on 4 small ones 742 and 732.)
template <bool EXTRA, bool GUARD, bool LONGS>
__global__ void __launch_bounds__(THREADS, 1)
attn_prompt_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map,
                      bf16* __restrict__ out, const int* __restrict__ cu_seqlens, int n_seqs,
                      const int* __restrict__ start_arr,
                      const int* __restrict__ page_table, int table_width, int n_heads, int n_kv, int gs, int T, int columns, int per_kv, int tiles, int n_items, int ordered,
                      float scale, int* status, int mask, int mask_size, const float* __restrict__ sink,
                      const __grid_constant__ CUtensorMap pool_map, const TcExtra X) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* q_s = smem_raw;                                       // two tiles of queries
    uint8_t* kv_s = q_s + 2 * TILE_BYTES;                          // NSLOT tiles: keys and values of the blocks in flight
    Shared& sh = *reinterpret_cast<Shared*>(kv_s + NSLOT * TILE_BYTES);
    volatile int* abort_flag = &sh.abort_flag;

    pdl_trigger();
    if (smem_u32(smem_raw) & 1023) {                               // (cannot be, see Shared)
        if (threadIdx.x == 0) atomicCAS(status, 0, 7);
        pdl_wait();
        return;
    }
    // (the step's description is written by the host before the step: no kernel produces it)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Item k of the block is the one at place(k) of all, the key heads of one item side by side, in falling order of length, dealt
    // to and fro over the blocks.
    auto place = [&](int k) { return k * (int)gridDim.x + (k & 1 ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x); };

    if (threadIdx.x == 0) {
        sh.abort_flag = 0;
        mbar_init(&sh.q_full, 1), mbar_init(&sh.q_empty, 1);
        for (int i = 0; i < NSLOT; ++i) mbar_init(&sh.full[i], 1), mbar_init(&sh.empty[i], 1);
        // Every waiter below sees every phase of the barrier it waits on, so that a parity is never ambiguous
        // (full as seen by the softmax warps: see there).
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.s_full[i], 1), mbar_init(&sh.o_full[i], 1), mbar_init(&sh.o_empty[i], 4);
            mbar_init(&sh.p_full[i][0], 4), mbar_init(&sh.p_full[i][1], 4);
        }
        mbar_init(&sh.join, 8), mbar_init(&sh.joined, 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0 && lane < 2 + (int)EXTRA) {
        const CUtensorMap* map = lane == 0 ? &q_map : (lane == 1 ? &kv_map : &pool_map);
        asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    {
        const Finder finder(cu_seqlens, start_arr, n_seqs, T * tiles, ordered != 0);
#pragma unroll 1
        for (int k = warp; k < MAX_ITEMS; k += THREADS / 32) {      // (a warp each, up to the first that is none)
            const int at = place(k);
            Item it;
            it.b = -1;
            const int rank = at / columns;
            if (rank < n_items) it = finder.find(rank);
            if (it.b >= 0) complete(it, at - rank * columns, per_kv, gs, T, tiles, mask, mask_size, EXTRA ? X.block : 0);
            if (lane == 0) sh.items[k] = it;
            if (it.b < 0) break;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_slot;
    // (item k, if there is one; the items of a block come in order, and none follows the first that is none)
    auto any = [&](int k) { return k < MAX_ITEMS && sh.items[k].b >= 0; };

    if (warp < 2) {
        if (warp == 0) {
            // ---------------- producer ----------------
            // A lane holds a page number of each of two runs of 32 (read ahead, so that a copy never waits for one).
            const bool one = elect_one();
            bool ok = true;
            int slot = 0, turn = 0;                                // of the ring
#pragma unroll 1
            for (int k = 0; ok && any(k); ++k) {
                const Item& w = sh.items[k];
                const int n_blk = w.n_blk, n_pool = w.n_pool, kvh = w.kvh;
                const bool split = w.split;
                auto pages = [&](int run) {
                    const int at = 2 * w.jb0 + run * 32 + lane;
                    return at < table_width ? page_table[(int64_t)w.b * table_width + at] : 0;
                };
                int even = pages(0), odd = pages(1);
                if (k == 0) pdl_wait();                            // q and the cache come from the kernel before this one
                else ok = __all_sync(0xffffffffu, mbar_wait(&sh.q_empty, (k - 1) & 1, abort_flag, status, 7));
                if (!ok) break;
                if (one) {
                    const int n_q = w.split ? 1 : 2;
                    mbar_expect_tx(&sh.q_full, n_q * TILE_BYTES);
#pragma unroll 1
                    for (int i = 0; i < n_q; ++i)
                        for (int pn = 0; pn < PANELS; ++pn)
                            tma_load_3d(&q_map, &sh.q_full, q_s + i * TILE_BYTES + pn * PANEL_BYTES, pn * 64, w.head0, w.tok0 + w.q0 + i * T);
                }
#pragma unroll 1
                for (int i = 0; i < 2 * n_blk; ++i) {
                    const bool last = split && i == 2 * n_blk - 1;    // (split: the last two tiles are values, or the first keys and values)
                    const int is_v = split ? (last || (i > 0 && !(i & 1))) : (i & 1);
                    const int j = last ? n_blk - 1 : (split ? (is_v ? (i - 2) >> 1 : (i + 1) >> 1) : i >> 1);
                    if (turn > 0 && !__all_sync(0xffffffffu, mbar_wait(&sh.empty[slot], (turn - 1) & 1, abort_flag, status, 7))) {
                        ok = false;
                        break;
                    }
                    const bool pooled = EXTRA && j < n_pool;
                    const int at = 2 * (j - n_pool);             // the key block's first page of those from 2 jb0 on
                    int page0, page1;
                    if (pooled) {
                        page0 = w.b * X.pool_tiles + min(2 * j, X.pool_tiles - 1);
                        page1 = w.b * X.pool_tiles + min(2 * j + 1, X.pool_tiles - 1);
                    } else {
                        const int held = (at >> 5) & 1 ? odd : even;
                        page0 = __shfl_sync(0xffffffffu, held, at & 31);
                        page1 = __shfl_sync(0xffffffffu, held, (at + 1) & 31);
                        if (is_v && at >= 32 && (at & 31) == 0) {  // (keys and values have left the run before)
                            if ((at >> 5) & 1) even = pages((at >> 5) + 1);
                            else odd = pages((at >> 5) + 1);
                        }
                    }
                    if (one) {
                        mbar_expect_tx(&sh.full[slot], TILE_BYTES);
                        uint8_t* dst = kv_s + slot * TILE_BYTES;
#pragma unroll 1
                        for (int h = 0; h < 2; ++h)
                            for (int pn = 0; pn < PANELS; ++pn)
                                tma_load_2d(pooled ? &pool_map : &kv_map, &sh.full[slot], dst + pn * PANEL_BYTES + h * (kPage * 128), pn * 64,
                                            (((h ? page1 : page0) * 2 + is_v) * n_kv + kvh) * kPage);
                    }
                    if (++slot == NSLOT) slot = 0, ++turn;
                    __syncwarp();
                }
            }
        } else {
            // ---------------- MMA issuer ----------------
            // The whole warp walks through the steps and one elected lane issues.  (Issued in a branch of one lane, beside busy softmax
            // warps, an instruction took 86 to 146 clocks instead of the tensor core's 64.)
            // kind::f16, bfloat16 operands, float32 accumulator, M = 128
            const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BK >> 3) << 17) | ((uint32_t)(BQ >> 4) << 24);
            const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(BQ >> 4) << 24);
            const uint32_t q_lo0 = desc_lo(smem_u32(q_s), 16);
            const uint32_t k_lo0 = desc_lo(smem_u32(kv_s), 16), v_lo0 = desc_lo(smem_u32(kv_s), PANEL_BYTES);
            const bool one = elect_one();
            bool ok = true;
            int slot = 0, turn = 0;                                // of the ring
            int steps0 = 0, steps1 = 0, uses0 = 0, uses1 = 0;      // steps and items of each stream so far
            // the next tile of the ring, when it has come
            auto take = [&](int& at) {
                at = slot;
                const bool here = __all_sync(0xffffffffu, mbar_wait(&sh.full[slot], turn & 1, abort_flag, status, 7));
                if (++slot == NSLOT) slot = 0, ++turn;
                return here;
            };
#pragma unroll 1
            for (int k = 0; ok && any(k); ++k) {
                const Item& w = sh.items[k];
                const int n_blk = w.n_blk;
                const bool split = w.split;
                auto block_of = [&](int s, int t) { return split ? 2 * t + s : t; };
                const bool guard = GUARD && !split;
                auto seen_by = [&](int s) {
                    const int first = w.start + w.q0 + s * T, last = min(first + T, w.start + w.q_len) - 1, before = w.n_pool - w.jb0;
                    return Seen{EXTRA ? (blocks_seen(last, mask_size, X.block) + BK - 1) / BK : 0,
                                before + first_visible_key(first, mask, mask_size) / BK, before + last / BK + 1};
                };
                Seen seen0 = {}, seen1 = {};
                if (guard) seen0 = seen_by(0), seen1 = seen_by(1);
                int k_at = 0, v_at = 0;                            // where the keys and values at hand lie (both streams read a tile, or one)
                ok = __all_sync(0xffffffffu, mbar_wait(&sh.q_full, k & 1, abort_flag, status, 7));
                // Turn t of stream s: the product of its step t, the scores of step t + 1.  Long items take the form in which the streams
                // are told apart when the kernel is built (8,192 tokens: 537 us in the other, 453), short ones the shorter code.
                auto turn = [&](auto form, int s, int t) {
                    constexpr int UNROLL = decltype(form)::value & 3;
                    constexpr bool SEEN_ONLY = decltype(form)::value >= GUARDED;
                    const int steps = s == 0 ? steps0 : steps1, uses = s == 0 ? uses0 : uses1;
                    const bool more = block_of(s, t + 1) < n_blk;
                    if (block_of(s, t) >= n_blk) return;
                    if (t >= 0) {
                        if (split || s == 0) ok = take(v_at);
                        // (the result of the stream's item before has been read)
                        if (ok && t == 0 && uses > 0) ok = __all_sync(0xffffffffu, mbar_wait(&sh.o_empty[s], (uses - 1) & 1, abort_flag, status, 7));
                        const uint32_t v_lo = v_lo0 + v_at * (TILE_BYTES >> 4), d = tmem + COL_O + s * HD, pa = tmem + COL_S + s * BK;
                        bool go = one;
                        int begun = t;                             // (0: the stream's first product of the item)
                        if constexpr (SEEN_ONLY) {
                            const Seen seen = s == 0 ? seen0 : seen1;
                            go = one && seen.has(t);
                            begun = t - seen.first();
                        }
#pragma unroll UNROLL
                        for (int part = 0; part < 2; ++part) {
                            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&sh.p_full[s][part], steps & 1, abort_flag, status, 7));
                            if (!ok) break;
                            tc_fence_after();
                            const uint32_t pp = pa + part * (P_FIRST / 2), vp = v_lo + part * (P_FIRST / 16) * (2048 >> 4);
                            if (go) {
                                mma_ts(d, pp, vp, idesc_o, begun > 0 || part > 0);
                                static_for<1, P_FIRST / 16>([&](auto ks) { mma_ts(d, pp + (int)ks * 8, vp + (int)ks * (2048 >> 4), idesc_o, 1); });
                            }
                        }
                        if (!ok) return;
                        if (one) {
                            if (split || s == 1) tc_commit(&sh.empty[v_at]);   // a tile is free behind its last reader
                            if (!more) tc_commit(&sh.o_full[s]);
                        }
                        if (s == 0) ++steps0, uses0 += more ? 0 : 1;
                        else ++steps1, uses1 += more ? 0 : 1;
                    }
                    if (more) {
                        if (split || s == 0) ok = take(k_at);
                        if (!ok) return;
                        tc_fence_after();
                        const uint32_t k_lo = k_lo0 + k_at * (TILE_BYTES >> 4), q_lo = q_lo0 + (split ? 0 : s * (TILE_BYTES >> 4));
                        const uint32_t d = tmem + COL_S + s * BK;
                        if (one) {
                            static_for<0, HD / 16>([&](auto ks) {
                                constexpr uint32_t off = (((int)ks >> 2) * PANEL_BYTES + ((int)ks & 3) * 32) >> 4;
                                mma_ss<((int)ks > 0)>(d, q_lo + off, k_lo + off, idesc_s);
                            });
                            tc_commit(&sh.s_full[s]);
                            if (split || s == 1) {
                                tc_commit(&sh.empty[k_at]);
                                if (block_of(s, t + 1) == n_blk - 1) tc_commit(&sh.q_empty);   // (the item's last scores)
                            }
                        }
                    }
                    __syncwarp();
                };
                auto looped = [&](auto form, int from, int to) {
#pragma unroll 1
                    for (int i = 2 * from; ok && i < 2 * to; ++i) turn(form, i & 1, i >> 1);
                };
                auto written_out = [&](int from, int to) {
#pragma unroll 1
                    for (int t = from; ok && t < to; ++t) {
                        turn(std::integral_constant<int, 2>{}, 0, t);
                        if (ok) turn(std::integral_constant<int, 2>{}, 1, t);
                    }
                };
                const int turns = split ? (n_blk + 1) / 2 : n_blk;
                int lo = -1, hi = turns;
                if (GUARD && guard) {
                    // (between the last block that either tile begins with and the first that either no longer sees: as without)
                    lo = max(seen0.from, seen1.from) + 1, hi = max(lo, min(seen0.to, seen1.to));
                    looped(std::integral_constant<int, GUARDED + 1>{}, -1, lo);
                }
                if (LONGS && n_blk >= LONG) written_out(lo, hi);
                else looped(std::integral_constant<int, 1>{}, lo, hi);
                if (GUARD && guard) looped(std::integral_constant<int, GUARDED + 1>{}, hi, turns);
            }
        }
    } else {
        // ---------------- softmax: a row per thread ----------------
        // (a warp reads the 32 lanes of tensor memory given by its index modulo 4)
        pdl_wait();                                                 // (the result's and the gate's memory may be in use until then)
        const int quad = warp & 3, s = (warp - 2) >> 2;             // s: the stream
        const int r = quad * 32 + lane, row_tok = r / gs, row_head = r % gs;    // (a tile is T tokens of gs heads, T gs = 128)
        const bool capped = EXTRA && X.cap > 0.f;
        const float sl2 = capped ? 1.0f : scale * 1.4426950408889634f;   // (a capped score comes in units of log2 e)
        const float cap2 = EXTRA ? X.cap * 1.4426950408889634f : 0.f, z_of_s = capped ? scale / X.cap : 0.f,
                    two_s = 2.0f * 1.4426950408889634f * z_of_s;
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
        const uint32_t s_addr = lane_base + COL_S + s * BK, o_addr = lane_base + COL_O + s * HD;
        bool ok = true;
        int base = 0, step = 0, uses[2] = {0, 0}, joins = 0;        // tiles of earlier items; this stream's steps, both streams' items, joins so far
#pragma unroll 1
        for (int k = 0; ok && any(k); ++k) {
            const Item& w = sh.items[k];
            const int n_blk = w.n_blk, kv_len = w.start + w.q_len, n_pool = w.n_pool, jw = w.jb0 - n_pool;
            const bool split = w.split;
            const int tok = w.q0 + (split ? 0 : s * T) + row_tok, head = w.head0 + row_head;   // token (of the sequence) and head of the row
            const bool store = tok < w.q_len;                       // (rows of tokens beyond the sequence's end are left out)
            const int limit = min(w.start + tok, kv_len - 1);       // last visible key position
            const int vis = first_visible_key(limit, mask, mask_size);  // first visible key position
            const int n_seen = EXTRA ? blocks_seen(limit, mask_size, X.block) : 0;
            const float sink2 = sink ? sink[head] * 1.4426950408889634f : -INFINITY;   // a score without a value
            // m: the maximum (in units of log2 e) that O and l are scaled by.  It follows
            // the true running maximum lazily; l: the row's sum.
            // (a sink: the scaling maximum starts there, and its share joins the row's sum at the end)
            float m = sink2, l = 0.f;
            int t = 0;
#pragma unroll 1
            for (int j = split ? s : 0; j < n_blk; j += split ? 2 : 1, ++t) {
                ok = __all_sync(0xffffffffu, mbar_wait(&sh.s_full[s], step & 1, abort_flag, status, 7));
                if (!ok) break;
                ++step;
                tc_fence_after();
                const bool pooled = EXTRA && j < n_pool;
                const int key0 = (pooled ? j : j + jw) * BK;
                const int last = pooled ? n_seen - 1 : limit, first_key = pooled ? 0 : vis;
                // Twice over the scores: masks where there are any and the row's maximum (in two passes of their own 1 to 5 % of the kernel's time
                // more: 400 tokens, 40 heads over 8 12.8 us, now 12.5; 300 with a cap and blocks 16.3 and 15.2), the probabilities, which take the place of scores
                // already read.  In loops, except in long items: an item of a short prompt meets this code once, and each 128 bytes of it come
                // from memory where weights have passed through the L2 cache since the layer before (the whole written out, 110 KB of code
                // instead of 72: a prompt of 100 tokens took 7 us longer a layer).
                const bool changed = capped || __any_sync(0xffffffffu, key0 + BK - 1 > last || key0 < first_key);
                auto cap = [&](float* v) {                                // of 32 scores
                    // cap tanh(z), z = s / cap: by a polynomial where all of the warp's |z| are small (two products and sums an
                    // instruction), else as cap (1 - 2 / (1 + exp(2 z))), whose two special functions a score would bound the block.
                    float big = 0.f;
#pragma unroll
                    for (int i = 0; i < 32; i += 2) big = max3(big, fabsf(v[i]), fabsf(v[i + 1]));
                    if (__all_sync(0xffffffffu, big * z_of_s <= TANH_SMALL)) {
                        const float2 zs = make_float2(z_of_s, z_of_s), c2 = make_float2(cap2, cap2);
#pragma unroll
                        for (int i = 0; i < 32; i += 2) {
                            const float2 z = mul2(make_float2(v[i], v[i + 1]), zs), q = mul2(z, z);
                            float2 p = make_float2(TANH_C4, TANH_C4);
                            p = fma2(p, q, make_float2(TANH_C3, TANH_C3));
                            p = fma2(p, q, make_float2(TANH_C2, TANH_C2));
                            p = fma2(p, q, make_float2(TANH_C1, TANH_C1));
                            p = fma2(p, q, make_float2(TANH_C0, TANH_C0));
                            const float2 r2 = mul2(mul2(p, z), c2);
                            v[i] = r2.x;
                            v[i + 1] = r2.y;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = fmaf(-2.0f * cap2, rcp(1.0f + ex2(v[i] * two_s)), cap2);
                    }
                };
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                float y[64];                                             // the scores read last
#pragma unroll 1
                for (int c = 0; c < BK; c += 64) {
                    tc_ld32_nowait(s_addr + c, reinterpret_cast<uint32_t*>(y));
                    tc_ld32_nowait(s_addr + c + 32, reinterpret_cast<uint32_t*>(y + 32));
                    tc_ld_wait();
                    if (changed) {
                        if (capped) cap(y), cap(y + 32);
                        const int lo = first_key - key0 - c, hi = last - key0 - c;
#pragma unroll
                        for (int i = 0; i < 64; ++i)
                            if (i > hi || i < lo) y[i] = -INFINITY;
                        tc_st32(s_addr + c, reinterpret_cast<uint32_t*>(y));
                        tc_st32(s_addr + c + 32, reinterpret_cast<uint32_t*>(y + 32));
                    }
#pragma unroll
                    for (int i = 0; i < 64; i += 8) {
                        mx4[0] = max3(mx4[0], y[i], y[i + 1]);
                        mx4[1] = max3(mx4[1], y[i + 2], y[i + 3]);
                        mx4[2] = max3(mx4[2], y[i + 4], y[i + 5]);
                        mx4[3] = max3(mx4[3], y[i + 6], y[i + 7]);
                    }
                }
                if (changed) tc_st_wait();
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;
                const bool grow = mx > m + 8.0f;
                float alpha = 1.0f;
                if (grow) {
                    alpha = ex2(m - mx);                                // 0 for the first keys a row sees
                    m = mx;
                }
                const float neg_m = m == -INFINITY ? 0.f : -m;          // a row that sees no key yet
                if (t > 0 && __any_sync(0xffffffffu, grow)) {
                    // Rare.  (O holds the product of the step before: the scores of this one say so.)
#pragma unroll 1
                    for (int c = 0; c < HD; c += 16) {
                        float o[16];
                        tc_ld16(o_addr + c, o);
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] *= alpha;
                        tc_st16(o_addr + c, reinterpret_cast<uint32_t*>(o));
                    }
                }
                // value rows that hold no token yet are made zero before they are multiplied
                const int valid = pooled ? BK : kv_len - (j + jw) * BK;  // (places without a block hold zeros)
                if (valid < BK && (split || s == 0)) {
                    // (The slot's phase before this one is complete: its tile was an earlier key block's keys, whose scores came
                    // before these.  The one after needs the product that waits for this warp.)
                    const int v_n = base + w.place_v(j), v_slot = v_n % NSLOT;
                    ok = __all_sync(0xffffffffu, mbar_wait(&sh.full[v_slot], (v_n / NSLOT) & 1, abort_flag, status, 7));
                    if (!ok) break;
                    const int first = max(valid, 0);
#pragma unroll 1
                    for (int i = r; i < (BK - first) * (HD / 8); i += BQ) {
                        const int row = first + i / (HD / 8), chunk = i % (HD / 8);
                        *reinterpret_cast<uint4*>(kv_s + v_slot * TILE_BYTES + (chunk >> 3) * PANEL_BYTES + row * 128 +
                                                  (((chunk & 7) ^ (row & 7)) << 4)) = make_uint4(0, 0, 0, 0);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the zeros before the tensor core reads them
                }
                // P over the scores; the product begins with the first half
                float2 sum2[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
                const float2 sl2_2 = make_float2(sl2, sl2), neg_m2 = make_float2(neg_m, neg_m);
                auto probs = [&](int c, const float* v) {                // of the 32 scores from column c on
                    uint32_t packed[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float2 e = fma2(make_float2(v[i], v[i + 1]), sl2_2, neg_m2);
                        const float2 pp = make_float2(ex2(e.x), ex2(e.y));
                        sum2[(i >> 1) & 3] = add2(sum2[(i >> 1) & 3], pp);
                        __nv_bfloat162 hh = __floats2bfloat162_rn(pp.x, pp.y);      // key 2k in the low half, key 2k + 1 in the high half
                        packed[i >> 1] = *reinterpret_cast<uint32_t*>(&hh);
                    }
                    tc_st16(s_addr + c / 2, packed);
                };
                auto hand_over = [&](int part) {
                    tc_st_wait();
                    tc_fence_before();                                   // P and the rescaled O before it multiplies and accumulates
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.p_full[s][part]);
                };
                if (LONGS && n_blk >= LONG) {
                    float z[32];
                    tc_ld32_nowait(s_addr, reinterpret_cast<uint32_t*>(z));
                    tc_ld_wait();
                    probs(0, z);
                    tc_ld32_nowait(s_addr + 32, reinterpret_cast<uint32_t*>(z));
                    tc_ld_wait();
                    probs(32, z);
                    hand_over(0);
                    probs(64, y);
                    probs(96, y + 32);
                    hand_over(1);
                } else {
#pragma unroll 1
                    for (int part = 0; part < 2; ++part) {
                        tc_ld32_nowait(s_addr + part * P_FIRST, reinterpret_cast<uint32_t*>(y));
                        tc_ld32_nowait(s_addr + part * P_FIRST + 32, reinterpret_cast<uint32_t*>(y + 32));
                        tc_ld_wait();
                        probs(part * P_FIRST, y);
                        probs(part * P_FIRST + 32, y + 32);
                        hand_over(part);
                    }
                }
                l = l * alpha + (((sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y)) + ((sum2[2].x + sum2[2].y) + (sum2[3].x + sum2[3].y)));
            }
            if (!ok) break;
            base += 2 * n_blk;
            // (rows of tokens beyond the sequence's end were computed from other tokens' queries and are left out here)
            bf16* dst = out + ((int64_t)(w.tok0 + min(tok, w.q_len - 1)) * n_heads + head) * HD;
            const float gate = EXTRA && X.gate && store ? X.gate[(int64_t)(w.tok0 + tok) * n_heads + head] : 1.0f;
            auto put = [&](int c, const float* v) {                  // 32 numbers of the row from column c on
#pragma unroll
                for (int g4 = 0; g4 < 4; ++g4) {
                    uint4 o;
                    __nv_bfloat162* hh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                    for (int i = 0; i < 4; ++i) hh[i] = __floats2bfloat162_rn(v[8 * g4 + 2 * i], v[8 * g4 + 2 * i + 1]);
                    *reinterpret_cast<uint4*>(dst + c + 8 * g4) = o;
                }
            };
            if (!split || n_blk == 1) {
                // the row is the stream's own (of one key block: the even stream's)
                if (!split || s == 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&sh.o_full[s], uses[s] & 1, abort_flag, status, 7));
                    if (!ok) break;
                    tc_fence_after();
                    const float l_row = l + (sink ? ex2(sink2 - m) : 0.f);
                    const float inv = l_row == 0.f ? 0.f : gate / l_row;
#pragma unroll 1
                    for (int c = 0; c < HD; c += 32) {               // (every lane takes part in the loads; only rows that exist are stored)
                        float v[32];
                        tc_ld32_nowait(o_addr + c, reinterpret_cast<uint32_t*>(v));
                        tc_ld_wait();
                        if (c + 32 == HD) {                          // read before the next item's product writes
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&sh.o_empty[s]);
                        }
                        if (store) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) v[i] *= inv;
                            put(c, v);
                        }
                        __syncwarp();
                    }
                }
                ++uses[0];
                uses[1] += split ? 0 : 1;
            } else {
                // both streams hold a part of every row: each stream's warps make half of the columns
                ok = __all_sync(0xffffffffu, mbar_wait(&sh.o_full[0], uses[0] & 1, abort_flag, status, 7) &&
                                                 mbar_wait(&sh.o_full[1], uses[1] & 1, abort_flag, status, 7));
                if (!ok) break;
                ++uses[0], ++uses[1];
                sh.ml[s][0][r] = m;
                sh.ml[s][1][r] = l;
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.join);
                ok = __all_sync(0xffffffffu, mbar_wait(&sh.join, joins & 1, abort_flag, status, 7));
                if (!ok) break;
                tc_fence_after();
                const float m0 = sh.ml[0][0][r], m1 = sh.ml[1][0][r], mm = fmaxf(m0, m1);
                const float f0 = m0 == -INFINITY ? 0.f : ex2(m0 - mm), f1 = m1 == -INFINITY ? 0.f : ex2(m1 - mm);
                const float l_row = sh.ml[0][1][r] * f0 + sh.ml[1][1][r] * f1 + (sink ? ex2(sink2 - mm) : 0.f);
                const float inv = l_row == 0.f ? 0.f : gate / l_row, i0 = f0 * inv, i1 = f1 * inv;
                constexpr int HALF = HD / 2;
#pragma unroll 1
                for (int c = s * HALF; c < (s + 1) * HALF; c += 32) {
                    float v[32], u[32];
                    tc_ld32_nowait(lane_base + COL_O + c, reinterpret_cast<uint32_t*>(v));
                    tc_ld32_nowait(lane_base + COL_O + HD + c, reinterpret_cast<uint32_t*>(u));
                    tc_ld_wait();
                    if (store) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = fmaf(u[i], i1, v[i] * i0);
                        put(c, v);
                    }
                    __syncwarp();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.joined);              // (both streams' warps have read both results)
                ok = __all_sync(0xffffffffu, mbar_wait(&sh.joined, joins & 1, abort_flag, status, 7));
                ++joins;
                if (lane == 0) mbar_arrive(&sh.o_empty[s]);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (sh.abort_flag) {
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);   // copies in flight land before the block leaves
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

}  // namespace prompttc
}  // namespace wick

using namespace wick;

WICK_API int wick_attn_prompt_tc_supported() { return prompttc::SUPPORTED ? 1 : 0; }

// Queries bfloat16 [tokens, heads, HD] as a TMA descriptor with boxes of 64 numbers x gs heads x T tokens: T gs rows of 128 bytes.
static int make_heads_map(CUtensorMap* map, const void* ptr, long long tokens, int heads, int gs, int T) {
    EncodeTiledFn fn = encode_tiled_fn();
    WICK_REQUIRE(fn != nullptr, "attention (tcgen05): the driver does not provide cuTensorMapEncodeTiled");
    WICK_REQUIRE(((uintptr_t)ptr & 15) == 0, "attention (tcgen05): operand is not 16-byte aligned");
    const int hd = prompttc::HD;
    cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)heads, (cuuint64_t)tokens};
    cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)heads * hd * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)gs, (cuuint32_t)T};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    WICK_REQUIRE(r == CUDA_SUCCESS, "attention (tcgen05): cuTensorMapEncodeTiled failed with code %d (tokens %lld, heads %d, box %d x %d)",
                 (int)r, tokens, heads, gs, T);
    return 0;
}

// q, out: bfloat16 [n_tokens, n_heads, HD]; kv: one schedule entry's cache, bfloat16
// [kv_pages, 2, n_kv, 64, HD] (it already holds the new tokens' keys and values);
// n_tiles: the step's 64-row work items (one per 64 new tokens of a sequence, numbered
// sequence by sequence); status: device int (code 7 if a block gave up waiting).
static int attn_prompt_tc(const void* q, long long n_tokens, const void* kv, long long kv_pages, void* out, int n_tiles, const int* cu_seqlens,
                          int n_seqs, const int* start, const int* page_table, int table_width, int n_heads, int n_kv, float scale,
                          int* status, int mask, int mask_size, const float* sink, const void* pool, const prompttc::TcExtra* extra, void* s) {
    using namespace prompttc;
    WICK_REQUIRE(mask == 0 || ((mask == 1 || mask == 2) && mask_size > 0), "attention: mask %d of size %d", mask, mask_size);
    WICK_REQUIRE(SUPPORTED, "attention (tcgen05): head_dim %d is not 64 or 128", (int)WICK_HD);
    WICK_REQUIRE(n_heads > 0 && n_kv > 0 && n_heads % n_kv == 0, "attention: %d heads over %d kv heads", n_heads, n_kv);
    WICK_REQUIRE(n_heads <= 65535, "attention: %d heads is beyond the grid limit", n_heads);
    if (n_tiles == 0) return 0;
    const int group = n_heads / n_kv;
    int gs = 1;                                                    // heads of a tile: as many as fill its rows with whole tokens
    while (group % (2 * gs) == 0 && 2 * gs <= BQ) gs *= 2;
    const int T = BQ / gs, columns = n_heads / gs;
    // the most work items of R tokens that sequences of n_tokens tokens (or of n_tiles 64-row items) can make
    auto items = [&](long long R) { return (int)min((n_tokens + n_seqs * (R - 1)) / R, n_tiles * ((64 + R - 1) / R)); };
    // Items of two tiles share every key and value tile; but as long as items of one tile find an SM each they take half as long
    // (512 tokens, 32 heads over 8: 64 items of two 16.4 us, 128 of one 13.2), with up to two an SM they are no worse unless every
    // sequence is one block of keys (2,048 tokens, 16 heads over 4: 39 and 31 us; 640 tokens, 32 over 8: 18.9 and 15.8; 16 x 64 tokens: 12.8
    // and 16.8), and beyond, where the last round of two is the emptier one and the keys are many (1,419 tokens behind 3,100: 118 and 103;
    // 4 x 700 alone, 16 over 4: 22.5 and 27.1).
    const long long one = (long long)items(T) * columns, two = (long long)items(2 * T) * columns, sms = sm_count();
    const long long keys = ((long long)table_width * kPage - n_tokens / max(n_seqs, 1) / 2) / BK;     // blocks of keys a tile sees, about
    // Steps of up to 64 tokens, in which no matrix product's sums depend on the other sequences, always take one tile: nor do these then.
    const int tiles = n_tokens <= 64 || one <= sms || (one <= 2 * sms && keys >= 1) || (two <= 2 * sms && (one + sms - 1) / sms < 2 * ((two + sms - 1) / sms) && keys >= 16) ? 1 : 2;
    const int n_items = items(T * tiles);
    WICK_REQUIRE((long long)n_items * columns <= INT32_MAX / 2, "attention (tcgen05): %d work items of %d columns are too many", n_items, columns);
    // a block an SM that works through its items one behind the other (more than MAX_ITEMS each: in several rounds)
    const int rounds = ceil_div((long long)n_items * columns, (long long)MAX_ITEMS * sm_count()), blocks = min(n_items * columns, rounds * sm_count());
    CUtensorMap q_map, kv_map, pool_map;
    if (int e = make_heads_map(&q_map, q, n_tokens, n_heads, gs, T)) return e;
    if (int e = make_bf16_map(&kv_map, kv, kv_pages * 2 * n_kv * kPage, HD, kPage, "attention (tcgen05)")) return e;
    pool_map = kv_map;
    TcExtra X = {0, 0, 0.f, nullptr};
    if (extra) X = *extra;
    if (pool) {
        WICK_REQUIRE(mask == 2 && X.block > 0 && X.pool_tiles > 0, "attention (tcgen05): blocks are seen beside a window");
        if (int e = make_bf16_map(&pool_map, pool, (long long)n_seqs * X.pool_tiles * 2 * n_kv * kPage, HD, kPage, "attention (tcgen05)")) return e;
    } else {
        X.block = 0;
    }
    // (up to four key blocks - every captured prompt step - the order is worth less than the ~2 us that finding it takes)
    const int ordered = table_width > 4 * BK / kPage ? 1 : 0;
    const bool guard = tiles == 2 && 2 * T > BK;
    // (all items are short: of a table of so few pages, every captured step's among them)
    const bool shorts = !extra && !guard && (long long)table_width * kPage <= (LONG - 1) * BK;
    auto kernel = extra ? (guard ? attn_prompt_tc_kernel<true, true, true> : attn_prompt_tc_kernel<true, false, true>)
                        : (guard ? attn_prompt_tc_kernel<false, true, true> : (shorts ? attn_prompt_tc_kernel<false, false, false> : attn_prompt_tc_kernel<false, false, true>));
    static bool raised[5] = {false, false, false, false, false};
    bool& done = raised[shorts ? 4 : (extra ? 2 : 0) + (guard ? 1 : 0)];
    if (!done) {
        WICK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        done = true;
    }
    WICK_CUDA(launch(kernel, dim3(blocks), dim3(THREADS), (size_t)SMEM_BYTES, (cudaStream_t)s, q_map,
                     kv_map, (bf16*)out, cu_seqlens, n_seqs, start, page_table, table_width, n_heads,
                     n_kv, gs, T, columns, group / gs, tiles, n_items, ordered, scale, status, mask, mask_size, sink, pool_map, X));
    return check_launch("attn_prompt_tc");
}

// ... then the mask (0, or 1 / 2 with its size) and the sinks (float32 [n_heads] or null).
WICK_API int wick_attn_prompt_tc_masked_bf16(const void* q, long long n_tokens, const void* kv, long long kv_pages, void* out,
                                             int n_tiles, const int* cu_seqlens, int n_seqs,
                                             const int* start, const int* page_table, int table_width, int n_heads, int n_kv,
                                             float scale, int* status, int mask, int mask_size, const float* sink, void* s) {
    return attn_prompt_tc(q, n_tokens, kv, kv_pages, out, n_tiles, cu_seqlens, n_seqs, start, page_table, table_width, n_heads, n_kv, scale,
                          status, mask, mask_size, sink, nullptr, nullptr, s);
}

// ... then the blocks' array (bfloat16 [n_seqs * pool_tiles, 2, n_kv, 64, HD], or null), its tiles a sequence and positions a block, the cap
// of the scores (0: none) and the factors of the result (float32 [n_tokens, n_heads] or null).
WICK_API int wick_attn_prompt_tc_pooled_bf16(const void* q, long long n_tokens, const void* kv, long long kv_pages, void* out,
                                             int n_tiles, const int* cu_seqlens, int n_seqs,
                                             const int* start, const int* page_table, int table_width, int n_heads, int n_kv,
                                             float scale, int* status, int mask, int mask_size, const float* sink, const void* pool,
                                             int pool_tiles, int block, float cap, const float* gate, void* s) {
    const prompttc::TcExtra X = {pool_tiles, block, cap, gate};
    return attn_prompt_tc(q, n_tokens, kv, kv_pages, out, n_tiles, cu_seqlens, n_seqs, start, page_table, table_width, n_heads, n_kv, scale,
                          status, mask, mask_size, sink, pool, &X, s);
}

WICK_API int wick_attn_prompt_tc_bf16(const void* q, long long n_tokens, const void* kv, long long kv_pages, void* out,
                                      int n_tiles, const int* cu_seqlens, int n_seqs,
                                      const int* start, const int* page_table, int table_width, int n_heads, int n_kv,
                                      float scale, int* status, void* s) {
    return wick_attn_prompt_tc_masked_bf16(q, n_tokens, kv, kv_pages, out, n_tiles, cu_seqlens, n_seqs, start, page_table,
                                           table_width, n_heads, n_kv, scale, status, 0, 0, nullptr, s);
}
