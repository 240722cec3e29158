// Attention of float32 queries over cached bfloat16 rows that all heads share (attention through a cached latent: a row's
// first r numbers are also its value), on the tensor cores (mma.sync m16n8k16) without giving up 32 bits: a float32 number is
// the exact sum of three bfloat16 numbers (8 + 8 + 8 bits), so a query, and a tile's probabilities, go through the tensor core as
// three operands against the cache's own bfloat16 numbers.  Sums stay short inside the tensor core (a warp's slice of a row; one
// tile's keys) and are carried on by float32 additions outside.
//
// A block takes one token, up to 16 MT heads and a run of the token's visible keys, 32 at a time:
//   * scores: warp w holds, for good, the query fragments of heads 16 (w % MT) .. and of slice w / MT of a row's numbers, and
//     scores all keys of the tile with them; the slices' sums meet in shared memory;
//   * the running maximum and sum and the tile's probabilities: MT * 2 heads a warp, a key a lane;
//   * values: warp w adds the tile's weighted rows into columns w * r / 8 .. of all heads' results.
// Tiles come by cp.async, two ahead (those of rows that no kernel of this step writes before the kernel before this one has
// finished).  A row lies on an odd number of 16-byte pieces in shared memory, so that ldmatrix meets no bank twice.
// A cached row that holds an infinity makes NaN of its tokens' results, also where float32 products would have left an infinity: the
// parts of a number have either sign.
// With `partial` a run's result goes there as a record (maximum, sum, two unused numbers, unnormalised values) for the merge.
//
// What bounds it: with few tokens the chain of a block's start, one or two tiles and its record; with many the tensor cores.  The form
// for other sizes (a key row per warp on the CUDA cores, four heads a block) reads rows and queries from shared memory once per four
// heads.  32 heads, rows of 576 numbers, values of 512, merge included, before -> now: 4 tokens of 700 to 1,500 positions 60 -> 22 us,
// 8 of 1,500 147 -> 25, 64 of 1,000 615 -> 71; prompts of 60 + 100 + 40 tokens 166 -> 29, of 2 x 200 688 -> 69.  Error against 64 bits
// 0.6 to 1.5e-7 of the result's norm (before 1.3 to 2.1e-7).
#pragma once
#include "common.cuh"

namespace wick {
namespace latent {

typedef __nv_bfloat16 bf16;
constexpr int TK = 32, WARPS = 8, STAGES = 3;          // (the sums below are spelled out for two 16-wide steps of a tile)
constexpr int MAX_ROW = 576, MAX_R = 512;
constexpr int SP = TK + 8;                       // floats of a head's row of scores in shared memory, and bfloat16 numbers of one of probabilities

struct Params {
    const float* q;                              // [n, H, R]
    const bf16* store;                           // pages of 64 rows of R numbers
    float* out;                                  // [n, H, r]
    float* partial;                              // [n, H, runs, 4 + r rounded up to 128] or null
    const int *seq_of_token, *positions, *page_table, *start;
    const float* sink;                           // [H] or null
    int table_width, H, R, r, window, keep_first;
    float scale;
};

__device__ __forceinline__ void cp16(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t* v, const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t* v, const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x = t[0] + t[1] + t[2], each a bfloat16 number (the differences are exact).  For x in [0, 1].
__device__ __forceinline__ void split3(float x, bf16* t) {
    t[0] = __float2bfloat16_rn(x);
    x -= __bfloat162float(t[0]);
    t[1] = __float2bfloat16_rn(x);
    x -= __bfloat162float(t[1]);
    t[2] = __float2bfloat16_rn(x);
}
// The same for any x: a number that would be rounded beyond bfloat16's largest is cut instead; an infinity and a NaN are their own first part.
__device__ __forceinline__ void split3_any(float x, bf16* t) {
    t[0] = fabsf(x) < 3.3895e38f ? __float2bfloat16_rn(x) : __float2bfloat16_rz(x);
    const float rest = isfinite(x) ? x - __bfloat162float(t[0]) : 0.f;
    t[1] = __float2bfloat16_rn(rest);
    t[2] = __float2bfloat16_rn(rest - __bfloat162float(t[1]));
}
__device__ __forceinline__ uint32_t pair(bf16 a, bf16 b) {
    __nv_bfloat162 v = __halves2bfloat162(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

template <int MT> struct Sizes {
    static constexpr int HG = 16 * MT, KSPLIT = WARPS / MT;              // heads of a block; slices of a row's numbers
    static constexpr int KPW = (MAX_ROW / 16 + KSPLIT - 1) / KSPLIT;      // 16-wide steps of a slice at most
};
inline int row_pieces(int R) { return (R / 8) | 1; }                      // 16-byte pieces from one row to the next in shared memory
template <int MT> inline size_t smem_bytes(int R) {
    typedef Sizes<MT> Z;
    return (size_t)STAGES * TK * row_pieces(R) * 16 + (size_t)Z::KSPLIT * Z::HG * SP * 4 + (size_t)3 * Z::HG * SP * 2 + 3 * Z::HG * 4;
}

template <int MT>
__global__ void __launch_bounds__(32 * WARPS, 1)
attn_latent_kernel(const Params P) {
    typedef Sizes<MT> Z;
    constexpr int HG = Z::HG, KSPLIT = Z::KSPLIT, KPW = Z::KPW, HPW = HG / WARPS;
    extern __shared__ __align__(128) uint8_t latent_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int R = P.R, r = P.r, pieces = (R / 8) | 1;
    bf16* tiles = reinterpret_cast<bf16*>(latent_smem);                                   // [STAGES][TK][pieces * 8]
    float* scores = reinterpret_cast<float*>(latent_smem + (size_t)STAGES * TK * pieces * 16);   // [KSPLIT][HG][SP]
    bf16* probs = reinterpret_cast<bf16*>(scores + KSPLIT * HG * SP);                     // [3][HG][SP]
    float* corrs = reinterpret_cast<float*>(probs + 3 * HG * SP);                         // [HG]; at the end maxima, sums
    const int groups = (P.H + HG - 1) / HG, t = blockIdx.x / groups, h0 = (blockIdx.x - t * groups) * HG;
    const int seq = P.seq_of_token[t], pos = P.positions[t], first_new = P.start[seq];
    const int* table = P.page_table + (int64_t)seq * P.table_width;
    const int lo = P.window > 0 ? max(0, pos - P.window + 1) : 0;
    const int n_kept = P.window > 0 ? min(P.keep_first, lo) : 0;
    const int total = n_kept + (pos - lo + 1);
    const int tiles_all = (total + TK - 1) / TK, per_run = (tiles_all + (int)gridDim.y - 1) / (int)gridDim.y;
    const int v_begin = TK * per_run * (int)blockIdx.y, v_end = min(total, TK * per_run * ((int)blockIdx.y + 1));
    const int n_tiles = v_end > v_begin ? (v_end - v_begin + TK - 1) / TK : 0;
    auto key_of = [&](int v) { return v < n_kept ? v : lo + (v - n_kept); };
    // (keys beyond the run's end name its last one: their rows are finite and weigh nothing)
    auto load_tile = [&](int i) {
        constexpr int TPK = 32 * WARPS / TK;     // threads that share a key
        const int kk = tid / TPK, c0 = tid % TPK, key = key_of(min(v_begin + i * TK + kk, v_end - 1));
        const bf16* src = P.store + ((int64_t)table[key / kPage] * kPage + key % kPage) * R;
        bf16* dst = tiles + ((int64_t)(i % STAGES) * TK + kk) * pieces * 8;
#pragma unroll 1
        for (int c = c0; c < R / 8; c += TPK) cp16(dst + c * 8, src + c * 8);
    };
    auto settled = [&](int i) { return key_of(min(v_begin + (i + 1) * TK, v_end) - 1) < first_new; };    // rows of earlier steps only
    const bool early0 = n_tiles > 0 && settled(0), early1 = n_tiles > 1 && settled(1);
    if (early0) load_tile(0);
    if (early1) load_tile(1);
    pdl_wait();
    if (n_tiles > 0 && !early0) load_tile(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (n_tiles > 1 && !early1) load_tile(1);
    asm volatile("cp.async.commit_group;" ::: "memory");

    // this warp's query fragments: heads 16 mt + lane / 4 (+ 8), numbers 16 k + 2 (lane % 4) + {0, 1} (+ 8) of its slice
    const int mt = warp % MT, slice = warp / MT, k_steps = R / 16;
    const int k0 = slice * ((k_steps + KSPLIT - 1) / KSPLIT), k_n = min(k_steps, k0 + (k_steps + KSPLIT - 1) / KSPLIT) - k0;
    uint32_t qf[KPW][3][4];
    {
        const float* q = fresh(P.q);
        const int ha = h0 + 16 * mt + (lane >> 2), hb = ha + 8;
        const float* qa = q + ((int64_t)t * P.H + min(ha, P.H - 1)) * R + 2 * (lane & 3);
        const float* qb = q + ((int64_t)t * P.H + min(hb, P.H - 1)) * R + 2 * (lane & 3);
#pragma unroll
        for (int k = 0; k < KPW; ++k) {
            float2 x[4];
            const int at = (k0 + k) * 16;
            const bool in = k < k_n;
            x[0] = in && ha < P.H ? ld2(qa + at) : make_float2(0.f, 0.f);
            x[1] = in && hb < P.H ? ld2(qb + at) : make_float2(0.f, 0.f);
            x[2] = in && ha < P.H ? ld2(qa + at + 8) : make_float2(0.f, 0.f);
            x[3] = in && hb < P.H ? ld2(qb + at + 8) : make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                bf16 a[3], b[3];
                split3_any(x[i].x, a);
                split3_any(x[i].y, b);
#pragma unroll
                for (int j = 0; j < 3; ++j) qf[k][j][i] = pair(a[j], b[j]);
            }
        }
    }
    float m[HPW], l[HPW];                        // of heads warp * HPW ..., the same in every lane
#pragma unroll
    for (int j = 0; j < HPW; ++j) m[j] = -INFINITY, l[j] = 0.f;
    constexpr int NDW = MAX_R / 64;              // 8-wide column blocks of a warp at most
    const int ndw = r / 64, col0 = warp * ndw * 8;
    float o[MT][NDW][4];
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int d = 0; d < NDW; ++d) o[a][d][0] = o[a][d][1] = o[a][d][2] = o[a][d][3] = 0.f;

    for (int i = 0; i < n_tiles; ++i) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                         // tile i is there; everyone is done with tile i - 1, its scores and probabilities
        if (i + 2 < n_tiles) load_tile(i + 2);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const bf16* tile = tiles + (int64_t)(i % STAGES) * TK * pieces * 8;
        const int n_keys = min(TK, v_end - (v_begin + i * TK));
        {
            float s[2][TK / 8][4], low[TK / 8][4];    // the queries' leading parts (even steps, odd steps), the rest
#pragma unroll
            for (int nb = 0; nb < TK / 8; ++nb)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[0][nb][j] = s[1][nb][j] = low[nb][j] = 0.f;
#pragma unroll
            for (int k = 0; k < KPW; ++k) {
                if (k >= k_n) break;
#pragma unroll
                for (int nb = 0; nb < TK / 8; nb += 2) {
                    uint32_t kf[4];
                    const int key = 8 * (nb + (lane >> 4)) + (lane & 7);
                    ldsm4(kf, tile + (key * pieces + 2 * (k0 + k) + ((lane >> 3) & 1)) * 8);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        mma(s[k & 1][nb + e], qf[k][0], kf[2 * e], kf[2 * e + 1]);
                        mma(low[nb + e], qf[k][1], kf[2 * e], kf[2 * e + 1]);
                        mma(low[nb + e], qf[k][2], kf[2 * e], kf[2 * e + 1]);
                    }
                }
            }
#pragma unroll
            for (int nb = 0; nb < TK / 8; ++nb)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[0][nb][j] = (s[0][nb][j] + s[1][nb][j]) + low[nb][j];
            float* sp = scores + ((int64_t)slice * HG + 16 * mt + (lane >> 2)) * SP + 2 * (lane & 3);
#pragma unroll
            for (int nb = 0; nb < TK / 8; ++nb) {
                *reinterpret_cast<float2*>(sp + 8 * nb) = make_float2(s[0][nb][0], s[0][nb][1]);
                *reinterpret_cast<float2*>(sp + 8 * SP + 8 * nb) = make_float2(s[0][nb][2], s[0][nb][3]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < HPW; ++j) {
            const int h = warp * HPW + j;
            float s = 0.f;
#pragma unroll
            for (int z = 0; z < KSPLIT; ++z) s += scores[((int64_t)z * HG + h) * SP + lane];
            s = lane < n_keys ? s * P.scale : -INFINITY;
            const float m_new = fmaxf(m[j], warp_max(s));                 // finite: the tile's first key is visible
            const float corr = expf(m[j] - m_new), p = lane < n_keys ? expf(s - m_new) : 0.f;   // (m = -inf at first: 0)
            l[j] = l[j] * corr + warp_sum(p);
            m[j] = m_new;
            bf16 ps[3];
            split3(p, ps);
#pragma unroll
            for (int z = 0; z < 3; ++z) probs[(z * HG + h) * SP + lane] = ps[z];
            if (lane == 0) corrs[h] = corr;
        }
        __syncthreads();
        // O <- corr O + P V: a tile's sums on their own, those of the probabilities' leading parts apart from the rest, so that what
        // the tensor core adds up stays short
#pragma unroll
        for (int a = 0; a < MT; ++a) {
            uint32_t pf[TK / 16][3][4];
#pragma unroll
            for (int k = 0; k < TK / 16; ++k)
#pragma unroll
                for (int z = 0; z < 3; ++z)
                    ldsm4(pf[k][z], probs + (z * HG + 16 * a + (lane & 7) + ((lane >> 3) & 1) * 8) * SP + 16 * k + (lane >> 4) * 8);
            const float c_lo = corrs[16 * a + (lane >> 2)], c_hi = corrs[16 * a + (lane >> 2) + 8];
#pragma unroll
            for (int d = 0; d < NDW; d += 2) {
                if (d >= ndw) break;
                float v[TK / 16][2][4], w[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[0][e][j] = v[1][e][j] = w[e][j] = 0.f;
#pragma unroll
                for (int k = 0; k < TK / 16; ++k) {
                    uint32_t vf[4];
                    const int key = 16 * k + (lane & 7) + ((lane >> 3) & 1) * 8;
                    // (an odd number of column blocks: the last pair's second block is the next warp's first, or the row's next numbers)
                    ldsm4_trans(vf, tile + key * pieces * 8 + col0 + 8 * (d + (lane >> 4)));
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        mma(v[k][e], pf[k][0], vf[2 * e], vf[2 * e + 1]);
                        mma(w[e], pf[k][2], vf[2 * e], vf[2 * e + 1]);
                        mma(w[e], pf[k][1], vf[2 * e], vf[2 * e + 1]);
                    }
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    o[a][d + e][0] = fmaf(o[a][d + e][0], c_lo, (v[0][e][0] + v[1][e][0]) + w[e][0]);
                    o[a][d + e][1] = fmaf(o[a][d + e][1], c_lo, (v[0][e][1] + v[1][e][1]) + w[e][1]);
                    o[a][d + e][2] = fmaf(o[a][d + e][2], c_hi, (v[0][e][2] + v[1][e][2]) + w[e][2]);
                    o[a][d + e][3] = fmaf(o[a][d + e][3], c_hi, (v[0][e][3] + v[1][e][3]) + w[e][3]);
                }
            }
        }
    }
    // (Not earlier: a block fills its multiprocessor, so that all blocks of the merge that follows would be placed on the few that have none,
    // and read their records through those: 4 tokens of 700 to 1,500 positions, the merge 10.3 us in a step.)
    pdl_trigger();
    // maxima and sums to everyone, then the results: records, or finished here
    float *ms = corrs + HG, *ls = corrs + 2 * HG;
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < HPW; ++j) ms[warp * HPW + j] = m[j], ls[warp * HPW + j] = l[j];
    }
    __syncthreads();
    const int e_pad = (r + 127) / 128 * 128;
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int hl = 16 * a + (lane >> 2) + 8 * half, h = h0 + hl;
            if (h >= P.H) continue;
            float f = 1.f;
            float* dst;
            if (P.partial) {
                float* rec = P.partial + (((int64_t)t * P.H + h) * gridDim.y + blockIdx.y) * (4 + e_pad);
                if (warp == 0 && (lane & 3) == 0) rec[0] = ms[hl], rec[1] = ls[hl];
                dst = rec + 4;
            } else {                             // (the block holds all visible keys, at least the token's own)
                const float big = P.sink ? fmaxf(ms[hl], P.sink[h]) : ms[hl], mine = expf(ms[hl] - big);
                f = mine / (ls[hl] * mine + (P.sink ? expf(P.sink[h] - big) : 0.f));
                dst = P.out + ((int64_t)t * P.H + h) * r;
            }
            dst += col0 + 2 * (lane & 3);
#pragma unroll
            for (int d = 0; d < NDW; ++d)
                if (d < ndw) *reinterpret_cast<float2*>(dst + 8 * d) = make_float2(o[a][d][2 * half] * f, o[a][d][2 * half + 1] * f);
        }
}

}  // namespace latent
}  // namespace wick
