// QVB8 mixture-of-experts MLP for a handful of tokens (decode / verify): out[t] = sum_j w[t,j] * down_e( act( up_e(x_t) ) ),
// e = idx[t,j], over stacked expert packs.
//
// Replaces the reference's fused expert stack (formats/qvb8/backends/cuda_qvb8/qvb8_cuda.cu:844-992 gated SiLU,
// :994-1058 relu^2; stacked layout built by formats/qvb8/backends_experts.py:144-196).  The reference makes every
// (token, expert) PAIR one row block of a grouped GEMV, so an expert chosen by several tokens is read once per
// token.  Here the pairs are first grouped by expert (one small kernel, deterministic), and every selected expert's
// rows are then streamed ONCE for all the tokens that chose it: the bytes read are those of the distinct experts.
//
// With per-expert plans (qvb8_moe_plan_build), column counts that are multiples of 128 and 16-byte aligned stacks, five
// launches (with programmatic dependent launch):
//   route    which pairs belong to which expert (one warp, match + popcount); the activations as saturated fp16
//            (qvb8_cuda.cu:1069, saturating_half) in operand order, and their sums
//   up       moe_tiles_kernel: 16-row tiles of the chosen experts x the tokens that chose them, on mma.sync
//   hidden   act(U) per pair, scaled by a power of two and split into two fp16 parts (22 bits), and its sum
//   down     moe_tiles_kernel over both parts
//   combine  out[t] = sum_j w[t,j] * Yd[pair] * 2^k, j ascending
// Without plans, or for other layouts: route -> up rows -> down rows -> combine, a warp per output row on the CUDA cores
// (for the gated form gate row i and up row I + i together), each lane taking 8 consecutive columns of a 256-column block,
// which are exactly nb whole bytes; the row sum is reduced with shuffles.
// Arithmetic: fp32 band value fma(id, tau_s, min_s) -- on the tiles in the factored form tau_s * sum x (id - c) +
// fma(c, tau_s, min_s) * sum x, c the row's id nearest a zero weight: products exact, sums fp32, and no sum
// larger than the result's own scale -- and fp32 hidden activations (22 to 23 of their 24 bits on the tiles).  Against 64 bits, tiles /
// row route: 1.8e-7 / 2.6e-7 (2048 x 768, SiLU), 1.7e-7 / 1.9e-7 (1024 x 512, relu^2), 1.9e-7 / 3.4e-7 (4096 x 1024, SiLU).
#include "common.cuh"
#include "fragment.cuh"
#include "plan.cuh"
#include "tile_reads.h"

namespace qv {

constexpr int MOE_WARPS = 8;
constexpr int MOE_TOK = 4;                 // tokens per pass over a row (row route)
constexpr int MOE_SMEM_EXPERTS = 2048;     // experts whose counts fit the route kernel's shared memory

struct MoeRoute {                          // device tables built by the route kernel
    int *counts;                           // [E] pairs that chose expert e
    int *first;                            // [E] position of expert e's first pair
    int *plist;                            // [npairs] pair numbers t * topk + j by position: expert by expert, ascending
    int *ppos;                             // [npairs] position of a pair; -1 = its expert index is outside [0, E), or the
                                           // token named one expert more than M times: its rows are never computed and the
                                           // combine step counts them as zero
    int *slots;                            // [min(E, npairs)] the distinct chosen experts, ascending
    int *nslots;                           // [1]
    int *bad;                              // [1] set when a pair could not be listed
};

__device__ __forceinline__ float moe_load(const void *__restrict__ X, int x_dtype, int64_t i) {
    return x_dtype == QVB8_F32 ? load_x<QVB8_F32>(X, i) : x_dtype == QVB8_BF16 ? load_x<QVB8_BF16>(X, i) : load_x<QVB8_F16>(X, i);
}

// Operand order of a row of P activations: the 16-byte slot of columns 128 chunk + 32 t + 8 i .. + 7 is number
// 16 chunk + 4 i + t, so that the four lanes of a token read 64 consecutive bytes; eight values per slot in pos_a order.
__device__ __forceinline__ int moe_slot(int c) { return ((c >> 7) << 4) | (((c >> 3) & 3) << 2) | ((c >> 5) & 3); }
__device__ __forceinline__ uint4 moe_pack8(const __half (&h)[8]) {
    auto two = [](__half a, __half b) { return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16); };
    return make_uint4(two(h[0], h[2]), two(h[1], h[3]), two(h[4], h[6]), two(h[5], h[7]));
}
// Block-wide sum in a fixed order.
__device__ __forceinline__ float moe_block_sum(float s, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    float t = red[0];
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    return t;
}

// Block 0: its first warp walks the pairs 32 at a time; a pair's place among its expert's pairs is the expert's count so
// far plus its rank in the warp's match mask: ascending, no atomics.  (A thread per expert that scanned all pairs took
// 20 us at 256 pairs.)  The other blocks: the activations, either one token per block in operand order with its sum
// (frag), or as fp32 values of their saturated-fp16 narrowing (Xf; qvb8_cuda.cu:963 `saturating_half(X).to(float)`).
__global__ void __launch_bounds__(256) moe_route_kernel(const int64_t *__restrict__ idx, int npairs, int E, int M, MoeRoute r,
                                                        const void *__restrict__ X, int x_dtype, int P, uint4 *__restrict__ frag,
                                                        float *__restrict__ sums, float *__restrict__ Xf) {
    __shared__ float red[8];
    const int lane = threadIdx.x & 31;
    if (blockIdx.x > 0 && frag) {
        const int t = blockIdx.x - 1;
        float s = 0.f;
        for (int c = threadIdx.x * 8; c < P; c += 256 * 8) {
            __half h[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                h[k] = sat_half(moe_load(X, x_dtype, (int64_t)t * P + c + k));
                s += __half2float(h[k]);
            }
            frag[(int64_t)t * (P >> 3) + moe_slot(c)] = moe_pack8(h);
        }
        s = moe_block_sum(s, red);
        if (threadIdx.x == 0) sums[t] = s;
        return;
    }
    if (blockIdx.x > 0) {
        const int64_t nx = (int64_t)M * P;
        for (int64_t i = (int64_t)(blockIdx.x - 1) * blockDim.x + threadIdx.x; i < nx; i += (int64_t)(gridDim.x - 1) * blockDim.x)
            Xf[i] = __half2float(sat_half(moe_load(X, x_dtype, i)));
        return;
    }
    __shared__ int s_cnt[MOE_SMEM_EXPERTS];
    int *cnt = E <= MOE_SMEM_EXPERTS ? s_cnt : r.counts;
    for (int e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;
    __syncthreads();
    if (threadIdx.x < 32) {
        bool bad = false;
        for (int p0 = 0; p0 < npairs; p0 += 32) {
            const int p = p0 + lane;
            const int64_t e64 = p < npairs ? idx[p] : -1;
            const int e = e64 >= 0 && e64 < E ? (int)e64 : -1;
            const uint32_t same = __match_any_sync(0xffffffffu, e);
            const int before = e >= 0 ? cnt[e] : 0, rank = before + __popc(same & ((1u << lane) - 1u));
            __syncwarp();
            const bool ok = e >= 0 && rank < M;
            if (e >= 0 && lane == __ffs(same) - 1) cnt[e] = min(M, before + __popc(same));
            __syncwarp();
            if (p < npairs) { r.ppos[p] = ok ? rank : -1; bad |= !ok; }
        }
        bad = __any_sync(0xffffffffu, bad);
        int nslots = 0, at = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {                           // positions: expert by expert
            const int e = e0 + lane, c = e < E ? cnt[e] : 0;
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const uint32_t chosen = __ballot_sync(0xffffffffu, c > 0);
            if (e < E) { r.counts[e] = c; r.first[e] = at + incl - c; }
            if (c > 0) r.slots[nslots + __popc(chosen & ((1u << lane) - 1u))] = e;
            nslots += __popc(chosen);
            at += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) { *r.nslots = nslots; *r.bad = bad; }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < npairs; p += blockDim.x) {
        const int rank = r.ppos[p];
        if (rank >= 0) {
            const int pos = r.first[idx[p]] + rank;
            r.ppos[p] = pos;
            r.plist[pos] = p;
        }
    }
}

// ---- tiles of the chosen experts -----------------------------------------------------------------------------------
//
// HBM roofline on the distinct experts' rows, and what keeps a kernel from it is that they are short: 2 KB (up) and 768
// bytes (down) in the 35B-A3B-class layer, 16 of them per tile.  Run as jobs of the streaming kernel a tile cost a visit
// of the finishing warp (2.2 us) and two hand-overs: 71 us per side at 8 tokens, 1.56 TB/s.  Here nothing is handed over:
// a WARP owns a tile from its bytes to its results.  It keeps a ring of MT_RING stages (256 columns of the 16 rows) that it
// fills itself with 16-byte cp.async, running ahead across tile boundaries, turns them into mma.sync operands as the
// streaming kernel does (fragment.cuh, ids centred), multiplies them with the expert's tokens straight from the L1 (the
// operand-ordered activations of a few tokens fit it) and writes the rows; what it needs to know of a tile is loaded while
// the tile before is multiplied.  Consecutive warps take consecutive tiles, i.e. the same expert's activations.  The layer
// at 8 / 32 tokens, a call with the host: 168 -> 92 us / 676 -> 178 us (239 and 519 MB of distinct experts).
//
// PARTS: operand rows per pair (1: an activation row per token; 2: the two parts of a hidden row).
constexpr int MT_WARPS = 4;                // warps per CTA
// CTAs per SM, as many as the registers allow (6 spill).  Warps in flight are what counts: a chunk is a chain of loads,
// conversions and eight dependent MMAs.  Up tiles at 8 tokens with 3 / 4 / 5 CTAs: 60 / 48 / 42 us; three or four stages
// per warp, stages of 128 columns, or two accumulator chains: 45 us and more.
__host__ __device__ constexpr int mt_ctas(int parts, int groups) { return groups == 2 ? (parts == 2 ? 3 : 4) : (parts == 2 ? 4 : 5); }
constexpr int MT_RING = 2;                 // stages of a warp's ring
constexpr int MT_COLS = 256;               // columns of a stage
// MMAs in a chain; 2 / 4 / 8: 2.4e-7 / 2.0e-7 / 2.3e-7 from 64 bits with sums of the whole row at once (relu^2, 1024 x 512), 1.7e-7 with 4
// and sums of 256 columns in between; 32 tokens 163 us with row-long chains, 178 now.
constexpr int MT_CHAIN = 4;
static_assert(row_stage_vecs_fit(MT_COLS) && row_stage_vecs(MT_COLS, MT_COLS, 8) <= 16, "a stage of a row: inside the row, a vector per lane");
__host__ __device__ constexpr int mt_stage_bytes() {
    int m = 0;
    for (int nb = 3; nb <= 8; ++nb) m = 16 * stage_row_stride(nb, 2) > m ? 16 * stage_row_stride(nb, 2) : m;
    return m;
}
__device__ __forceinline__ int stage_row_stride_of(int nb) {           // stage_row_stride(nb, 2)
    constexpr uint32_t s3 = stage_row_stride(3, 2) / 16, s4 = stage_row_stride(4, 2) / 16, s5 = stage_row_stride(5, 2) / 16,
                       s6 = stage_row_stride(6, 2) / 16, s7 = stage_row_stride(7, 2) / 16, s8 = stage_row_stride(8, 2) / 16;
    constexpr unsigned long long packed = (unsigned long long)s3 | ((unsigned long long)s4 << 8) | ((unsigned long long)s5 << 16) |
                                          ((unsigned long long)s6 << 24) | ((unsigned long long)s7 << 32) | ((unsigned long long)s8 << 40);
    return (int)((packed >> (8 * (nb - 3))) & 0xff) * 16;
}
struct MoeTiles {
    const uint8_t *ids, *nbits;
    const int64_t *bit_off;
    const uint8_t *plan;       // per expert: a plan (plan_layout(Q, 0)), `stride` bytes apart
    int64_t stride, tiles_off;
    int ntiles, Q, P, topk;
    MoeRoute route;
    const uint4 *frag;         // operand-ordered rows, P / 8 slots each; part k of row i at frag + k * part_slots
    int64_t part_slots;
    const float *sums;         // per row, over its parts
    int by_pair;               // rows are numbered by pair position (down) or by token (up)
    float *out;                // (positions, Q)
};

// One 128-column chunk of a 16-row tile: 8 MMAs per operand row set.  The MMA's own additions truncate, and a chain as long as
// the row drifts towards zero: MT_CHAIN of them run from zero and are added to `stage`, the sums of the 256 columns at hand
// (additions that round).  Second parts (2^-11 of the first) go straight to the row's sums.
template <int NB, int NX, int PARTS>
__device__ __forceinline__ void mt_chunk(uint32_t wa, uint32_t wb, const uint4 *const (&xp)[NX], float (&stage)[NX / PARTS][4], float (&sum)[NX][4],
                                         const PairConst &pa, const PairConst &pb) {
    constexpr int D = Pairing<NB>::D;
    constexpr bool AHEAD = NX <= 2;                                    // the chunk's activations are requested together
    uint32_t Wa[NB], Wb[NB];
    uint4 xa[AHEAD ? 4 : 1][NX];
    float acc[NX / PARTS][4];
    if constexpr (AHEAD) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int n = 0; n < NX; ++n) xa[i][n] = __ldg(xp[n] + i * 4);
    }
    load_block<NB>(wa, Wa);
    load_block<NB>(wb, Wb);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint4 x[NX];
#pragma unroll
        for (int n = 0; n < NX; ++n) x[n] = AHEAD ? xa[AHEAD ? i : 0][n] : __ldg(xp[n] + i * 4);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int f0 = D == 2 ? 8 * i + 4 * h : 8 * i + 2 * h;
            if ((2 * i + h) % MT_CHAIN == 0) {
#pragma unroll
                for (int n = 0; n < NX / PARTS; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
            }
            const uint32_t a0 = pair_reg<NB, true>(Wa, f0, pa), a2 = pair_reg<NB, true>(Wa, f0 + 1, pa);
            const uint32_t a1 = pair_reg<NB, true>(Wb, f0, pb), a3 = pair_reg<NB, true>(Wb, f0 + 1, pb);
#pragma unroll
            for (int n = 0; n < NX; ++n) {
                float (&c)[4] = n % PARTS == 0 ? acc[n / PARTS] : sum[n];
                if constexpr (D == 2) {
                    mma16816(c, a0, a1, a2, a3, h == 0 ? x[n].x : x[n].z, h == 0 ? x[n].y : x[n].w);
                } else {                                               // slots hold (x0 x2)(x1 x3)(x4 x6)(x5 x7): pairs (x[2h] x[2h+4]), (x[2h+1] x[2h+5])
                    const uint32_t sel = h == 0 ? 0x5410u : 0x7632u;
                    mma16816(c, a0, a1, a2, a3, __byte_perm(x[n].x, x[n].z, sel), __byte_perm(x[n].y, x[n].w, sel));
                }
            }
            if ((2 * i + h) % MT_CHAIN == MT_CHAIN - 1) {
#pragma unroll
                for (int n = 0; n < NX / PARTS; ++n)
#pragma unroll
                    for (int k = 0; k < 4; ++k) stage[n][k] += acc[n][k];
            }
        }
    }
}

// One row times one operand row, id by id, lanes over columns (the sum in every lane).  For rows that the fragments cannot take,
// and for sums that are not finite: an infinity times a centred id is a NaN at id = centre and has the wrong sign below it.
template <int PARTS>
__device__ __forceinline__ float mt_row_product(const MoeTiles &p, int64_t meta, int64_t xrow, float ts, float ms) {
    const int nb = __ldg(p.nbits + meta), lane = threadIdx.x & 31;
    const int64_t base = __ldg(p.bit_off + meta);
    const __half *x = reinterpret_cast<const __half *>(p.frag + xrow * (p.P >> 3));
    float a = 0.f;
    for (int c = lane; c < p.P; c += 32) {
        const int at = (moe_slot(c) << 3) + pos_a(c & 7);
        float xv = __half2float(x[at]);
        if (PARTS == 2) xv += __half2float(x[p.part_slots * 8 + at]);
        a = __fmaf_rn(xv, band(field_bytes(p.ids, base + (int64_t)c * nb, nb), ts, ms), a);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// What a warp needs to know of a tile; loaded while the tile before is multiplied.  Lane r (and r + 16) holds row r's: two tiles of
// it are live at a time, and the registers decide how many CTAs an SM takes.
struct MoeTile {
    int nb, npair, first, row;
    float ms, ts;
};

// GROUPS: token groups of eight that a pass over a tile takes.
template <int PARTS, int GROUPS>
__global__ void __launch_bounds__(MT_WARPS * 32, mt_ctas(PARTS, GROUPS)) moe_tiles_kernel(const __grid_constant__ MoeTiles p) {
    constexpr int NX = GROUPS * PARTS;
    extern __shared__ __align__(128) uint8_t smem[];                   // [warp][stage][16 rows]
    __shared__ __align__(16) uint32_t pair_table[PAIR_TABLE_WORDS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (tid < PAIR_TABLE_WORDS) pair_table[tid] = pair_const_word(3 + (tid >> 2), tid & 3);
    __syncthreads();
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int total = *p.route.nslots * p.ntiles, nwarps = gridDim.x * MT_WARPS, item0 = blockIdx.x * MT_WARPS + warp;
    const uint32_t ring32 = smem_u32(smem + warp * MT_RING * mt_stage_bytes());
    const int nst_row = (p.P + MT_COLS - 1) / MT_COLS;
    auto expert_of = [&](int item) { return item < total ? p.route.slots[item / p.ntiles] : 0; };
    auto desc = [&](int item, int e) {
        return reinterpret_cast<const TileDesc *>(p.plan + (int64_t)e * p.stride + p.tiles_off) + item % p.ntiles;
    };
    // ---- the fetch cursor: tile, stage, and the row offsets of its tile (lane r holds row r's)
    int f_item = item0, f_st = 0, f_slot = 0, f_nb = 0, f_cnt = 0, n_nb = 0, n_cnt = 0, nn_e;
    uint32_t f_b16 = 0, n_b16 = 0;
    auto look = [&](int item, int e, int &nb, int &cnt, uint32_t &b16) {
        nb = cnt = 0;
        b16 = 0;
        if (item < total) {
            const TileDesc *d = desc(item, e);
            nb = __ldg(&d->nb);
            cnt = __ldg(&d->cnt);
            b16 = __ldg(&d->b16[lane & 15]);
        }
    };
    auto step_tile = [&]() {                                           // to the next tile that streams; two more are looked up ahead
        do {
            f_item += nwarps;
            f_nb = n_nb; f_cnt = n_cnt; f_b16 = n_b16;
            look(f_item + nwarps, nn_e, n_nb, n_cnt, n_b16);
            nn_e = expert_of(f_item + 2 * nwarps);
        } while (f_nb == 0 && f_item < total);
        f_st = 0;
    };
    look(f_item, expert_of(f_item), f_nb, f_cnt, f_b16);
    look(f_item + nwarps, expert_of(f_item + nwarps), n_nb, n_cnt, n_b16);
    nn_e = expert_of(f_item + 2 * nwarps);
    if (f_nb == 0 && f_item < total) step_tile();
    // 256 columns of 16 rows into a stage: two rows per step, a lane a 16-byte vector
    auto copy_rows = [&](int slot, int st, int nb, int cnt, uint32_t b16l) {
        const int vecs = row_stage_vecs(p.P - st * MT_COLS, MT_COLS, nb);   // of a row: 2 nb, nb for a last chunk of 128 columns
        const uint32_t stride = (uint32_t)stage_row_stride_of(nb);
        const uint32_t dst = ring32 + (uint32_t)(slot * mt_stage_bytes()) + (uint32_t)((lane >> 4) * stride + (lane & 15) * 16);
        const uint8_t *src = p.ids + (int64_t)st * (32 * nb) + (lane & 15) * 16;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 2 * i + (lane >> 4);
            const uint32_t b16 = __shfl_sync(0xffffffffu, b16l, r);
            if ((lane & 15) < vecs && r < cnt)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + (uint32_t)(2 * i) * stride), "l"(src + (int64_t)b16 * 16) : "memory");
        }
    };
    auto fetch = [&]() {                                               // one stage of the stream of tiles, one commit group
        if (f_item < total) {
            copy_rows(f_slot, f_st, f_nb, f_cnt, f_b16);
            if (++f_st == nst_row) step_tile();
            if (++f_slot == MT_RING) f_slot = 0;
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int k = 0; k < MT_RING - 1; ++k) fetch();
    auto tile_info = [&](int item, int e) {
        MoeTile m{};
        if (item < total) {
            const TileDesc *d = desc(item, e);
            m.nb = __ldg(&d->nb);
            m.npair = p.route.counts[e];
            m.first = p.route.first[e];
            m.row = __ldg(&d->row[lane & 15]);                         // (-1 for padding)
            m.ms = __ldg(&d->ms[lane & 15]);
            m.ts = __ldg(&d->ts[lane & 15]);
        }
        return m;
    };
    // operand row of the expert's j-th pair
    auto xrow = [&](const MoeTile &m, int j) { return p.by_pair ? m.first + j : p.route.plist[m.first + j] / p.topk; };
    MoeTile nxt = tile_info(item0, expert_of(item0));
    int nxt_e = expert_of(item0 + nwarps), nxt_row = item0 < total ? xrow(nxt, min(g, nxt.npair - 1)) : 0;
    int slot = 0;
    for (int item = item0; item < total; item += nwarps) {
        const MoeTile m = nxt;
        const int myrow = nxt_row;                                     // of pair g (or the last)
        nxt = tile_info(item + nwarps, nxt_e);
        nxt_e = expert_of(item + 2 * nwarps);
        const int nb = m.nb, npair = m.npair;
        if (nb == 0) {
            // rows the fragments cannot take (widths outside 3..8, or not on 16 bytes): id by id, lanes over columns
            const int e = expert_of(item);
            const TileDesc *d = desc(item, e);
            for (int rr = 0; rr < __ldg(&d->cnt); ++rr) {
                const int q = __ldg(&d->row[rr]);
                const float rms = __ldg(&d->ms[rr]), rts = __ldg(&d->ts[rr]);
                for (int j = 0; j < npair; ++j) {
                    const float a = mt_row_product<PARTS>(p, (int64_t)e * p.Q + q, xrow(m, j), rts, rms);
                    if (lane == 0) p.out[(int64_t)(m.first + j) * p.Q + q] = a;
                }
            }
            nxt_row = item + nwarps < total ? xrow(nxt, min(g, nxt.npair - 1)) : 0;
            continue;
        }
        const float centre = zero_id(m.ms, m.ts, nb);
        const PairConst pc = pair_const(pair_table, nb);
        const PairConst pa = centred(pc, __shfl_sync(0xffffffffu, centre, g)), pb = centred(pc, __shfl_sync(0xffffffffu, centre, g + 8));
        const uint32_t stride = (uint32_t)stage_row_stride_of(nb);
        const uint32_t woff = (uint32_t)g * stride + (uint32_t)(t * 4 * nb);
        // a tile chosen by more tokens than a pass takes is streamed again per pass (the bytes come from the L2 then)
        for (int j0 = 0; j0 < npair; j0 += 8 * GROUPS) {
            const uint4 *xp[NX];
#pragma unroll
            for (int n = 0; n < GROUPS; ++n) {
                const int r = n == 0 && j0 == 0 ? myrow : xrow(m, min(j0 + 8 * n + g, npair - 1));
#pragma unroll
                for (int k = 0; k < PARTS; ++k) xp[n * PARTS + k] = p.frag + (int64_t)r * (p.P >> 3) + t + k * p.part_slots;
            }
            float acc[NX][4];
#pragma unroll
            for (int n = 0; n < NX; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
            for (int st = 0; st < nst_row; ++st) {
                int at = slot;
                if (j0 == 0) {
                    fetch();
                    asm volatile("cp.async.wait_group %0;\n" ::"n"(MT_RING - 1) : "memory");
                } else {                                               // on its own, into the stage that was consumed last
                    at = slot == 0 ? MT_RING - 1 : slot - 1;
                    const TileDesc *d = desc(item, expert_of(item));
                    copy_rows(at, st, nb, __ldg(&d->cnt), __ldg(&d->b16[lane & 15]));
                    asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;\n" ::: "memory");
                }
                __syncwarp();
                const uint32_t wa = ring32 + (uint32_t)(at * mt_stage_bytes()) + woff;
                const int chunks = min(2, (p.P >> 7) - 2 * st);
                float stage[GROUPS][4];
#pragma unroll
                for (int n = 0; n < GROUPS; ++n) stage[n][0] = stage[n][1] = stage[n][2] = stage[n][3] = 0.f;
#define MT_STAGE(NB_)                                                                  \
    for (int c = 0; c < chunks; ++c) {                                                 \
        const uint32_t w = wa + c * (16 * NB_);                                        \
        mt_chunk<NB_, NX, PARTS>(w, w + 8 * stride, xp, stage, acc, pa, pb);           \
        _Pragma("unroll") for (int n = 0; n < NX; ++n) xp[n] += 16;                    \
    }
                switch (nb) {                                          // uniform over the warp
                    case 8: MT_STAGE(8); break;
                    case 7: MT_STAGE(7); break;
                    case 6: MT_STAGE(6); break;
                    case 5: MT_STAGE(5); break;
                    case 4: MT_STAGE(4); break;
                    default: MT_STAGE(3); break;
                }
#undef MT_STAGE
#pragma unroll
                for (int n = 0; n < GROUPS; ++n)
#pragma unroll
                    for (int k = 0; k < 4; ++k) acc[n * PARTS][k] += stage[n][k];
                __syncwarp();                                          // the stage may be refilled
                if (j0 == 0 && ++slot == MT_RING) slot = 0;
            }
            if (j0 + 8 * GROUPS >= npair) nxt_row = item + nwarps < total ? xrow(nxt, min(g, nxt.npair - 1)) : 0;
            // rows g, g + 8 x tokens 2 t, 2 t + 1 of each eight
            const float mid = __fmaf_rn(zero_id(m.ms, m.ts, nb), m.ts, m.ms);      // the band value that the centred ids count from
            int row[2];
            float ts[2], ms[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                row[h] = __shfl_sync(0xffffffffu, m.row, g + 8 * h);
                ts[h] = __shfl_sync(0xffffffffu, m.ts, g + 8 * h);
                ms[h] = __shfl_sync(0xffffffffu, mid, g + 8 * h);
            }
#pragma unroll
            for (int n = 0; n < GROUPS; ++n)
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int j = j0 + 8 * n + 2 * t + k;
                    const float sx = j < npair ? p.sums[xrow(m, j)] : 0.f;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float v = acc[n * PARTS][2 * h + k];
                        if (PARTS == 2) v += acc[n * PARTS + PARTS - 1][2 * h + k];
                        const bool live = j < npair && row[h] >= 0;
                        const float y = __fmaf_rn(ts[h], v, ms[h] * sx);
                        if (live) p.out[(int64_t)(m.first + j) * p.Q + row[h]] = y;
                        if constexpr (PARTS == 2) {                    // (the activations of the up tiles are saturated)
                            // once more, without a centre, where the hidden row holds an infinity (and no NaN: sx)
                            uint32_t again = __ballot_sync(0xffffffffu, live && !(fabsf(y) <= 3.402823466e38f) && sx == sx);
                            while (again) {
                                const int src = __ffs(again) - 1, r = (src >> 2) + 8 * h;
                                again &= again - 1;
                                const int jj = __shfl_sync(0xffffffffu, j, src), q = __shfl_sync(0xffffffffu, m.row, r);
                                const float rts = __shfl_sync(0xffffffffu, m.ts, r), rms = __shfl_sync(0xffffffffu, m.ms, r);
                                const float a = mt_row_product<PARTS>(p, (int64_t)expert_of(item) * p.Q + q, xrow(m, jj), rts, rms);
                                if (lane == src) p.out[(int64_t)(m.first + jj) * p.Q + q] = a;
                            }
                        }
                    }
                }
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// A block per pair: h = act(U[pos]) * 2^-k, k chosen so that the row's largest magnitude lies in [2^14, 2^15) (k = 0 for a
// zero row), as the sum of two fp16 parts in operand order, and the parts' sum.  ACT 0: U holds gate (first I values) and
// up (next I); ACT 1: relu^2 of the I values.
template <int ACT>
__global__ void __launch_bounds__(128) moe_hidden_kernel(const float *__restrict__ U, uint4 *__restrict__ frag, int64_t part_slots,
                                                         float *__restrict__ sums, int *__restrict__ kexp, const MoeRoute r, int E, int I) {
    asm volatile("griddepcontrol.launch_dependents;\n griddepcontrol.wait;\n" ::: "memory");
    const int pos = blockIdx.x;
    if (pos >= r.first[E - 1] + r.counts[E - 1]) return;               // pairs without a place (bad experts) leave a tail
    const float *u = U + (int64_t)pos * (ACT == 0 ? 2 * I : I);
    auto value = [&](int i) {
        if (ACT == 0) {
            const float gt = u[i];
            return (gt / (1.0f + __expf(-gt))) * u[I + i];
        }
        const float v = fmaxf(u[i], 0.f);
        return v * v;
    };
    float amax = 0.f;
    for (int i = threadIdx.x; i < I; i += 128) {
        const float v = fabsf(value(i));
        if (v <= 3.402823466e38f) amax = fmaxf(amax, v);               // (infinities and NaNs keep their own scale-free fate)
    }
    __shared__ float red[4], red2[4];
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    int k = 0;
    if (amax > 0.f) {
        int e;
        frexpf(amax, &e);                                               // amax = m * 2^e, m in [0.5, 1)
        k = e - 15;                                                     // amax * 2^-k in [2^14, 2^15)
    }
    if (threadIdx.x == 0) kexp[pos] = k;
    float s = 0.f;
    uint4 *f = frag + (int64_t)pos * (I >> 3);
    for (int c = threadIdx.x * 8; c < I; c += 128 * 8) {
        __half hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float v = ldexpf(value(c + j), -k);
            hi[j] = __float2half_rn(v);
            const float h = __half2float(hi[j]);
            const bool inf = fabsf(h) == INFINITY;                     // (left out of the sum, which is a NaN only for a NaN)
            lo[j] = inf ? __float2half_rn(0.f) : __float2half_rn(v - h);
            s += inf ? 0.f : h + __half2float(lo[j]);
        }
        f[moe_slot(c)] = moe_pack8(hi);
        f[part_slots + moe_slot(c)] = moe_pack8(lo);
    }
    s = moe_block_sum(s, red2);
    if (threadIdx.x == 0) sums[pos] = s;
}

struct MoeRows {
    const float *X;            // ACT 0/1: (M, P) narrowed activations, by token; ACT 2: (npairs, P) hidden, by pair
    int topk;
    const uint8_t *ids;
    const float *min_s, *tau_s;   // [E][Q]
    const uint8_t *nbits;
    const int64_t *bit_off;       // global bit offsets into ids
    int Q, P;                     // rows per expert, columns
    int R;                        // outputs per pair: ACT 0: Q / 2, else Q
    float *out;                   // (npairs, R) fp32
    MoeRoute route;
    int M;
};

// 8 ids of width nb (<= 8) that start at byte `a` of the stream: exactly nb bytes, fetched as two aligned 8-byte words
// (the stream carries pad bytes after its last row).
__device__ __forceinline__ uint64_t load_8_fields(const uint8_t *__restrict__ ids, int64_t a) {
    const uint64_t *w = reinterpret_cast<const uint64_t *>(ids + (a & ~(int64_t)7));
    const uint64_t lo = __ldg(w), hi = __ldg(w + 1);
    const int sh = (int)(a & 7) * 8;
    return sh ? (lo >> sh) | (hi << (64 - sh)) : lo;
}

__device__ __forceinline__ void load_x8(const float *__restrict__ X, int64_t off, float (&x)[8]) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(X + off));
    const float4 b = __ldg(reinterpret_cast<const float4 *>(X + off) + 1);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}

// ACT: 0 = gated SiLU (rows i and I + i of the up pack -> H[p, i] = silu(g) * u), 1 = relu^2 (row i -> H[p, i]),
// 2 = none (row d of the down pack, X by pair -> Y[p, d]).
struct MoeRowMeta {
    int nb;
    int64_t bit0;
    float ms, ts;
};
__device__ __forceinline__ MoeRowMeta moe_row_meta(const MoeRows &p, size_t mi) {
    MoeRowMeta m;
    m.nb = __ldg(p.nbits + mi);
    m.bit0 = __ldg(p.bit_off + mi);
    m.ms = __ldg(p.min_s + mi);
    m.ts = __ldg(p.tau_s + mi);
    return m;
}

template <int ACT>
__global__ void __launch_bounds__(MOE_WARPS * 32, 4) moe_rows_kernel(const MoeRows p) {
    const int s = blockIdx.y;
    if (s >= *p.route.nslots) return;
    const int e = p.route.slots[s];
    const int c = p.route.counts[e];
    const int *plist = p.route.plist + p.route.first[e];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wstride = gridDim.x * MOE_WARPS;
    constexpr int NR = ACT == 0 ? 2 : 1;
    int r = blockIdx.x * MOE_WARPS + warp;
    if (r >= p.R) return;
    MoeRowMeta nxt[NR];
#pragma unroll
    for (int k = 0; k < NR; ++k) nxt[k] = moe_row_meta(p, (size_t)e * p.Q + r + (size_t)k * p.R);
    for (; r < p.R; r += wstride) {
        MoeRowMeta m[NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) m[k] = nxt[k];
        if (r + wstride < p.R) {                                       // the next row's metadata loads under this row's work
#pragma unroll
            for (int k = 0; k < NR; ++k) nxt[k] = moe_row_meta(p, (size_t)e * p.Q + r + wstride + (size_t)k * p.R);
        }
        for (int g0 = 0; g0 < c; g0 += MOE_TOK) {
            const int nt = min(MOE_TOK, c - g0);
            float acc[NR][MOE_TOK];
#pragma unroll
            for (int k = 0; k < NR; ++k)
#pragma unroll
                for (int j = 0; j < MOE_TOK; ++j) acc[k][j] = 0.f;
            const bool fast = NR == 1 ? (m[0].nb <= 8 && (m[0].bit0 & 7) == 0)
                                      : (m[0].nb <= 8 && (m[0].bit0 & 7) == 0 && m[NR - 1].nb <= 8 && (m[NR - 1].bit0 & 7) == 0);
            constexpr int UN = 2;                                       // 256-column blocks whose ids are fetched together
            for (int col0 = lane * 8; col0 < p.P; col0 += 256 * UN) {
                uint64_t v[NR][UN];
                if (fast) {                                             // all the row bytes of this step in flight at once
#pragma unroll
                    for (int u = 0; u < UN; ++u)
#pragma unroll
                        for (int k = 0; k < NR; ++k) {
                            const int col = col0 + 256 * u;
                            v[k][u] = col < p.P ? load_8_fields(p.ids, (m[k].bit0 >> 3) + (int64_t)(col >> 3) * m[k].nb) : 0ull;
                        }
                }
#pragma unroll
                for (int u = 0; u < UN; ++u) {
                    const int col = col0 + 256 * u;
                    if (col >= p.P) break;
                    float wv[NR][8];
#pragma unroll
                    for (int k = 0; k < NR; ++k) {
                        if (fast) {
                            const uint32_t mask = (1u << m[k].nb) - 1u;
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                wv[k][i] = __fmaf_rn(small_u2f((uint32_t)(v[k][u] >> (i * m[k].nb)) & mask), m[k].ts, m[k].ms);
                        } else {
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                wv[k][i] = band(field_bytes(p.ids, m[k].bit0 + (int64_t)(col + i) * m[k].nb, m[k].nb), m[k].ts, m[k].ms);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < MOE_TOK; ++j) {
                        if (j < nt) {
                            const int pp = plist[g0 + j];
                            float x[8];
                            load_x8(p.X, (int64_t)(ACT == 2 ? pp : pp / p.topk) * p.P + col, x);
#pragma unroll
                            for (int k = 0; k < NR; ++k)
#pragma unroll
                                for (int i = 0; i < 8; ++i) acc[k][j] = __fmaf_rn(x[i], wv[k][i], acc[k][j]);
                        }
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < MOE_TOK; ++j) {
                if (j < nt) {                                           // warp-uniform
#pragma unroll
                    for (int k = 0; k < NR; ++k)
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) acc[k][j] += __shfl_xor_sync(0xffffffffu, acc[k][j], o);
                    if (lane == 0) {
                        float v;
                        if (ACT == 0) {
                            const float gt = acc[0][j];
                            v = (gt / (1.0f + __expf(-gt))) * acc[NR - 1][j];
                        } else if (ACT == 1) {
                            const float u = fmaxf(acc[0][j], 0.f);
                            v = u * u;
                        } else {
                            v = acc[0][j];
                        }
                        p.out[(size_t)plist[g0 + j] * p.R + r] = v;
                    }
                }
            }
        }
    }
}

// out[t, d] = sum_j w[t, j] * Yd[row of pair (t, j), d] * 2^k, j ascending (qvb8_cuda.cu:936-947); a pair that was never
// computed counts as zero.  Rows by position with their exponents (kexp), or by pair number (kexp null).
template <typename OutT>
__global__ void __launch_bounds__(256) moe_combine_kernel(const float *__restrict__ Yd, const float *__restrict__ w, const int *__restrict__ kexp,
                                                          OutT *__restrict__ out, int topk, int D, const int *__restrict__ ppos) {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int t = blockIdx.y, d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= D) return;
    float a = 0.f;
#pragma unroll 4
    for (int j = 0; j < topk; ++j) {
        const int p = t * topk + j, pos = ppos[p];
        if (pos < 0) continue;
        float y = Yd[(int64_t)(kexp ? pos : p) * D + d];
        if (kexp) y = ldexpf(y, kexp[pos]);
        a = __fmaf_rn(__ldg(w + p), y, a);
    }
    out[(size_t)t * D + d] = narrow<OutT>(a);
}

struct MoeScratch {
    int64_t counts, first, plist, ppos, slots, nslots, bad, Xf, H, Yd, total, total_rows;   // (total_rows: the row route's)
    int64_t kexp, xsum, hsum, frag, U;                                 // the tiles' sections (frag: X, then the hidden parts in H)
};
static MoeScratch moe_scratch(int64_t M, int64_t topk, int64_t E, int64_t Pup, int64_t R_up, int64_t Qdn, int64_t Qup) {
    MoeScratch s{};
    const int64_t npairs = M * topk;
    auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
    s.counts = 0;
    s.first = s.counts + up(E * 4);
    s.plist = s.first + up(E * 4);
    s.ppos = s.plist + up(npairs * 4);
    s.slots = s.ppos + up(npairs * 4);
    s.nslots = s.slots + up(E * 4);
    s.bad = s.nslots + 256;
    s.kexp = s.bad + 256;
    s.xsum = s.kexp + up(npairs * 4);
    s.hsum = s.xsum + up(M * 4);
    s.Xf = s.hsum + up(npairs * 4);                                    // row route: fp32; tiles: the fp16 operands
    s.frag = s.Xf;
    s.H = s.Xf + up(M * Pup * 4);                                      // row route: fp32; tiles: two fp16 parts
    s.Yd = s.H + up(npairs * R_up * 4);
    s.U = s.Yd;                                                        // (read by the hidden kernel, before the down tiles write)
    s.total_rows = s.Yd + up(npairs * Qdn * 4);
    s.total = s.Yd + up(npairs * (Qup > Qdn ? Qup : Qdn) * 4);
    return s;
}

static int check_stack(const qvb8_expert_stack *st, const char *who) {
    if (!st || !st->ids || !st->min_s || !st->tau_s || !st->nbits || !st->bit_off)
        return fail(QVB8_ERR_ARG, "%s: null expert stack", who);
    if (st->Q <= 0 || st->P <= 0 || st->Q > 0x7fffffff || st->P > 0x7fffffff || st->P % 8 != 0)
        return fail(QVB8_ERR_ARG, "%s: Q=%lld P=%lld (P must be a multiple of 8)", who, (long long)st->Q, (long long)st->P);
    if (!aligned(st->ids, 8)) return fail(QVB8_ERR_ALIGN, "%s: the stacked ids must be 8-byte aligned", who);
    return QVB8_OK;
}

}  // namespace qv

QV_API int64_t qvb8_moe_scratch_bytes(int64_t M, int64_t topk, int64_t E, int64_t Pup, int64_t Qup, int64_t Qdn, int act) {
    if (M <= 0 || topk <= 0 || E <= 0 || Pup <= 0 || Qup <= 0 || Qdn <= 0) return 0;
    return qv::moe_scratch(M, topk, E, Pup, act == 0 ? Qup / 2 : Qup, Qdn, Qup).total;
}

/* Bytes of the plans of all E experts of a stack with Q rows per expert (one plan per expert, back to back). */
QV_API int64_t qvb8_moe_plan_bytes(int64_t E, int64_t Q) {
    if (E <= 0 || Q <= 0) return 0;
    return E * qv::plan_layout(Q, 0).total;
}

/* Builds the per-expert plans of a stack (the row ordering of qvb8_plan_build, once per expert) into `plan`. */
QV_API int qvb8_moe_plan_build(const qvb8_expert_stack *stk, int64_t E, void *plan, int64_t plan_bytes, void *stream) {
    using namespace qv;
    if (int rc = check_device("qvb8_moe_plan_build")) return rc;
    if (int rc = check_stack(stk, "qvb8_moe_plan_build")) return rc;
    const int64_t need = qvb8_moe_plan_bytes(E, stk->Q);
    if (E <= 0 || !plan || plan_bytes < need || !aligned(plan, 256))
        return fail(QVB8_ERR_SCRATCH, "qvb8_moe_plan_build: plan buffer of %lld bytes (256-byte aligned) needed", (long long)need);
    if (E > 0x7fffffff) return fail(QVB8_ERR_ARG, "qvb8_moe_plan_build: too many experts");
    return build_plans(stk->nbits, stk->bit_off, stk->min_s, stk->tau_s, E, stk->Q, plan, reinterpret_cast<cudaStream_t>(stream));
}

/* 1 for a layer of few tokens: up to 8, at most 128 distinct experts, column counts that are multiples of 128 and 16-byte
 * aligned stacks; 0 otherwise.  (Plans serve any number of tokens; this is the question callers have asked so far.) */
QV_API int qvb8_moe_streams(int64_t M, int64_t topk, int64_t E, const qvb8_expert_stack *up, const qvb8_expert_stack *dn) {
    using namespace qv;
    if (!up || !dn || M <= 0 || topk <= 0 || E <= 0) return 0;
    return M <= 8 && (E < M * topk ? E : M * topk) <= 128 && up->P % 128 == 0 && dn->P % 128 == 0 && aligned(up->ids, 16) && aligned(dn->ids, 16);
}

namespace qv {
template <typename... Args>
static int moe_launch(void (*kernel)(Args...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool pdl, const char *what, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kernel, args...) != cudaSuccess) return cuda_status(what);
    return cuda_status(what);
}
template <int PARTS, int GROUPS>
static int moe_tiles_launch(const MoeTiles &p, cudaStream_t st) {
    constexpr int smem = MT_WARPS * MT_RING * mt_stage_bytes();
    static thread_local int granted_dev = -1;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    if (dev != granted_dev) {
        if (cudaFuncSetAttribute(moe_tiles_kernel<PARTS, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return cuda_status("qvb8_moe: shared memory opt-in");
        granted_dev = dev;
    }
    return moe_launch(moe_tiles_kernel<PARTS, GROUPS>, dim3(sms * mt_ctas(PARTS, GROUPS)), MT_WARPS * 32, smem, st, true, "qvb8_moe tiles", p);
}
static int moe_combine_launch(const float *Yd, const float *w, const int *kexp, int x_dtype, void *out, int topk, int D, int M, const int *ppos, bool pdl,
                              cudaStream_t st) {
    const dim3 g((unsigned)((D + 255) / 256), (unsigned)M);
    if (x_dtype == QVB8_BF16) return moe_launch(moe_combine_kernel<__nv_bfloat16>, g, 256, 0, st, pdl, "qvb8_moe combine", Yd, w, kexp, reinterpret_cast<__nv_bfloat16 *>(out), topk, D, ppos);
    if (x_dtype == QVB8_F16) return moe_launch(moe_combine_kernel<__half>, g, 256, 0, st, pdl, "qvb8_moe combine", Yd, w, kexp, reinterpret_cast<__half *>(out), topk, D, ppos);
    return moe_launch(moe_combine_kernel<float>, g, 256, 0, st, pdl, "qvb8_moe combine", Yd, w, kexp, reinterpret_cast<float *>(out), topk, D, ppos);
}
}  // namespace qv

QV_API int qvb8_moe_experts_planned(const void *X, int x_dtype, int64_t M, const int64_t *idx, const float *w, int64_t topk,
                                    int64_t E, const qvb8_expert_stack *up, const qvb8_expert_stack *dn, const void *up_plan,
                                    const void *dn_plan, int act, void *out, void *scratch, int64_t scratch_bytes,
                                    void *stream) {
    using namespace qv;
    const char *who = act == 0 ? "qvb8_moe_experts" : "qvb8_moe_experts(relu2)";
    if (int rc = check_device(who)) return rc;
    if (int rc = check_stack(up, who)) return rc;
    if (int rc = check_stack(dn, who)) return rc;
    if (act != 0 && act != 1) return fail(QVB8_ERR_ARG, "%s: act must be 0 (gated SiLU) or 1 (relu^2)", who);
    if (!X || !idx || !w || !out) return fail(QVB8_ERR_ARG, "%s: null argument", who);
    if (x_dtype != QVB8_F16 && x_dtype != QVB8_BF16 && x_dtype != QVB8_F32) return fail(QVB8_ERR_ARG, "%s: bad X dtype", who);
    if (M <= 0 || topk <= 0 || E <= 0 || M * topk > 65535) return fail(QVB8_ERR_ARG, "%s: M=%lld topk=%lld E=%lld out of range", who, (long long)M, (long long)topk, (long long)E);
    const int64_t R_up = act == 0 ? up->Q / 2 : up->Q;
    if (act == 0 && up->Q % 2 != 0) return fail(QVB8_ERR_ARG, "%s: gate_up must have an even number of rows", who);
    if (R_up != dn->P) return fail(QVB8_ERR_ARG, "%s: up and down shapes disagree (%lld hidden vs %lld columns)", who, (long long)R_up, (long long)dn->P);
    if (!aligned(X, 16)) return fail(QVB8_ERR_ALIGN, "%s: X must be 16-byte aligned", who);
    const MoeScratch L = moe_scratch(M, topk, E, up->P, R_up, dn->Q, up->Q);
    // tiles: plans, whole chunks of 128 columns, rows that start where the plans say
    const bool tiles = up_plan && dn_plan && up->P % 128 == 0 && dn->P % 128 == 0 && aligned(up->ids, 16) && aligned(dn->ids, 16) &&
                       aligned(up_plan, 256) && aligned(dn_plan, 256);
    const int64_t need = tiles ? L.total : L.total_rows;
    if (!scratch || scratch_bytes < need || !aligned(scratch, 256))
        return fail(QVB8_ERR_SCRATCH, "%s: scratch of %lld bytes (256-byte aligned) needed, %lld given", who, (long long)need, (long long)scratch_bytes);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    uint8_t *base = reinterpret_cast<uint8_t *>(scratch);
    auto ints = [&](int64_t off) { return reinterpret_cast<int *>(base + off); };
    auto floats = [&](int64_t off) { return reinterpret_cast<float *>(base + off); };
    MoeRoute route{ints(L.counts), ints(L.first), ints(L.plist), ints(L.ppos), ints(L.slots), ints(L.nslots), ints(L.bad)};
    const int npairs = (int)(M * topk);
    float *Xf = floats(L.Xf), *H = floats(L.H), *Yd = floats(L.Yd);
    if (tiles) {
        uint4 *xfrag = reinterpret_cast<uint4 *>(base + L.frag), *hfrag = reinterpret_cast<uint4 *>(base + L.H);
        moe_route_kernel<<<1 + (unsigned)M, 256, 0, st>>>(idx, npairs, (int)E, (int)M, route, X, x_dtype, (int)up->P, xfrag, floats(L.xsum), nullptr);
        if (int rc = cuda_status("qvb8_moe route")) return rc;
        const PlanLayout pu = plan_layout(up->Q, 0), pd = plan_layout(dn->Q, 0);
        const int64_t part = (int64_t)npairs * (dn->P / 8);            // operand slots of one part of all hidden rows
        // two token groups per pass where an expert sees more than four tokens on average
        const bool many = M > 8 && npairs > 4 * E;
        const MoeTiles tu{up->ids, up->nbits, up->bit_off, reinterpret_cast<const uint8_t *>(up_plan), pu.total, pu.tiles, pu.max_tiles,
                                                  (int)up->Q, (int)up->P, (int)topk, route, xfrag, 0, floats(L.xsum), 0, floats(L.U)};
        if (int rc = many ? moe_tiles_launch<1, 2>(tu, st) : moe_tiles_launch<1, 1>(tu, st)) return rc;
        if (int rc = moe_launch(act == 0 ? moe_hidden_kernel<0> : moe_hidden_kernel<1>, dim3((unsigned)npairs), 128, 0, st, true, "qvb8_moe hidden",
                                (const float *)floats(L.U), hfrag, part, floats(L.hsum), ints(L.kexp), (const MoeRoute)route, (int)E, (int)R_up))
            return rc;
        const MoeTiles td{dn->ids, dn->nbits, dn->bit_off, reinterpret_cast<const uint8_t *>(dn_plan), pd.total, pd.tiles, pd.max_tiles,
                                                  (int)dn->Q, (int)dn->P, (int)topk, route, hfrag, part, floats(L.hsum), 1, Yd};
        if (int rc = many ? moe_tiles_launch<2, 2>(td, st) : moe_tiles_launch<2, 1>(td, st)) return rc;
        return moe_combine_launch(Yd, w, ints(L.kexp), x_dtype, out, (int)topk, (int)dn->Q, (int)M, route.ppos, true, st);
    }
    const int64_t nx = M * up->P;
    moe_route_kernel<<<1 + (unsigned)((nx + 2047) / 2048), 256, 0, st>>>(idx, npairs, (int)E, (int)M, route, X, x_dtype, (int)up->P, nullptr, nullptr, Xf);
    if (int rc = cuda_status("qvb8_moe route")) return rc;
    const int max_slots = (int)(E < npairs ? E : npairs);
    MoeRows a{Xf, (int)topk, up->ids, up->min_s, up->tau_s, up->nbits, up->bit_off, (int)up->Q, (int)up->P,
              (int)R_up, H, route, (int)M};
    // a few CTAs per expert, every warp walking several rows: short rows (a kilobyte or two) would otherwise be all
    // start-up latency
    auto row_blocks = [&](int64_t rows) {                              // about eight CTAs per SM over all experts
        const int64_t all = (rows + MOE_WARPS - 1) / MOE_WARPS, want = (1184 + max_slots - 1) / max_slots;
        return (unsigned)(all < want ? all : (want < 4 ? 4 : want));
    };
    const dim3 gu(row_blocks(R_up), (unsigned)max_slots);
    if (act == 0) moe_rows_kernel<0><<<gu, MOE_WARPS * 32, 0, st>>>(a);
    else moe_rows_kernel<1><<<gu, MOE_WARPS * 32, 0, st>>>(a);
    if (int rc = cuda_status("qvb8_moe up")) return rc;
    MoeRows b{H, (int)topk, dn->ids, dn->min_s, dn->tau_s, dn->nbits, dn->bit_off, (int)dn->Q, (int)dn->P,
              (int)dn->Q, Yd, route, (int)M};
    const dim3 gd(row_blocks(dn->Q), (unsigned)max_slots);
    moe_rows_kernel<2><<<gd, MOE_WARPS * 32, 0, st>>>(b);
    if (int rc = cuda_status("qvb8_moe down")) return rc;
    return moe_combine_launch(Yd, w, nullptr, x_dtype, out, (int)topk, (int)dn->Q, (int)M, route.ppos, false, st);
}

QV_API int qvb8_moe_experts(const void *X, int x_dtype, int64_t M, const int64_t *idx, const float *w, int64_t topk,
                            int64_t E, const qvb8_expert_stack *up, const qvb8_expert_stack *dn, int act, void *out,
                            void *scratch, int64_t scratch_bytes, void *stream) {
    return qvb8_moe_experts_planned(X, x_dtype, M, idx, w, topk, E, up, dn, nullptr, nullptr, act, out, scratch,
                                    scratch_bytes, stream);
}

// Expert index check of the last qvb8_moe_experts call that used `scratch` (after the stream has run it):
// 1 if a pair was left out (its expert index outside [0, E), or its token named one expert more than M times); such a
// pair contributes zero to the output.  Synchronises the host.
QV_API int qvb8_moe_bad_index(const void *scratch, int64_t M, int64_t topk, int64_t E, int64_t Pup, int64_t Qup, int64_t Qdn,
                              int act, int *bad) {
    using namespace qv;
    if (!scratch || !bad) return fail(QVB8_ERR_ARG, "qvb8_moe_bad_index: null argument");
    const MoeScratch L = moe_scratch(M, topk, E, Pup, act == 0 ? Qup / 2 : Qup, Qdn, Qup);
    if (cudaMemcpy(bad, reinterpret_cast<const uint8_t *>(scratch) + L.bad, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return cuda_status("qvb8_moe_bad_index");
    return QVB8_OK;
}
