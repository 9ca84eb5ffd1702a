// QVB8R (entropy-coded QVB8) for sm_100a: ids, dense restore and small-M products straight from the rANS stream.
//
// Replaces the reference's qvb8r_cuda kernels (formats/qvb8r/backends/cuda_qvb8r/qvb8r_cuda.cu:36-75 stream,
// :85-270 gemv / multi / tc, :272-308 decode, :310-320 fix_escapes).  The format (container.py:1-12, codec.py:4-21):
// rows sorted by class; a tile = a few consecutive sorted rows of one class coded by 32 interleaved 64-bit rANS
// states; state j codes column 32 * step + j; per symbol  E = tab[class][x & 4095],  s = E & 2047,
// x = ((E >> 22) + 1) * (x >> 12) + ((E >> 11) & 2047);  symbols go in pairs and after a pair every state below
// 2^32 takes the tile's next 32-bit word, lanes in ascending order; id = s + drow[row]; w = fma(id, tau_s, min_s).
//
// This is integer work with a serial dependency per state, so it is bound by instruction issue and latency, not by
// HBM (the stream is ~5 bits per weight); what a B200 offers it is many resident warps.  One warp walks one tile
// (lane j = state j), four tiles of one class per CTA share the class's 16 KB slot table in shared memory.  The word
// stream of a warp passes through a 256-word ring in shared memory that 4-byte asynchronous copies fill two to three
// 64-word blocks ahead of the cursor; a state that refills reads its word with one shared load at cursor + rank, the
// rank from a ballot and a popcount.  A restore and a one-token product take four tiles per CTA: 2560 tiles are then at
// most 20 warps on an SM, against 24 in CTAs of eight (5120 x 5120, one token: 40 against 45 us; two tiles per CTA: 42, and
// 13 against 10 us on short tiles, which the slot table's 16 KB per CTA then outweighs).  Restore of 5120 x 17408 weights
// to fp16: 119 us (157 us with whole blocks, a refill check after every pair and 67 instructions per pair; 53 now), 58 % of
// the issue slots; the rest waits on the chain: two look-ups, a ballot, a popcount and a ring read per pair, 365 cycles
// with four warps per scheduler.
//
// Products follow the reference's contracts: `gemv` / `multi` multiply the fp32 band value with fp32 X (bf16 X is
// exact in fp32); `tc` rounds the band value once to fp16 and multiplies fp16 X, fp32 accumulation.  One token is summed
// lane by lane next to the decoder; several tokens go to the tensor cores (qvb8r_mma_kernel).  Every row sum has a fixed
// order: results are identical from run to run.  Escapes are corrected afterwards from their stored differences, one
// thread per (token, output) in stored order (:310-320).
#include "common.cuh"

namespace qv {

constexpr int R_WPB = 8;                   // warps = tiles per CTA (a block of the schedule holds at most this many)
constexpr int R_RING = 256;                // words of a warp's ring (four blocks of 64)
constexpr int R_RESTORE_WARPS = 4;         // tiles per CTA where the tiles of a block need not meet: half a block

__device__ __forceinline__ uint32_t r_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

struct RStream {
    uint32_t lo, hi;                       // the state
    uint32_t c, lim;                       // bytes consumed; the cursor value at which the next block is fetched
    uint32_t ring;                         // shared address of the warp's ring (1 KB aligned)
    const uint32_t *next;                  // this lane's word of the block to fetch next
};

__device__ __forceinline__ void rstream_fetch(RStream &z, uint32_t dst) {       // the next block of 64 words
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n cp.async.ca.shared.global [%0+128], [%1+128], 4;\n"
                 "cp.async.commit_group;\n" ::"r"(dst), "l"(z.next) : "memory");
    z.next += 64;
}
// Blocks 0..3 are requested; rstream_ready awaits 0 and 1 (two pairs take at most 64 words, so they end inside the next block).
__device__ __forceinline__ void rstream_init(RStream &z, const uint32_t *ring, const uint32_t *__restrict__ words, int64_t off,
                                             const uint64_t *__restrict__ states, int tile, int lane) {
    const uint64_t x = __ldg(states + (int64_t)tile * 32 + lane);
    z.lo = (uint32_t)x;
    z.hi = (uint32_t)(x >> 32);
    z.c = 0;
    z.lim = 256;
    z.ring = r_smem(ring);
    z.next = words + off + lane;
#pragma unroll
    for (int b = 0; b < 4; ++b) rstream_fetch(z, z.ring + b * 256 + lane * 4);
}
__device__ __forceinline__ void rstream_ready() {
    asm volatile("cp.async.wait_group 2;\n" ::: "memory");
    __syncwarp();
}

// One symbol: the slot entry, and the state behind it.  Entries lie in shared memory as sym << 10 | offset | F << 21
// (an offset is below its frequency, a frequency is at most 1024: every field comes out with at most one instruction on
// the decoder's dependency chain); RAW entries are the format's own (symbol | offset << 11 | (F - 1) << 22).
template <bool RAW>
__device__ __forceinline__ uint32_t rstream_symbol(RStream &z, const uint32_t *st) {
    const uint32_t E = st[z.lo & 4095u];
    const uint32_t F = RAW ? (E >> 22) + 1u : E >> 21, o = RAW ? (E >> 11) & 2047u : E & 1023u;
    const uint32_t l = __funnelshift_r(z.lo, z.hi, 12), fh = F * (z.hi >> 12);
    asm("{\n .reg .b64 a;\n mov.b64 a, {%4, %5};\n mad.wide.u32 a, %2, %3, a;\n mov.b64 {%0, %1}, a;\n}\n"
        : "=r"(z.lo), "=r"(z.hi) : "r"(F), "r"(l), "r"(o), "r"(fh));
    return E;
}
__device__ __forceinline__ uint32_t r_sym(uint32_t E) { return (E >> 10) & 2047u; }
// 2^23 + 1024 * symbol as a float: the symbol's field dropped into the mantissa
__device__ __forceinline__ float r_symf(uint32_t E) { return __uint_as_float((E & 0x1FFC00u) | 0x4B000000u); }

// Two symbols per lane (their entries), then the refill; at most two pairs may follow one another without a
// rstream_advance.
template <bool RAW>
__device__ __forceinline__ void rstream_pair(RStream &z, const uint32_t *st, uint32_t &e1, uint32_t &e2) {
    e1 = rstream_symbol<RAW>(z, st);
    e2 = rstream_symbol<RAW>(z, st);
    const bool need = z.hi == 0u;
    const uint32_t mask = __ballot_sync(0xffffffffu, need);
    uint32_t below, v;
    asm("mov.u32 %0, %%lanemask_lt;\n" : "=r"(below));
    const uint32_t a = ((z.c + __popc(mask & below) * 4u) & (R_RING * 4 - 1)) | z.ring;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(a) : "memory");
    z.hi = need ? z.lo : z.hi;
    z.lo = need ? v : z.lo;
    z.c += __popc(mask) * 4u;
}
// Once a block has been used up its place takes a new one (uniform over the warp; at most one block per two pairs).
__device__ __forceinline__ void rstream_advance(RStream &z, int lane) {
    if (z.c >= z.lim) {
        __syncwarp();
        rstream_fetch(z, z.ring + ((z.lim - 256u) & (R_RING * 4 - 1)) + lane * 4);
        z.lim += 256;
        asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        __syncwarp();
    }
}
__device__ __forceinline__ void rstream_done() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

struct RCore {
    const uint32_t *words;
    const int64_t *tile_off;
    const uint64_t *states;
    const int64_t *tiles;                  // (nt, 3): class, first sorted row, rows
    const int32_t *blocks;                 // (nb, 3): class, first tile, tiles (<= R_WPB)
    const uint32_t *tab;                   // (K, 4096)
    const int32_t *perm;                   // sorted row -> original row
    const float *min_s, *tau_s;            // by original row
    const int32_t *drow;                   // by original row
    int Q, P;
};

// Metadata of a tile's rows, 32 rows at a time (one per lane): the loads of a tile's rows are one round trip together.
struct RRows {
    int orow, dr;
    float m, t;
};
__device__ __forceinline__ RRows r_rows(const RCore &c, int r0, int r, int nr, int lane) {
    RRows g{0, 0, 0.f, 0.f};
    if (r + lane < nr) {
        g.orow = c.perm[r0 + r + lane];
        g.m = c.min_s[g.orow];
        g.t = c.tau_s[g.orow];
        g.dr = c.drow[g.orow];
    }
    return g;
}
__device__ __forceinline__ RRows r_row(const RRows &g, int r) {
    RRows o;
    o.orow = __shfl_sync(0xffffffffu, g.orow, r & 31);
    o.dr = __shfl_sync(0xffffffffu, g.dr, r & 31);
    o.m = __shfl_sync(0xffffffffu, g.m, r & 31);
    o.t = __shfl_sync(0xffffffffu, g.t, r & 31);
    return o;
}
// The band value of a symbol: fma(id, tau_s, min_s), id = symbol + drow.  symf - (2^23 - 1024 drow) = 1024 id exactly
// (multiples of 1024 far below 2^34), and 2^-10 tau_s is exact, so the one rounding is the fused multiply-add's.
struct RBand {
    float off, t, m;
};
__device__ __forceinline__ RBand r_band(const RRows &w) {
    return RBand{8388608.0f - 1024.0f * (float)w.dr, w.t * 0.0009765625f, w.m};
}
// pairs of floats in one instruction (each half rounds as the scalar operation does)
__device__ __forceinline__ float2 r_add2(float2 a, float b) {
    float2 d;
    asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n add.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x;\n}\n"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b));
    return d;
}
__device__ __forceinline__ float2 r_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mov.b64 z, {%6, %7};\n fma.rn.f32x2 x, x, y, z;\n"
        " mov.b64 {%0, %1}, x;\n}\n" : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 r_weights(uint32_t e1, uint32_t e2, const RBand &b) {
    return r_fma2(r_add2(make_float2(r_symf(e1), r_symf(e2)), -b.off), make_float2(b.t, b.t), make_float2(b.m, b.m));
}

// The class's slot table into shared memory in the decoder's arrangement; `least` and `most` become the range of the symbols
// this thread saw (the CTA then synchronises, as callers need the table anyway).  Eight 16-byte loads in flight per thread: a
// CTA has few threads, and one load at a time made the table a seventh of a one-token product.
__device__ __forceinline__ uint32_t r_entry(uint32_t E) {
    return ((E & 2047u) << 10) | ((E >> 11) & 1023u) | (((E >> 22) + 1u) << 21);
}
struct RRange {
    uint32_t least = 2047u, most = 0u;
    __device__ __forceinline__ void see(uint32_t E) { least = min(least, E & 2047u); most = max(most, E & 2047u); }
};
__device__ __forceinline__ RRange r_load_table(const RCore &c, int cls, uint32_t *st) {
    RRange range;
    const uint32_t *src = c.tab + (int64_t)cls * 4096;
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll 8
        for (int i = threadIdx.x; i < 1024; i += blockDim.x) {
            const uint4 E = __ldg(reinterpret_cast<const uint4 *>(src) + i);
            range.see(E.x); range.see(E.y); range.see(E.z); range.see(E.w);
            reinterpret_cast<uint4 *>(st)[i] = make_uint4(r_entry(E.x), r_entry(E.y), r_entry(E.z), r_entry(E.w));
        }
    } else {
        for (int i = threadIdx.x; i < 4096; i += blockDim.x) {
            const uint32_t E = __ldg(src + i);
            range.see(E);
            st[i] = r_entry(E);
        }
    }
    return range;
}

// MODE 0: ids (int16).  MODE 1: dense restore to OutT.  The grid is R_WPB / R_RESTORE_WARPS CTAs per block.
template <int MODE, typename OutT>
__global__ void __launch_bounds__(32 * R_RESTORE_WARPS) qvb8r_restore_kernel(const RCore c, int b0, int64_t row_base, OutT *__restrict__ out) {
    __shared__ __align__(16) uint32_t st[4096];
    __shared__ __align__(1024) uint32_t ring[R_RESTORE_WARPS * R_RING];
    constexpr int SUB = R_WPB / R_RESTORE_WARPS;
    const int32_t *blk = c.blocks + 3 * (int64_t)(b0 + blockIdx.x / SUB);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = (blockIdx.x % SUB) * R_RESTORE_WARPS + w, ntb = blk[2];
    if (k - w >= ntb) return;
    const int tile = blk[1] + min(k, ntb - 1);
    const int r0 = (int)c.tiles[3 * (int64_t)tile + 1], nr = (int)c.tiles[3 * (int64_t)tile + 2];
    RStream z;
    rstream_init(z, ring + w * R_RING, c.words, c.tile_off[tile], c.states, tile, lane);
    RRows grp = r_rows(c, r0, 0, nr, lane);
    r_load_table(c, blk[0], st);
    rstream_ready();
    __syncthreads();
    if (k >= ntb) {
        rstream_done();
        return;
    }
    for (int r = 0; r < nr; ++r) {
        if (r > 0 && (r & 31) == 0) grp = r_rows(c, r0, r, nr, lane);
        const RRows row = r_row(grp, r);
        const RBand bd = r_band(row);
        OutT *o = out + (row_base < 0 ? (int64_t)row.orow : (int64_t)(r0 + r) - row_base) * c.P + lane;
        auto pair = [&](OutT *p) {
            uint32_t e1, e2;
            rstream_pair<false>(z, st, e1, e2);
            if constexpr (MODE == 0) {
                p[0] = (int16_t)((int)r_sym(e1) + row.dr);
                p[32] = (int16_t)((int)r_sym(e2) + row.dr);
            } else {
                const float2 v = r_weights(e1, e2, bd);
                p[0] = narrow<OutT>(v.x);
                p[32] = narrow<OutT>(v.y);
            }
        };
        for (int s = c.P >> 7; s > 0; --s, o += 128) {
            pair(o);
            pair(o + 64);
            rstream_advance(z, lane);
        }
        if (c.P & 64) {
            pair(o);
            rstream_advance(z, lane);
        }
    }
    rstream_done();
}

// One warp's tile multiplied lane by lane: lane j sums columns 32 s + j (even and odd s apart), a shuffle tree adds the
// lanes.
template <int MP, typename XT, bool WROUND>
__device__ __forceinline__ void r_tile_products(const RCore &c, const uint32_t *st, RStream &z, RRows grp, int r0, int nr, int lane,
                                                const XT *__restrict__ X, int M, float *__restrict__ Y) {
    const int np = c.P >> 6;                                   // pairs of a row
    for (int r = 0; r < nr; ++r) {
        if (r > 0 && (r & 31) == 0) grp = r_rows(c, r0, r, nr, lane);
        const RRows row = r_row(grp, r);
        const RBand bd = r_band(row);
        float2 acc[MP];
#pragma unroll
        for (int k = 0; k < MP; ++k) acc[k] = make_float2(0.f, 0.f);
        // the activations of two pairs are requested two pairs ahead of their use
        constexpr bool AHEAD = MP <= 4;
        const XT *xp = X + lane;
        float2 cur[2][MP];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < MP; ++k) {
                cur[h][k] = make_float2(0.f, 0.f);
                if (AHEAD && k < M && h < np) cur[h][k] = make_float2((float)xp[(int64_t)k * c.P + h * 64], (float)xp[(int64_t)k * c.P + h * 64 + 32]);
            }
#pragma unroll(MP <= 2 ? 2 : 1)
        for (int s = 0; s < np; s += 2, xp += 128) {
            float2 nxt[2][MP];
            if constexpr (AHEAD) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int k = 0; k < MP; ++k) {
                        nxt[h][k] = cur[h][k];
                        if (k < M && s + 2 + h < np) nxt[h][k] = make_float2((float)xp[(int64_t)k * c.P + 128 + h * 64], (float)xp[(int64_t)k * c.P + 160 + h * 64]);
                    }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (s + h >= np) break;
                uint32_t e1, e2;
                rstream_pair<false>(z, st, e1, e2);
                float2 wt = r_weights(e1, e2, bd);
                if (WROUND) wt = make_float2(__half2float(__float2half_rn(wt.x)), __half2float(__float2half_rn(wt.y)));
#pragma unroll
                for (int k = 0; k < MP; ++k) {
                    if constexpr (AHEAD) {
                        acc[k] = r_fma2(cur[h][k], wt, acc[k]);
                        cur[h][k] = nxt[h][k];
                    } else if (k < M) {
                        const XT *p = xp + (int64_t)k * c.P + h * 64;
                        acc[k] = r_fma2(make_float2((float)p[0], (float)p[32]), wt, acc[k]);
                    }
                }
            }
            rstream_advance(z, lane);
        }
#pragma unroll
        for (int k = 0; k < MP; ++k) {
            float a = acc[k].x + acc[k].y;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (lane == 0 && k < M) Y[(int64_t)k * c.Q + row.orow] = a;
        }
    }
}

// Products with MP tokens of XT on the CUDA cores; WROUND: round the band value to fp16 first (the reference's
// tensor-core contract).  The grid is as the restore's.
template <int MP, typename XT, bool WROUND>
__global__ void __launch_bounds__(32 * R_RESTORE_WARPS) qvb8r_kernel(const RCore c, const XT *__restrict__ X, int M, float *__restrict__ Y) {
    __shared__ __align__(16) uint32_t st[4096];
    __shared__ __align__(1024) uint32_t ring[R_RESTORE_WARPS * R_RING];
    constexpr int SUB = R_WPB / R_RESTORE_WARPS;
    const int32_t *blk = c.blocks + 3 * (int64_t)(blockIdx.x / SUB);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = (blockIdx.x % SUB) * R_RESTORE_WARPS + w, ntb = blk[2];
    if (k - w >= ntb) return;
    const int tile = blk[1] + min(k, ntb - 1);
    const int r0 = (int)c.tiles[3 * (int64_t)tile + 1], nr = (int)c.tiles[3 * (int64_t)tile + 2];
    RStream z;
    rstream_init(z, ring + w * R_RING, c.words, c.tile_off[tile], c.states, tile, lane);
    const RRows grp = r_rows(c, r0, 0, nr, lane);
    r_load_table(c, blk[0], st);
    rstream_ready();
    __syncthreads();
    if (k < ntb) r_tile_products<MP, XT, WROUND>(c, st, z, grp, r0, nr, lane, X, M, Y);
    rstream_done();
}

// ---- several tokens: the tensor cores ------------------------------------------------------------------------------
//
// The decoder is what a product costs, so it must not also pay for the contraction: with 12 tokens the 24 multiply-adds
// and 24 activation loads per pair of symbols were ten times the decoder's own work.  Here the four warps of a CTA decode
// 256 columns of their rows into shared memory (16-bit operands), meet, and each warp multiplies two of the eight
// 32-column groups of all four rows: m16n8k16 with 16 tokens as m and the tiles' rows as n.  Lane (g, t) of a fragment
// takes the eight columns 8 t .. of its group on both sides (one 16-byte load each), the first four in one instruction
// and the last four in the next; the order within k is free.  Two buffers: one barrier per 256 columns.  The warps' sums
// are added in warp order at the end of a row.  Four tiles per CTA rather than eight leave half of n unused, but tiles
// are all the parallelism there is, and whole blocks of eight fill the 148 SMs unevenly (448 blocks: four on some, three
// on most: 207 us against 192).  17408 x 5120, 12 tokens: 179 us; 1190 us with the multiply-adds beside the decoder.
//
//   KIND 0 (`tc`): operand = fp16(band value), X fp16 as given; up to 48 tokens (NT fragments of 16) from one decoding.
//   KIND 1 (`multi`, bf16 X) / KIND 2 (`multi`, fp32 X): up to 8 tokens.  The operand is (symbol - c) / 256, exact in bf16
//     where no symbol of the class is further than 256 from the row's c, and
//     y = 256 tau_s * sum x (symbol - c) / 256 + fma(c + drow, tau_s, min_s) * sum x: the products are exact and only the
//     sums round; a fifth row of ones brings the sums of x.  c is the symbol nearest a zero weight, so that the second
//     term is small (with 256 for every row, activations with a mean left 2.9e-6 over 17408 columns, the lane-by-lane
//     product 4.4e-7; now 3.5e-7).  fp32 activations are split into three bf16 parts (8 + 8 + 8 bits, exact).  A class whose symbols
//     span more than 512, or a sum that is not finite (infinities, NaNs, overflow: the factored form would turn them into
//     NaNs), goes through the lane-by-lane product.
constexpr int RM_WARPS = 4;
constexpr int RM_COLS = 256;                                           // columns decoded between two barriers
constexpr int RM_STRIDE = RM_COLS * 2 + 64;                            // bytes of a row in a buffer (64: rows g, g + 1 on
                                                                       // different banks of the 16-byte fragment loads)
template <bool BF16>
__device__ __forceinline__ void r_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// x = p0 + p1 + p2 exactly, bf16 parts by truncation, each as the upper half of a word (an infinity or a NaN leaves NaNs or
// infinities: the sums are then not finite and the product is redone lane by lane)
__device__ __forceinline__ void r_split(float x, uint32_t &p0, uint32_t &p1, uint32_t &p2) {
    p0 = __float_as_uint(x) & 0xffff0000u;
    const float r = x - __uint_as_float(p0);
    p1 = __float_as_uint(r) & 0xffff0000u;
    p2 = __float_as_uint(r - __uint_as_float(p1));
}

// X is 16-byte aligned (P is a multiple of 64: every row then is).
template <int KIND, int NT>
__global__ void __launch_bounds__(32 * RM_WARPS, KIND == 2 || NT > 1 ? 5 : 7) qvb8r_mma_kernel(const RCore c, const void *__restrict__ Xv,
                                                                                              int M, float *__restrict__ Y) {
    constexpr bool FACTORED = KIND != 0;
    constexpr int NA = KIND == 2 ? 2 : NT;                             // A fragments: fp32 splits take tokens x 3 rows
    constexpr int ROWS = FACTORED ? RM_WARPS + 1 : RM_WARPS;           // rows of a buffer: the tiles' (and the ones)
    constexpr bool AHEAD = KIND != 2 && NT == 1;
    constexpr int SUB = R_WPB / RM_WARPS;
    __shared__ __align__(16) uint32_t st[4096];
    __shared__ __align__(1024) uint32_t ring[RM_WARPS * R_RING];
    __shared__ __align__(16) uint8_t buf[2][ROWS * RM_STRIDE];
    __shared__ float part[RM_WARPS][128];                              // [warp][token][row]
    __shared__ float s_m[2][RM_WARPS], s_t[2][RM_WARPS];
    __shared__ float s_mid[2][RM_WARPS];                               // centre + drow: the id the factored sum counts from
    __shared__ int s_row[2][RM_WARPS];
    __shared__ uint32_t s_least[RM_WARPS], s_most[RM_WARPS];
    const int32_t *blk = c.blocks + 3 * (int64_t)(blockIdx.x / SUB);
    const int sub = (blockIdx.x % SUB) * RM_WARPS, ntb = min(RM_WARPS, blk[2] - sub), tb = blk[1] + sub;
    if (ntb <= 0) return;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int tile = tb + min(w, ntb - 1);
    const int r0 = (int)c.tiles[3 * (int64_t)tile + 1], nr = w < ntb ? (int)c.tiles[3 * (int64_t)tile + 2] : 0;
    RStream z;
    rstream_init(z, ring + w * R_RING, c.words, c.tile_off[tile], c.states, tile, lane);
    RRows grp = r_rows(c, r0, 0, nr, lane);
    int rows = 0;
    for (int k = 0; k < ntb; ++k) rows = max(rows, (int)c.tiles[3 * (int64_t)(tb + k) + 2]);
    RRange range = r_load_table(c, blk[0], st);
    bool scalar = false;
    rstream_ready();
    if (FACTORED) {
        for (int i = threadIdx.x; i < 2 * RM_COLS / 2; i += 32 * RM_WARPS)
            *reinterpret_cast<uint32_t *>(buf[i / (RM_COLS / 2)] + RM_WARPS * RM_STRIDE + (i % (RM_COLS / 2)) * 4) = 0x3f803f80u;
        range.least = __reduce_min_sync(0xffffffffu, range.least);
        range.most = __reduce_max_sync(0xffffffffu, range.most);
        if (lane == 0) { s_least[w] = range.least; s_most[w] = range.most; }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < RM_WARPS; ++k) { range.least = min(range.least, s_least[k]); range.most = max(range.most, s_most[k]); }
        scalar = range.most - range.least > 512u;
    } else {
        __syncthreads();
    }
    // A row's centre: where its weight is zero, as near as exact operands let it be.  They have 8 bits: whole symbols where the
    // class's symbols span 129 to 512, halves from 65, quarters from 33 and so on.
    const int span = (int)(range.most - range.least);
    const float reach = (float)(span <= 1 ? 1 : min(256, 1 << (32 - __clz(span - 1)))), grid = 256.0f / reach;
    const float centre_lo = (float)range.most - reach, centre_hi = (float)range.least + reach;
    if (!scalar) {
        int par = 0;                                                   // buffer of the next chunk
        bool redo = false;
        // (a token beyond M repeats the last: its sums are not written)
        const uint16_t *xa = reinterpret_cast<const uint16_t *>(Xv) + (int64_t)min(g, M - 1) * c.P + w * 64 + t * 8;
        const uint16_t *xb = reinterpret_cast<const uint16_t *>(Xv) + (int64_t)min(g + 8, M - 1) * c.P + w * 64 + t * 8;
        const float *xf = reinterpret_cast<const float *>(Xv) + (int64_t)min(g, M - 1) * c.P + w * 64 + t * 8;
        const uint8_t *bfrag = buf[0] + min(g, ROWS - 1) * RM_STRIDE + t * 16;   // (columns of D beyond ROWS are not read)
        for (int r = 0; r < rows; ++r) {
            if (r > 0 && (r & 31) == 0) grp = r_rows(c, r0, r, nr, lane);
            const RRows row = r_row(grp, r);
            const RBand bd = r_band(row);
            const bool live = r < nr;
            const float centre = fminf(fmaxf(rintf((__fdividef(-row.m, row.t) - (float)row.dr) * grid) / grid, centre_lo), centre_hi);
            const float shift = -32.0f - centre * 0x1p-8f;             // (2^23 + 1024 s) 2^-18 + shift = (s - centre) / 256
            if (lane == 0) { s_row[r & 1][w] = live ? row.orow : -1; s_m[r & 1][w] = row.m; s_t[r & 1][w] = row.t; s_mid[r & 1][w] = centre + (float)row.dr; }
            float sum[NA][4];
#pragma unroll
            for (int n = 0; n < NA; ++n)
#pragma unroll
                for (int k = 0; k < 4; ++k) sum[n][k] = 0.f;
            for (int c0 = 0; c0 < c.P; c0 += RM_COLS, par ^= 1) {
                const int nc = min(RM_COLS, c.P - c0);
                uint16_t *dst = reinterpret_cast<uint16_t *>(buf[par] + w * RM_STRIDE) + lane;
                // one fragment of tokens: its activations are requested here and arrive while the chunk is decoded
                uint4 xu[2], xv[2];
                if constexpr (KIND == 2) {
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        xu[b] = xv[b] = make_uint4(0u, 0u, 0u, 0u);
                        if ((2 * w + b) * 32 < nc) {
                            xu[b] = __ldg(reinterpret_cast<const uint4 *>(xf + c0 + b * 32));
                            xv[b] = __ldg(reinterpret_cast<const uint4 *>(xf + c0 + b * 32) + 1);
                        }
                    }
                } else if constexpr (AHEAD) {
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        xu[b] = xv[b] = make_uint4(0u, 0u, 0u, 0u);
                        if ((2 * w + b) * 32 < nc) {
                            xu[b] = __ldg(reinterpret_cast<const uint4 *>(xa + c0 + b * 32));
                            if (KIND == 0) xv[b] = __ldg(reinterpret_cast<const uint4 *>(xb + c0 + b * 32));
                        }
                    }
                }
                auto pair = [&](uint16_t *p) {
                    uint32_t e1, e2;
                    rstream_pair<false>(z, st, e1, e2);
                    if constexpr (!FACTORED) {
                        const float2 x = r_weights(e1, e2, bd);
                        p[0] = __half_as_ushort(__float2half_rn(x.x));
                        p[32] = __half_as_ushort(__float2half_rn(x.y));
                    } else {
                        const float2 x = r_fma2(make_float2(r_symf(e1), r_symf(e2)), make_float2(0x1p-18f, 0x1p-18f), make_float2(shift, shift));
                        p[0] = __bfloat16_as_ushort(__float2bfloat16_rn(x.x));
                        p[32] = __bfloat16_as_ushort(__float2bfloat16_rn(x.y));
                    }
                };
                if (live) {
#pragma unroll 1
                    for (int i = nc >> 7; i > 0; --i, dst += 128) {
                        pair(dst);
                        pair(dst + 64);
                        rstream_advance(z, lane);
                    }
                    if (nc & 64) {
                        pair(dst);
                        rstream_advance(z, lane);
                    }
                }
                __syncthreads();
                // this warp's two 32-column groups of all rows: two MMAs from zero each, added to the row's sums afterwards (the
                // MMA's own additions truncate: 80 of them in a chain left 1.5e-6 over 5120 columns, fp32 additions 2e-7)
                uint4 q[2];
#pragma unroll
                for (int b = 0; b < 2; ++b)
                    if ((2 * w + b) * 32 < nc) q[b] = *reinterpret_cast<const uint4 *>(bfrag + par * (ROWS * RM_STRIDE) + (2 * w + b) * 64);
                if constexpr (AHEAD) {
                    float acc[2][4] = {};
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        if ((2 * w + b) * 32 >= nc) break;
                        r_mma<FACTORED>(acc[b], xu[b].x, xv[b].x, xu[b].y, xv[b].y, q[b].x, q[b].y);
                        r_mma<FACTORED>(acc[b], xu[b].z, xv[b].z, xu[b].w, xv[b].w, q[b].z, q[b].w);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) sum[0][k] += acc[0][k] + acc[1][k];
                } else if constexpr (KIND != 2) {
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const int col = (2 * w + b) * 32;
                        if (col >= nc) break;
                        const uint16_t *X = reinterpret_cast<const uint16_t *>(Xv) + c0 + col + t * 8;
#pragma unroll
                        for (int n = 0; n < NA; ++n) {
                            const uint4 u = __ldg(reinterpret_cast<const uint4 *>(X + (int64_t)min(16 * n + g, M - 1) * c.P));
                            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(X + (int64_t)min(16 * n + 8 + g, M - 1) * c.P));
                            float acc[4] = {0.f, 0.f, 0.f, 0.f};
                            r_mma<FACTORED>(acc, u.x, v.x, u.y, v.y, q[b].x, q[b].y);
                            r_mma<FACTORED>(acc, u.z, v.z, u.w, v.w, q[b].z, q[b].w);
#pragma unroll
                            for (int k = 0; k < 4; ++k) sum[n][k] += acc[k];
                        }
                    }
                } else {
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};               // (the third parts, 2^-16 of the first, stay in one chain)
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        if ((2 * w + b) * 32 >= nc) break;
                        const uint32_t x[8] = {xu[b].x, xu[b].y, xu[b].z, xu[b].w, xv[b].x, xv[b].y, xv[b].z, xv[b].w};
                        uint32_t a[3][4];                              // parts, pairs of columns
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint32_t l0, l1, l2, h0, h1, h2;
                            r_split(__uint_as_float(x[2 * j]), l0, l1, l2);
                            r_split(__uint_as_float(x[2 * j + 1]), h0, h1, h2);
                            a[0][j] = __byte_perm(l0, h0, 0x7632);
                            a[1][j] = __byte_perm(l1, h1, 0x7632);
                            a[2][j] = __byte_perm(l2, h2, 0x7632);
                        }
                        r_mma<true>(acc, a[0][0], a[1][0], a[0][1], a[1][1], q[b].x, q[b].y);
                        r_mma<true>(acc, a[0][2], a[1][2], a[0][3], a[1][3], q[b].z, q[b].w);
                        r_mma<true>(sum[1], a[2][0], 0u, a[2][1], 0u, q[b].x, q[b].y);
                        r_mma<true>(sum[1], a[2][2], 0u, a[2][3], 0u, q[b].z, q[b].w);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) sum[0][k] += acc[k];
                }
            }
            // the warps' sums, added in warp order; one thread per (token, row)
#pragma unroll
            for (int n = 0; n < (FACTORED ? 1 : NT); ++n) {
                if (KIND == 2) {                                       // smallest parts first
                    sum[0][0] += sum[1][0] + sum[0][2];
                    sum[0][1] += sum[1][1] + sum[0][3];
                }
                *reinterpret_cast<float2 *>(&part[w][g * 8 + 2 * t]) = make_float2(sum[n][0], sum[n][1]);
                if (!FACTORED) *reinterpret_cast<float2 *>(&part[w][(g + 8) * 8 + 2 * t]) = make_float2(sum[n][2], sum[n][3]);
                __syncthreads();
                const int m = 16 * n + (threadIdx.x >> 3), k = threadIdx.x & 7;
                if (m < M && k < ntb && s_row[r & 1][k] >= 0 && (!FACTORED || threadIdx.x < 64)) {
                    float y = 0.f;
#pragma unroll
                    for (int v = 0; v < RM_WARPS; ++v) y += part[v][threadIdx.x];
                    if (FACTORED) {
                        float sumx = 0.f;
#pragma unroll
                        for (int v = 0; v < RM_WARPS; ++v) sumx += part[v][(threadIdx.x & ~7) + RM_WARPS];
                        const float tt = s_t[r & 1][k];
                        y = __fmaf_rn(256.0f * tt, y, __fmaf_rn(s_mid[r & 1][k], tt, s_m[r & 1][k]) * sumx);
                        redo |= !(fabsf(y) <= 3.4e38f);
                    }
                    Y[(int64_t)m * c.Q + s_row[r & 1][k]] = y;
                }
                if (n + 1 < NT && !FACTORED) __syncthreads();
            }
        }
        if (FACTORED && __syncthreads_or(redo)) {
            rstream_done();
            rstream_init(z, ring + w * R_RING, c.words, c.tile_off[tile], c.states, tile, lane);
            rstream_ready();
            grp = r_rows(c, r0, 0, nr, lane);
            scalar = true;
        }
    }
    if constexpr (FACTORED) {
        if (scalar) {
            if constexpr (KIND == 1) r_tile_products<8, __nv_bfloat16, false>(c, st, z, grp, r0, nr, lane, reinterpret_cast<const __nv_bfloat16 *>(Xv), M, Y);
            else r_tile_products<8, float, false>(c, st, z, grp, r0, nr, lane, reinterpret_cast<const float *>(Xv), M, Y);
        }
    }
    rstream_done();
}

// Y[m, uq[u]] += sum_e x[m, ec[e]] * ed[e], e in [ptr[u], ptr[u + 1]) in stored order (qvb8r_cuda.cu:310-320)
__global__ void __launch_bounds__(128) qvb8r_fix_kernel(const float *__restrict__ X, const int64_t *__restrict__ uq,
                                                        const int64_t *__restrict__ ptr, const int64_t *__restrict__ ec,
                                                        const float *__restrict__ ed, float *__restrict__ Y, int64_t U, int M,
                                                        int P, int Q) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= U * M) return;
    const int64_t u = i % U;
    const int m = (int)(i / U);
    const float *x = X + (int64_t)m * P;
    float a = 0.f;
    for (int64_t e = ptr[u]; e < ptr[u + 1]; ++e) a = __fmaf_rn(x[ec[e]], ed[e], a);
    Y[(int64_t)m * Q + uq[u]] += a;
}

// out[m, q] = T(Y[m, q] + sum_e x[m, col[e]] * ed[e]), e in [row_ptr[q], row_ptr[q + 1]) in stored order: the escapes and
// the narrowing of a product behind one launch, the activations in the type they came in.  A thread per output; a row has
// a handful of entries, fetched four at a time so that their latencies overlap.
template <typename XT, typename OutT>
__global__ void __launch_bounds__(128) qvb8r_finish_kernel(const XT *__restrict__ X, const int *__restrict__ row_ptr,
                                                           const int64_t *__restrict__ ec, const float *__restrict__ ed,
                                                           const float *__restrict__ Y, OutT *__restrict__ out, int P, int Q) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
    if (q >= Q) return;
    const XT *x = X + (int64_t)m * P;
    const int e0 = __ldg(row_ptr + q), e1 = __ldg(row_ptr + q + 1);
    float a = 0.f;
    for (int e = e0; e < e1; e += 4) {
        float v[4], d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int ee = min(e + k, e1 - 1);
            v[k] = (float)x[__ldg(ec + ee)];
            d[k] = __ldg(ed + ee);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (e + k < e1) a = __fmaf_rn(v[k], d[k], a);
    }
    const int64_t i = (int64_t)m * Q + q;
    const float y = Y[i];
    out[i] = narrow<OutT>(e1 > e0 ? y + a : y);
}

// Embedding lookup: out[i, :] = row rows[i] of the table, restored as the reference's CPU reader restores it -- a
// multiplication and then an addition, min_s + float(id) * tau_s, not fused (qvb8r_cpu.cpp:44) -- with the row's escapes
// written over.  One warp per requested row: it walks the row's tile from the tile's start (a tile is a few rows) and
// keeps only the last row it decodes.  The slot table is read through the read-only cache: the warps of a CTA need
// different classes, and a lookup touches a handful of rows.
__global__ void __launch_bounds__(32 * R_WPB) qvb8r_embed_kernel(const RCore c, const int64_t *__restrict__ rows, int64_t n,
                                                                const int32_t *__restrict__ inv_perm,
                                                                const int32_t *__restrict__ row_tile,
                                                                const int64_t *__restrict__ esc_ptr,
                                                                const int32_t *__restrict__ esc_col,
                                                                const float *__restrict__ esc_val, float *__restrict__ out) {
    __shared__ __align__(1024) uint32_t ring[R_WPB * R_RING];
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * R_WPB + (threadIdx.x >> 5);
    if (i >= n) return;
    const int64_t q = rows[i];
    float *o = out + i * c.P;
    if (q < 0 || q >= c.Q) {                                           // refused on the host; never read out of range
        for (int col = lane; col < c.P; col += 32) o[col] = 0.f;
        return;
    }
    const int sp = inv_perm[q], tile = row_tile[sp];
    const int k = sp - (int)c.tiles[3 * (int64_t)tile + 1];            // rows of the tile in front of this one
    const uint32_t *st = c.tab + c.tiles[3 * (int64_t)tile] * 4096;
    const float m = c.min_s[q], t = c.tau_s[q];
    const int dr = c.drow[q];
    const int S = c.P / 32;
    RStream z;
    rstream_init(z, ring + (threadIdx.x >> 5) * R_RING, c.words, c.tile_off[tile], c.states, tile, lane);
    rstream_ready();
    for (int r = 0; r <= k; ++r)
        for (int s0 = 0; s0 < S; s0 += 2) {
            uint32_t e1, e2;
            rstream_pair<true>(z, st, e1, e2);
            rstream_advance(z, lane);
            if (r == k) {
                o[s0 * 32 + lane] = __fadd_rn(m, __fmul_rn((float)((int)(e1 & 2047u) + dr), t));
                o[s0 * 32 + 32 + lane] = __fadd_rn(m, __fmul_rn((float)((int)(e2 & 2047u) + dr), t));
            }
        }
    rstream_done();
    __syncwarp();
    for (int64_t e = esc_ptr[q] + lane; e < esc_ptr[q + 1]; e += 32) o[esc_col[e]] = esc_val[e];
}

static int check_rpack(const qvb8r_pack *w, const char *who) {
    if (!w) return fail(QVB8_ERR_ARG, "%s: null pack", who);
    if (!w->words || !w->tile_off || !w->states || !w->tiles || !w->blocks || !w->tab || !w->perm || !w->min_s ||
        !w->tau_s || !w->drow)
        return fail(QVB8_ERR_ARG, "%s: null core array", who);
    if (w->Q <= 0 || w->P <= 0 || w->Q > 0x7fffffff || w->P > 0x7fffffff || w->P % 64 != 0)
        return fail(QVB8_ERR_ARG, "%s: Q=%lld P=%lld (P must be a multiple of 64)", who, (long long)w->Q, (long long)w->P);
    if (w->n_blocks < 0 || w->n_tiles < 0 || w->n_blocks > 0x7fffffff)
        return fail(QVB8_ERR_ARG, "%s: bad tile / block counts", who);
    return QVB8_OK;
}
static RCore core_of(const qvb8r_pack *w) {
    return RCore{w->words, w->tile_off, w->states, w->tiles, w->blocks, w->tab, w->perm, w->min_s, w->tau_s, w->drow,
                 (int)w->Q, (int)w->P};
}

template <int MP, typename XT, bool WROUND>
static void launch_mm(const RCore &c, int nb, const void *X, int M, float *Y, cudaStream_t st) {
    qvb8r_kernel<MP, XT, WROUND><<<nb * (R_WPB / R_RESTORE_WARPS), 32 * R_RESTORE_WARPS, 0, st>>>(c, reinterpret_cast<const XT *>(X), M, Y);
}
template <typename XT, bool WROUND>
static void launch_mm_mp(const RCore &c, int nb, const void *X, int M, float *Y, cudaStream_t st) {
    if (M <= 1) launch_mm<1, XT, WROUND>(c, nb, X, M, Y, st);
    else if (M <= 2) launch_mm<2, XT, WROUND>(c, nb, X, M, Y, st);
    else if (M <= 4) launch_mm<4, XT, WROUND>(c, nb, X, M, Y, st);
    else if (M <= 8) launch_mm<8, XT, WROUND>(c, nb, X, M, Y, st);
    else launch_mm<16, XT, WROUND>(c, nb, X, M, Y, st);
}
// The tensor-core product where it holds the contract: fp16 X with the rounded band value, bf16 / fp32 X of up to 8 tokens
// with the unrounded one; X 16-byte aligned (its fragments are 16-byte loads).
static bool launch_mma(const RCore &c, int nb, const void *X, int x_dtype, int M, int round_w, float *Y, cudaStream_t st) {
    // (fp32 activations cost three operands and their splitting: 5120 x 5120, 2 / 4 / 5 tokens lane by lane 49 / 65 / 101 us,
    // here 69; bf16 61 / 95 / 113 us and 53)
    if (M < (x_dtype == QVB8_F32 ? 5 : 2) || !aligned(X, 16)) return false;
    const int grid = nb * (R_WPB / RM_WARPS), thr = 32 * RM_WARPS;
    if (x_dtype == QVB8_F16 && round_w) {
        if (M <= 16) qvb8r_mma_kernel<0, 1><<<grid, thr, 0, st>>>(c, X, M, Y);
        else if (M <= 32) qvb8r_mma_kernel<0, 2><<<grid, thr, 0, st>>>(c, X, M, Y);
        else qvb8r_mma_kernel<0, 3><<<grid, thr, 0, st>>>(c, X, M, Y);
        return true;
    }
    if (round_w || M > 8) return false;
    if (x_dtype == QVB8_BF16) qvb8r_mma_kernel<1, 1><<<grid, thr, 0, st>>>(c, X, M, Y);
    else if (x_dtype == QVB8_F32) qvb8r_mma_kernel<2, 1><<<grid, thr, 0, st>>>(c, X, M, Y);
    else return false;
    return true;
}

}  // namespace qv

QV_API int qvb8r_ids(const qvb8r_pack *w, int16_t *out, void *stream) {
    using namespace qv;
    if (int rc = check_rpack(w, "qvb8r_ids")) return rc;
    if (int rc = check_device("qvb8r_ids")) return rc;
    if (!out) return fail(QVB8_ERR_ARG, "qvb8r_ids: null output");
    if (w->n_blocks == 0) return QVB8_OK;
    qvb8r_restore_kernel<0, int16_t><<<(unsigned)w->n_blocks * (R_WPB / R_RESTORE_WARPS), 32 * R_RESTORE_WARPS, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        core_of(w), 0, -1, out);
    return cuda_status("qvb8r_ids");
}

QV_API int qvb8r_decode(const qvb8r_pack *w, int out_dtype, void *out, int64_t b0, int64_t nb, int64_t row_base,
                        void *stream) {
    using namespace qv;
    if (int rc = check_rpack(w, "qvb8r_decode")) return rc;
    if (int rc = check_device("qvb8r_decode")) return rc;
    if (!out) return fail(QVB8_ERR_ARG, "qvb8r_decode: null output");
    if (b0 < 0 || nb < 0 || b0 + nb > w->n_blocks) return fail(QVB8_ERR_ARG, "qvb8r_decode: block range out of bounds");
    if (nb == 0) return QVB8_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const RCore c = core_of(w);
    if (out_dtype == QVB8_F16)
        qvb8r_restore_kernel<1, __half><<<(unsigned)nb * (R_WPB / R_RESTORE_WARPS), 32 * R_RESTORE_WARPS, 0, st>>>(c, (int)b0, row_base, reinterpret_cast<__half *>(out));
    else if (out_dtype == QVB8_BF16)
        qvb8r_restore_kernel<1, __nv_bfloat16><<<(unsigned)nb * (R_WPB / R_RESTORE_WARPS), 32 * R_RESTORE_WARPS, 0, st>>>(c, (int)b0, row_base, reinterpret_cast<__nv_bfloat16 *>(out));
    else if (out_dtype == QVB8_F32)
        qvb8r_restore_kernel<1, float><<<(unsigned)nb * (R_WPB / R_RESTORE_WARPS), 32 * R_RESTORE_WARPS, 0, st>>>(c, (int)b0, row_base, reinterpret_cast<float *>(out));
    else
        return fail(QVB8_ERR_ARG, "qvb8r_decode: bad output dtype");
    return cuda_status("qvb8r_decode");
}

QV_API int qvb8r_small_m(const qvb8r_pack *w, const void *X, int x_dtype, int64_t M, int round_w_fp16, float *Y,
                         void *stream) {
    using namespace qv;
    if (int rc = check_rpack(w, "qvb8r_small_m")) return rc;
    if (int rc = check_device("qvb8r_small_m")) return rc;
    if (!X || !Y) return fail(QVB8_ERR_ARG, "qvb8r_small_m: null argument");
    if (M < 1 || M > 16) return fail(QVB8_ERR_ARG, "qvb8r_small_m: M=%lld is outside 1..16", (long long)M);
    if (w->n_blocks == 0) return QVB8_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const RCore c = core_of(w);
    const int nb = (int)w->n_blocks;
    if (launch_mma(c, nb, X, x_dtype, (int)M, round_w_fp16, Y, st)) return cuda_status("qvb8r_small_m");
    if (x_dtype == QVB8_F32) {
        if (round_w_fp16) launch_mm_mp<float, true>(c, nb, X, (int)M, Y, st); else launch_mm_mp<float, false>(c, nb, X, (int)M, Y, st);
    } else if (x_dtype == QVB8_BF16) {
        if (round_w_fp16) launch_mm_mp<__nv_bfloat16, true>(c, nb, X, (int)M, Y, st); else launch_mm_mp<__nv_bfloat16, false>(c, nb, X, (int)M, Y, st);
    } else if (x_dtype == QVB8_F16) {
        if (round_w_fp16) launch_mm_mp<__half, true>(c, nb, X, (int)M, Y, st); else launch_mm_mp<__half, false>(c, nb, X, (int)M, Y, st);
    } else {
        return fail(QVB8_ERR_ARG, "qvb8r_small_m: bad X dtype");
    }
    return cuda_status("qvb8r_small_m");
}

QV_API int qvb8r_fix_escapes(const float *X, const int64_t *uq, const int64_t *ptr, const int64_t *ec, const float *ed,
                             float *Y, int64_t U, int64_t M, int64_t P, int64_t Q, void *stream) {
    using namespace qv;
    if (int rc = check_device("qvb8r_fix_escapes")) return rc;
    if (U == 0) return QVB8_OK;
    if (!X || !uq || !ptr || !ec || !ed || !Y || U < 0 || M <= 0 || P <= 0 || Q <= 0)
        return fail(QVB8_ERR_ARG, "qvb8r_fix_escapes: bad argument");
    const int64_t n = U * M;
    qvb8r_fix_kernel<<<(unsigned)((n + 127) / 128), 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(X, uq, ptr, ec, ed, Y, U,
                                                                                                      (int)M, (int)P, (int)Q);
    return cuda_status("qvb8r_fix_escapes");
}

namespace qv {
template <typename XT>
static int launch_finish(const void *X, const int *row_ptr, const int64_t *ec, const float *ed, const float *Y, void *out, int out_dtype,
                         int64_t M, int P, int Q, cudaStream_t st) {
    const dim3 g((unsigned)((Q + 127) / 128), (unsigned)M);
    const XT *x = reinterpret_cast<const XT *>(X);
    if (out_dtype == QVB8_F16) qvb8r_finish_kernel<XT, __half><<<g, 128, 0, st>>>(x, row_ptr, ec, ed, Y, reinterpret_cast<__half *>(out), P, Q);
    else if (out_dtype == QVB8_BF16) qvb8r_finish_kernel<XT, __nv_bfloat16><<<g, 128, 0, st>>>(x, row_ptr, ec, ed, Y, reinterpret_cast<__nv_bfloat16 *>(out), P, Q);
    else if (out_dtype == QVB8_F32) qvb8r_finish_kernel<XT, float><<<g, 128, 0, st>>>(x, row_ptr, ec, ed, Y, reinterpret_cast<float *>(out), P, Q);
    else return fail(QVB8_ERR_ARG, "qvb8r_finish: bad output dtype");
    return cuda_status("qvb8r_finish");
}
}  // namespace qv

QV_API int qvb8r_finish(const void *X, int x_dtype, const int32_t *row_ptr, const int64_t *ec, const float *ed, const float *Y, void *out,
                        int out_dtype, int64_t M, int64_t P, int64_t Q, void *stream) {
    using namespace qv;
    if (int rc = check_device("qvb8r_finish")) return rc;
    if (!X || !row_ptr || !Y || !out || M <= 0 || M > 65535 || P <= 0 || Q <= 0 || P > 0x7fffffff || Q > 0x7fffffff)
        return fail(QVB8_ERR_ARG, "qvb8r_finish: bad argument");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (x_dtype == QVB8_F32) return launch_finish<float>(X, row_ptr, ec, ed, Y, out, out_dtype, M, (int)P, (int)Q, st);
    if (x_dtype == QVB8_BF16) return launch_finish<__nv_bfloat16>(X, row_ptr, ec, ed, Y, out, out_dtype, M, (int)P, (int)Q, st);
    if (x_dtype == QVB8_F16) return launch_finish<__half>(X, row_ptr, ec, ed, Y, out, out_dtype, M, (int)P, (int)Q, st);
    return fail(QVB8_ERR_ARG, "qvb8r_finish: bad X dtype");
}

/* The `tc` product for up to 48 rows of fp16 X from one decoding. */
QV_API int qvb8r_tc_rows(const qvb8r_pack *w, const void *X, int64_t M, float *Y, void *stream) {
    using namespace qv;
    if (int rc = check_rpack(w, "qvb8r_tc_rows")) return rc;
    if (int rc = check_device("qvb8r_tc_rows")) return rc;
    if (!X || !Y) return fail(QVB8_ERR_ARG, "qvb8r_tc_rows: null argument");
    if (M < 2 || M > 48) return fail(QVB8_ERR_ARG, "qvb8r_tc_rows: M=%lld is outside 2..48", (long long)M);
    if (!aligned(X, 16)) return fail(QVB8_ERR_ALIGN, "qvb8r_tc_rows: X must be 16-byte aligned");
    if (w->n_blocks == 0) return QVB8_OK;
    launch_mma(core_of(w), (int)w->n_blocks, X, QVB8_F16, (int)M, 1, Y, reinterpret_cast<cudaStream_t>(stream));
    return cuda_status("qvb8r_tc_rows");
}

QV_API int qvb8r_embed_rows(const qvb8r_pack *w, const int64_t *rows, int64_t n, const int32_t *inv_perm,
                            const int32_t *row_tile, const int64_t *esc_ptr, const int32_t *esc_col, const float *esc_val,
                            float *out, void *stream) {
    using namespace qv;
    if (int rc = check_rpack(w, "qvb8r_embed_rows")) return rc;
    if (int rc = check_device("qvb8r_embed_rows")) return rc;
    if (n == 0) return QVB8_OK;
    if (!rows || !inv_perm || !row_tile || !esc_ptr || !out || n < 0)
        return fail(QVB8_ERR_ARG, "qvb8r_embed_rows: bad argument");
    qvb8r_embed_kernel<<<(unsigned)((n + R_WPB - 1) / R_WPB), 32 * R_WPB, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        core_of(w), rows, n, inv_perm, row_tile, esc_ptr, esc_col, esc_val, out);
    return cuda_status("qvb8r_embed_rows");
}
