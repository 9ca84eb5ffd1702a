// QVB8 prefill for sm_100a: Y (M, Q) fp32 = X (M, P) @ W^T for hundreds to thousands of tokens, the weight tile restored
// from the packed ids inside the kernel and contracted on the 5th-generation tensor cores (tcgen05.mma, accumulators in
// tensor memory).
//
// Replaces the reference's M > 8 path (formats/qvb8/backends/cuda_qvb8/qvb8_cuda.cu:1542-1671: restore the whole
// weight to fp16 in HBM, then cublasGemmEx fp16 x fp16 -> fp32).  Arithmetic here: the factored form the small-M
// kernels use, y[m, q] = tau_s[q] * sum_c x[m, c] * id[q, c] + min_s[q] * sum_c x[m, c]: the ids are exact in fp16, X is
// narrowed to saturated fp16 first (:761-841), products are exact and accumulated in fp32, so the weight enters
// un-narrowed (the reference rounds it once to fp16; both are within the certificate).  Rows wider than 11 bits, whose
// ids fp16 cannot hold exactly, are recomputed in fp32 afterwards; escapes are then added from the plan's differences
// (exact - band), one thread per (row, token) in stored order.
//
// Launches:
//   narrow   X -> saturated fp16, stored tile by tile in the order the tensor cores read it (256 tokens x 64 columns =
//            32 KB contiguous: [8-column group][token][8 values]), plus partial sums of the narrowed values
//   main     a CTA owns 128 output rows (in the plan's width-sorted order) and 256 tokens; K advances in blocks of 64
//            columns.  The weights reach the tensor cores through TENSOR MEMORY (tcgen05.mma with the A operand in
//            tensor memory), so shared memory carries only the activations and the packed ids:
//              unpack warps (PF_G groups of four; three by default).  A thread owns one row = one lane of tensor
//                          memory; group g takes the pairs of K blocks g, g + PF_G, ...  A warp fetches its own 32
//                          rows x 128 ids with 16-byte cp.async (eight lanes per row: whole lines, not one line per
//                          lane) into a private buffer whose row stride is an odd multiple of 16 bytes; then every
//                          thread reads its row (nb 16-byte vectors), turns pairs of ids into fp16 integers (one
//                          window, mask | 0x6400.., one HFMA2 for 6..8 bits) and stores 2 x 32 registers with
//                          tcgen05.st into its lane of one of four 64-column weight slots
//              copy warp   one thread: one 32 KB bulk copy per K block for the activations (four stages, freed in pairs)
//              MMA warp    one thread: waits for a weight slot and an activation stage, issues four tcgen05.mma
//                          (128 x 256 x 16, accumulator in columns 0..255) per K block and, per pair of K blocks,
//                          commits them to the barriers that free the two stages and the slot
//            At the end eight of the unpack warps read the accumulator with tcgen05.ld, apply tau_s, min_s * sum(x)
//            and write Y.
//   wide, escapes   the corrections described above
//
// Waits are bounded: a wait that runs out raises an abort flag and the error word, everybody falls through, copies in
// flight are given time to land, and the tensor memory is released before the CTA exits.
#include "common.cuh"
#include "plan.cuh"

namespace qv {

constexpr int PF_TOK = 256;                // tokens per CTA = MMA N
constexpr int PF_BK = 64;                  // columns per stage
#ifndef QVB8_PF_GROUPS
#define QVB8_PF_GROUPS 3
#endif
constexpr int PF_G = QVB8_PF_GROUPS;       // unpack groups of four warps (a group owns whole pairs of K blocks)
constexpr int PF_UW = 4 * PF_G;            // unpack warps
constexpr int PF_UNPACK = 32 * PF_UW;      // unpack threads
constexpr int PF_THREADS = PF_UNPACK + 64; // + copy warp + MMA warp
constexpr int PF_NBUF = PF_G <= 2 ? 2 : 1; // buffers of packed ids per unpack warp
constexpr int PF_EG = PF_G >= 4 ? 4 : 2;   // groups of four warps that share the epilogue
// registers: the allocation is per four warps, so 14 warps (three groups) may use 128 each, 18 warps only 96
constexpr int PF_B_BYTES = PF_TOK * PF_BK * 2;      // 32 KB
constexpr int PF_SPIN = 1 << 22;
constexpr int PF_KS = 8;                   // column ranges of the partial activation sums
constexpr int PF_EXACT_BITS = 11;          // ids up to this width are exact in fp16
constexpr int PF_NBS = 4;                  // activation stages in shared memory (even: they are freed in pairs)
constexpr int PF_NU = 4;                   // weight units (pairs of K blocks, 64 columns) in tensor memory
constexpr int PF_VECS = 8;                 // 16-byte vectors of a pair of K blocks (128 ids) of the widest row that is copied
constexpr int PF_RAW_BUF = 32 * 16 * (PF_VECS | 1);   // bytes of one warp's buffer for a pair at the widest row stride
constexpr int PF_TMEM_COLS = 512;          // 256 accumulator columns + PF_NU * 64 weight columns
constexpr int PF_SMEM = PF_NBS * PF_B_BYTES + PF_UW * PF_NBUF * PF_RAW_BUF + 1024;

__device__ int g_prefill_error = 0;

__device__ __forceinline__ uint32_t pf_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool pf_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}
__device__ __noinline__ bool pf_wait_slow(uint32_t bar, uint32_t parity, volatile int *abort_flag, int code, unsigned backoff_ns) {
    uint64_t t0;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (int i = 0; i < PF_SPIN; ++i) {
        if (pf_try_wait(bar, parity)) return true;
        if (backoff_ns) __nanosleep(backoff_ns);         // a polling warp takes issue slots from the unpack warps of its scheduler
        if ((i & 7) == 7) {
            if (*abort_flag) return false;
            uint64_t t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t - t0 > 2000000000ull) break;
        }
    }
    *abort_flag = 1;
    atomicCAS(&g_prefill_error, 0, code);
    return false;
}
__device__ __forceinline__ bool pf_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int code, unsigned backoff_ns = 0) {
    if (pf_try_wait(bar, parity)) return true;
    return pf_wait_slow(bar, parity, abort_flag, code, backoff_ns);
}
// Polling wait (tuning switch 64) for the single threads whose wake-up latency is on the critical path (MMA issue,
// activation copies): mbarrier.test_wait never suspends the thread.  Bounded like pf_wait.  Measured slower than the
// suspending wait (0.63 against 0.50 ms per call on 5120 x 17408 x 2048): the polling warps take issue slots.
__device__ __noinline__ bool pf_wait_poll(uint32_t bar, uint32_t parity, volatile int *abort_flag, int code) {
    uint64_t t0 = 0;
    for (int i = 0; i < (1 << 28); ++i) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((i & 255) == 255) {
            if (*abort_flag) return false;
            uint64_t t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            if (t - t0 > 2000000000ull) break;
        }
    }
    *abort_flag = 1;
    atomicCAS(&g_prefill_error, 0, code);
    return false;
}
__device__ __forceinline__ void pf_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

// Shared-memory matrix descriptor, K-major, no swizzle: core matrices of 8 rows x 16 bytes stored as 128 contiguous
// bytes; `sbo` bytes between core matrices along the rows, `lbo` bytes between core matrices along K; version 1.
__device__ __forceinline__ uint64_t pf_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// Position (in halves) of activation (token n, column c) in the tiled fp16 copy; nkb = P / 64.  Inside every group of
// four columns the order is 0, 2, 1, 3: the unpack threads build fp16 pairs from ids two columns apart (for 6..8-bit
// rows such a pair comes out of ONE 32-bit window), so a 32-bit operand register holds columns (k, k + 2) and the
// activations follow the same order.
__host__ __device__ __forceinline__ int pair_order(int a) { return (((a >> 1) ^ a) & 1) ? (a ^ 3) : a; }
__host__ __device__ __forceinline__ int64_t x16_index(int n, int c, int nkb) {
    return ((((int64_t)(n >> 8) * nkb + (c >> 6)) * 8 + ((c >> 3) & 7)) * PF_TOK + (n & 255)) * 8 + pair_order(c & 7);
}

struct PrefillParams {
    const uint8_t *ids;
    const float *min_s, *tau_s;
    const uint8_t *nbits;
    const int64_t *bit_off;
    const TileDesc *tiles;     // the plan's width-sorted row order, 16 rows per entry
    int max_tiles;
    const __half *X16;         // tiled saturated fp16 copy of X, tokens padded to a multiple of 256 with zeros
    const float *sumx;         // (PF_KS, Mpad) partial sums of the narrowed activations
    float *Y;                  // (M, Q)
    int Q, P, M, Mpad;
    int debug;                 // tuning aid: 1 = no unpack arithmetic, 2 = no activation copies, 4 = no weight fetch, 8 = no tensor-memory stores, 16 = no MMAs, 48 = no MMAs and plain barrier arrivals instead of commits, 64 = polling waits
};

// The output row of a slot of the plan's order, -1 for padding.
__device__ __forceinline__ int slot_row(const PrefillParams &p, int slot) {
    if ((slot >> 4) >= p.max_tiles) return -1;
    const TileDesc *td = p.tiles + (slot >> 4);
    return (slot & 15) < __ldg(&td->cnt) ? __ldg(&td->row[slot & 15]) : -1;
}

// 32-bit word K of the row words held as 16-byte vectors.
template <int K, int NV>
__device__ __forceinline__ uint32_t word32(const uint4 (&q)[NV]) {
    static_assert(K >= 0 && K < 4 * NV, "word outside the pair");
    return (K & 3) == 0 ? q[K >> 2].x : (K & 3) == 1 ? q[K >> 2].y : (K & 3) == 2 ? q[K >> 2].z : q[K >> 2].w;
}

// 32 bits of the pair's bit string such that bit `G` of the string lands at bit `AT` of the result; the caller uses
// the SPAN bits from AT on.
template <int G, int AT, int SPAN, int NV>
__device__ __forceinline__ uint32_t window(const uint4 (&q)[NV]) {
    constexpr int P0 = G - AT;                            // string position of result bit 0
    if constexpr (P0 < 0) return word32<0, NV>(q) << (-P0);
    else {
        constexpr int idx = P0 >> 5, sh = P0 & 31;
        if constexpr (sh == 0) return word32<idx, NV>(q);
        else if constexpr (sh + AT + SPAN <= 32) return word32<idx, NV>(q) >> sh;
        else return __funnelshift_r(word32<idx, NV>(q), word32<idx + 1, NV>(q), sh);
    }
}

// The 64 ids of K block H (0 / 1) of a pair of K blocks -> 32 registers of two fp16 integers each.  Register c holds
// columns k and k + 2, k = 4 * (c >> 1) + (c & 1) (see pair_order).  q holds the 128 ids (NB 16-byte vectors).
//   6..8 bits: ONE window puts id k at bit E = 16 - 2 NB and id k + 2 at bit 16; mask | 0x64006400 gives the fp16
//              numbers 1024 + id * 2^E and 1024 + id; one HFMA2 scales and removes the 1024 (exact)
//   others:    two windows, two masks, one subtraction of 1024
// The shifts and logic operations run on the half-rate integer pipe, which is what bounds this kernel: two instead of
// four of them per pair for the common widths.
// The constants of a width, read once per thread from a shared-memory table through volatile loads: as literals the
// compiler re-creates them with a move in front of every use, which doubles the work of the integer pipe.
struct PairConst {
    uint32_t mask;      // (m << E) | (m << 16) for 6..8 bits; m for the others
    uint32_t mask_hi;   // m << 16
    uint32_t k64;       // 0x64006400
    uint32_t scale;     // half2 (2^-E, 1)
    uint32_t bias;      // half2 (-1024 * 2^-E, -1024)
};
__device__ __forceinline__ PairConst pair_const_of(int nb) {
    const uint32_t m = (1u << nb) - 1u;
    const int e = (nb >= 6 && nb <= 8) ? 16 - 2 * nb : 0;
    PairConst c;
    c.mask = (nb >= 6 && nb <= 8) ? ((m << e) | (m << 16)) : m;
    c.mask_hi = m << 16;
    c.k64 = 0x64006400u;
    const __half2 sc = __floats2half2_rn(1.0f / (float)(1 << e), 1.0f), bi = __floats2half2_rn(-1024.0f / (float)(1 << e), -1024.0f);
    c.scale = *reinterpret_cast<const uint32_t *>(&sc);
    c.bias = *reinterpret_cast<const uint32_t *>(&bi);
    return c;
}

template <int NB, int H, int I = 0>
__device__ __forceinline__ void unpack64(const uint4 (&q)[NB], const PairConst &pc, uint32_t (&out)[32]) {
    if constexpr (I < 32) {
        constexpr int k = 4 * (I >> 1) + (I & 1);
        constexpr int G0 = (H * 64 + k) * NB, G1 = G0 + 2 * NB;
        uint32_t u;
        if constexpr (NB >= 6 && NB <= 8) {
            constexpr int E = 16 - 2 * NB;
            u = (window<G0, E, 16 - E + NB, NB>(q) & pc.mask) | pc.k64;
        } else {
            u = (window<G1, 16, NB, NB>(q) & pc.mask_hi) | ((window<G0, 0, NB, NB>(q) & pc.mask) | pc.k64);
        }
        const __half2 v = __hfma2(*reinterpret_cast<const __half2 *>(&u), *reinterpret_cast<const __half2 *>(&pc.scale),
                                  *reinterpret_cast<const __half2 *>(&pc.bias));
        out[I] = *reinterpret_cast<const uint32_t *>(&v);
        unpack64<NB, H, I + 1>(q, pc, out);
    }
}

// K block H of a row of width NB: the vectors it touches from the warp's buffer, 64 ids to registers.
template <int NB, int H>
__device__ __forceinline__ void unpack_row_half(const uint4 *__restrict__ src, const PairConst &pc, uint32_t (&out)[32]) {
    uint4 q[NB];
    // vectors of half H (a window of the second half may start in the last word of the first)
    constexpr int V0 = H == 0 ? 0 : (NB / 2 > 0 ? NB / 2 - 1 : 0), V1 = H == 0 ? (NB + 1) / 2 + (NB > 1 ? 1 : 0) : NB;
#pragma unroll
    for (int i = V0; i < (V1 < NB ? V1 : NB); ++i) q[i] = src[i];
    unpack64<NB, H>(q, pc, out);
}

// 32 registers -> 32 columns of tensor memory, lane = this thread's lane of the warp's quarter.
__device__ __forceinline__ void tmem_store32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
        :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
           "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
           "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
           "r"(r[30]), "r"(r[31])
        : "memory");
}

// Row of the CTA's tile: output row, width, first byte, and how its ids reach the unpack thread.
//   mode 0: nothing to contract (padding, or a row wider than fp16 holds exactly: recomputed afterwards)
//   mode 1: 16-byte copies into the warp's buffer (widths 1..8, row start 16-byte aligned);  mode 2: id by id from global memory
struct RowInfo { int row, nb, mode; int64_t bit0; };
__device__ __forceinline__ RowInfo row_info(const PrefillParams &p, int slot) {
    RowInfo r;
    r.row = slot_row(p, slot);
    r.nb = r.row >= 0 ? __ldg(p.nbits + r.row) : 0;
    r.bit0 = r.row >= 0 ? __ldg(p.bit_off + r.row) : 0;
    const bool bulk_ok = (r.bit0 & 127) == 0 && (reinterpret_cast<uintptr_t>(p.ids) & 15) == 0 && r.nb >= 1 && r.nb <= PF_VECS;
    r.mode = (r.row < 0 || r.nb > PF_EXACT_BITS || r.nb < 1) ? 0 : (bulk_ok ? 1 : 2);
    return r;
}

// The rare rows that are read id by id (11 bits wide, or not starting on 16 bytes): one K block to registers.
__device__ __noinline__ void unpack_generic(const uint8_t *__restrict__ ids, int64_t bit0, int nb, int kb, int centre, uint32_t *out) {
    for (int i = 0; i < 32; ++i) {
        const int col = kb * PF_BK + 4 * (i >> 1) + (i & 1);          // register i holds columns col, col + 2
        const int a0 = (int)field_bytes(ids, bit0 + (int64_t)col * nb, nb) - centre;
        const int a1 = (int)field_bytes(ids, bit0 + (int64_t)(col + 2) * nb, nb) - centre;
        const __half2 hh = __halves2half2(__short2half_rn((short)a0), __short2half_rn((short)a1));
        out[i] = *reinterpret_cast<const uint32_t *>(&hh);
    }
}

// K block H of this thread's pair -> 32 registers.  No tensor-memory access in here: rows of different widths or
// modes diverge inside, and tcgen05.st is a warp-wide instruction that every lane must reach together.
template <int H>
__device__ __forceinline__ void unpack_half(const PrefillParams &p, const RowInfo &me, const uint4 *__restrict__ src, const PairConst &pc,
                                            int kb, int nkb, uint32_t (&out)[32], int centre = 0) {
    if (me.mode == 1) {
        switch (me.nb) {
        case 1: unpack_row_half<1, H>(src, pc, out); break;
        case 2: unpack_row_half<2, H>(src, pc, out); break;
        case 3: unpack_row_half<3, H>(src, pc, out); break;
        case 4: unpack_row_half<4, H>(src, pc, out); break;
        case 5: unpack_row_half<5, H>(src, pc, out); break;
        case 6: unpack_row_half<6, H>(src, pc, out); break;
        case 7: unpack_row_half<7, H>(src, pc, out); break;
        default: unpack_row_half<8, H>(src, pc, out); break;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) out[i] = 0u;
        if (me.mode == 2 && kb < nkb) {                  // through a stack buffer, so that `out` stays in registers
            uint32_t tmp[32];
            unpack_generic(p.ids, me.bit0, me.nb, kb, centre, tmp);
#pragma unroll
            for (int i = 0; i < 32; ++i) out[i] = tmp[i];
        }
    }
}

__global__ void __maxnreg__(PF_G == 2 ? 168 : PF_G == 3 ? 128 : 96) prefill_kernel(const PrefillParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];         // PF_NBS activation stages, then 8 warps x 2 buffers of packed ids
    __shared__ alignas(8) uint64_t a_full[PF_NU];             // a pair of K blocks of weights is in tensor memory
    __shared__ alignas(8) uint64_t a_empty[PF_NU];            // ... and the MMAs that read it have completed
    __shared__ alignas(8) uint64_t b_full[PF_NBS];            // a stage's activations have landed
    __shared__ alignas(8) uint64_t b_empty[PF_NBS / 2];       // ... and the MMAs that read a PAIR of stages have completed
    __shared__ alignas(8) uint64_t all_done;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_word, nb_max;
    __shared__ const uint8_t *row_src[128];                   // first byte of each row of the tile (mode 1 rows)
    __shared__ int row_nb1[128];                              // its width, 0 unless mode 1
    __shared__ float sx[PF_TOK];                              // sum of the narrowed activations of each token of the tile
    __shared__ PairConst ctab[11];                            // per width, see PairConst
    volatile int *abort_flag = &abort_word;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slot0 = blockIdx.x * 128;                 // first row slot (plan order) of this CTA
    const int n0 = blockIdx.y * PF_TOK;
    // surplus tiles at the end of the plan's table are empty: a CTA that starts in them has no rows at all
    if ((slot0 >> 4) >= p.max_tiles || __ldg(&p.tiles[slot0 >> 4].cnt) == 0) return;
    if (tid == 0) {
        for (int s = 0; s < PF_NU; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(pf_smem(&a_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&a_empty[s])) : "memory");
        }
        for (int s = 0; s < PF_NBS; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&b_full[s])) : "memory");
            if (s < PF_NBS / 2) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&b_empty[s])) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&all_done)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        abort_word = 0;
        nb_max = 0;
        for (int nb = 1; nb <= PF_VECS; ++nb) ctab[nb] = pair_const_of(nb);
    }
    if (warp == 0) {                                    // one warp allocates (and later frees) the tensor-memory columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(pf_smem(&tmem_base)), "r"((uint32_t)PF_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    __syncthreads();
    // the widest copied row fixes the row stride of the warps' buffers
    RowInfo me{};
    if (tid < 128) {
        me = row_info(p, slot0 + tid);
        const int nb1 = me.mode == 1 ? me.nb : 0;
        row_src[tid] = p.ids + (me.bit0 >> 3);
        row_nb1[tid] = nb1;
        const int wmax = __reduce_max_sync(0xffffffffu, nb1);
        if (lane == 0) atomicMax(&nb_max, wmax);
    } else if (tid < PF_UNPACK) {
        me = row_info(p, slot0 + (tid & 127));
    }
    if (tid < PF_TOK) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < PF_KS; ++k) t += __ldg(p.sumx + (int64_t)k * p.Mpad + n0 + tid);
        sx[tid] = t;
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;
    const int nkb = p.P / PF_BK;
    const int nunits = (nkb + 1) >> 1;                  // pairs of K blocks
    const int stride = 16 * (nb_max | 1);               // bytes per row in a warp's buffer: an odd multiple of 16

    if (warp < PF_UW) {
        // ------------------------------------------------------------------------------------------ unpack warps
        // group g = warp >> 2 takes the pairs of K blocks u = g, g + PF_G, ...; a thread owns row (warp & 3) * 32 + lane
        const int g = warp >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 256u;
        uint8_t *const mybuf = smem + PF_NBS * PF_B_BYTES + warp * PF_NBUF * PF_RAW_BUF;
        PairConst pc;
        {
            const volatile PairConst *vc = &ctab[me.mode == 1 ? me.nb : 1];
            pc.mask = vc->mask; pc.mask_hi = vc->mask_hi; pc.k64 = vc->k64; pc.scale = vc->scale; pc.bias = vc->bias;
        }
        // the warp's rows of a pair -> its buffer: eight lanes per row, 16 bytes each; one commit group per pair.  Per-lane constants: this lane's vector of rows 4 pp + lane / 8.
        uint32_t soff[8];
        int step[8];
#pragma unroll
        for (int pp = 0; pp < 8; ++pp) {
            const int rr = (warp & 3) * 32 + pp * 4 + (lane >> 3);
            step[pp] = 16 * row_nb1[rr];
            soff[pp] = (uint32_t)(row_src[rr] - p.ids) + (uint32_t)((lane & 7) * 16);
        }
        const uint32_t dst0 = pf_smem(mybuf) + (uint32_t)((lane >> 3) * stride + (lane & 7) * 16);
        auto fetch = [&](int u_, int b_) {
            if (u_ < nunits && !(p.debug & 4)) {
                const int nkv = min(2, nkb - 2 * u_);
                const uint32_t dst = dst0 + (uint32_t)(b_ * PF_RAW_BUF);
#pragma unroll
                for (int pp = 0; pp < 8; ++pp) {
                    // a last, single K block is 8 * nb bytes: rounded up to 16 (a row is followed by the next row or by
                    // the buffer's 8 bytes of padding)
                    const int nbr = step[pp] >> 4;
                    const int nv = nkv == 2 ? nbr : (8 * nbr + 15) >> 4;
                    const uint8_t *src = p.ids + soff[pp] + (int64_t)u_ * step[pp];
                    if ((lane & 7) < nv)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + (uint32_t)(pp * 4 * stride)), "l"(src) : "memory");
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        fetch(g, 0);
        // every wait result is made warp-uniform: the tensor-memory stores below need the whole warp
        int it = 0;
        for (int u = g; u < nunits; u += PF_G, ++it) {
            const int kb0 = 2 * u;
            const int b = PF_NBUF == 2 ? (it & 1) : 0;
            if (PF_NBUF == 2) {                          // the next pair travels while this one is unpacked
                fetch(u + PF_G, b ^ 1);
                asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            }
            __syncwarp();
            const int slot = u & (PF_NU - 1), use = u / PF_NU;
            const uint32_t taddr = lane_base + (uint32_t)(slot * 64);
            const uint4 *src = reinterpret_cast<const uint4 *>(mybuf + b * PF_RAW_BUF + lane * stride);
            uint32_t out[32];
            if (p.debug & 1) {
#pragma unroll
                for (int i = 0; i < 32; ++i) out[i] = 0u;
            } else unpack_half<0>(p, me, src, pc, kb0, nkb, out);
            // only now is the slot needed: the MMAs that read its previous contents must have completed
            bool ok = true;
            if (use > 0) ok = pf_wait(pf_smem(&a_empty[slot]), (use - 1) & 1, abort_flag, 22);
            if (!__all_sync(0xffffffffu, ok)) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (!(p.debug & 8)) tmem_store32(taddr, out);
            if (!(p.debug & 1)) unpack_half<1>(p, me, src, pc, kb0 + 1, nkb, out);
            __syncwarp();                                // every lane has read its row: the buffer is free
            if (PF_NBUF == 1) fetch(u + PF_G, 0);
            if (!(p.debug & 8)) tmem_store32(taddr + 32, out);
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) pf_arrive(pf_smem(&a_full[slot]));
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    } else if (warp == PF_UW) {
        // ------------------------------------------------------------------------------------------ activation copies
        if (lane == 0) {
            const uint8_t *xsrc = reinterpret_cast<const uint8_t *>(p.X16) + (int64_t)blockIdx.y * nkb * PF_B_BYTES;
            bool alive = true;
            for (int kb = 0; kb < nkb && alive; ++kb) {
                const int s = kb % PF_NBS, u = kb / PF_NBS;
                if (u > 0 && (s & 1) == 0) alive = (p.debug & 64) ? pf_wait_poll(pf_smem(&b_empty[s >> 1]), (u - 1) & 1, abort_flag, 24) : pf_wait(pf_smem(&b_empty[s >> 1]), (u - 1) & 1, abort_flag, 24, 20);
                if (!alive) break;
                const uint32_t bar = pf_smem(&b_full[s]);
                if (p.debug & 2) { pf_arrive(bar); continue; }
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"((uint32_t)PF_B_BYTES) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                             :: "r"(pf_smem(smem + s * PF_B_BYTES)), "l"(xsrc + (int64_t)kb * PF_B_BYTES), "r"((uint32_t)PF_B_BYTES), "r"(bar)
                             : "memory");
            }
        }
    } else {
        // ------------------------------------------------------------------------------------------ MMA issue
        if (lane == 0) {
            // instruction descriptor: fp32 accumulate, fp16 x fp16, both operands K-major, N = 256, M = 128
            constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(PF_TOK >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
            // descriptors of the activation stages differ only in the start address field: one addition per MMA
            const uint64_t dbase = pf_desc(pf_smem(smem), PF_TOK * 16, 128);
            const uint32_t dlo0 = (uint32_t)dbase, dhi = (uint32_t)(dbase >> 32);
            bool alive = true;
            int s = 0;                                   // activation stage and the parity of its current use
            uint32_t bpar = 0;
            for (int kb = 0; kb < nkb && alive; ++kb) {
                const int unit = kb >> 1, slot = unit & (PF_NU - 1);
                if ((kb & 1) == 0) alive = (p.debug & 64) ? pf_wait_poll(pf_smem(&a_full[slot]), (uint32_t)(unit / PF_NU) & 1u, abort_flag, 25) : pf_wait(pf_smem(&a_full[slot]), (uint32_t)(unit / PF_NU) & 1u, abort_flag, 25, 32);
                if (alive) alive = (p.debug & 64) ? pf_wait_poll(pf_smem(&b_full[s]), bpar, abort_flag, 26) : pf_wait(pf_smem(&b_full[s]), bpar, abort_flag, 26, 32);
                if (!alive) break;
                if ((kb & 1) == 0) asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t a_t = tmem + 256u + (uint32_t)(slot * 64 + (kb & 1) * 32);
                const uint32_t dlo = dlo0 + (uint32_t)(s * (PF_B_BYTES >> 4));
                if (!(p.debug & 16)) {
#pragma unroll
                    for (int kk = 0; kk < PF_BK / 16; ++kk) {
                        // 16 columns of K: 8 columns of tensor memory (two fp16 each) and two 8-column groups of activations
                        uint64_t db;
                        asm volatile("mov.b64 %0, {%1, %2};\n" : "=l"(db) : "r"(dlo + (uint32_t)(kk * ((2 * PF_TOK * 16) >> 4))), "r"(dhi));
                        const uint32_t accumulate = (kb > 0 || kk > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                            " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n}\n"
                            :: "r"(tmem), "r"(a_t + (uint32_t)(8 * kk)), "l"(db), "r"(IDESC), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                            : "memory");
                    }
                }
                if ((kb & 1) || kb == nkb - 1) {         // a pair of K blocks frees its two activation stages and its weight slot
                    if ((p.debug & 48) == 48) {          // tuning aid, only without MMAs: plain arrivals instead of commits
                        pf_arrive(pf_smem(&b_empty[s >> 1]));
                        pf_arrive(pf_smem(&a_empty[slot]));
                    } else {
                        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(pf_smem(&b_empty[s >> 1])) : "memory");
                        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(pf_smem(&a_empty[slot])) : "memory");
                    }
                }
                if (kb == nkb - 1)
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(pf_smem(&all_done)) : "memory");
                if (++s == PF_NBS) { s = 0; bpar ^= 1u; }
            }
        }
    }

    // ---- epilogue: tensor memory -> registers -> Y.  A warp reads the 32 lanes (warp & 3) * 32 ...; every group of four
    // warps takes its share of the 256 tokens.
    if (warp < 4 * PF_EG) {
        bool alive = !*abort_flag;
        if (alive) alive = pf_wait(pf_smem(&all_done), 0, abort_flag, 27, 100);
        alive = __all_sync(0xffffffffu, alive);          // tcgen05.ld is warp-wide: all lanes or none
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (alive) {
            const int lq = (warp & 3) * 32;
            const int cbeg = (warp >> 2) * (PF_TOK / PF_EG), cend = cbeg + PF_TOK / PF_EG;
            const int row = me.row;
            const float ts = row >= 0 ? __ldg(p.tau_s + row) : 0.f, ms = row >= 0 ? __ldg(p.min_s + row) : 0.f;
            for (int c0 = cbeg; c0 < cend; c0 += 32) {
                uint32_t d[32];
                const uint32_t taddr = tmem + ((uint32_t)lq << 16) + (uint32_t)c0;
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                    "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
                    : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]),
                      "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]), "=r"(d[16]),
                      "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]), "=r"(d[21]), "=r"(d[22]), "=r"(d[23]), "=r"(d[24]),
                      "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]), "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const int nn = n0 + c0 + j;
                    if (row >= 0 && nn < p.M) p.Y[(int64_t)nn * p.Q + row] = __fmaf_rn(ts, __uint_as_float(d[j]), ms * sx[c0 + j]);
                }
            }
        }
    }
    if (*abort_flag && warp == PF_UW) {                      // copies may still be in flight: let them land before the CTA goes
        uint64_t t0, t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
        for (int i = 0; i < (1 << 16); ++i) {
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t - t0 > 200000ull) break;
            __nanosleep(1000);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)PF_TMEM_COLS) : "memory");
}

// X (M, P) of any input type -> saturated fp16 in the tiled order, tokens padded to Mpad with zeros, and the sums of
// the narrowed values per token and column range (fixed order: a thread sums its groups in order, then eight warps are
// added in order).  With escapes a second, column-major copy (P, Mpad) is written for the escape pass.  Block = 32 tokens (lane) x 8 warps; blockIdx.y = column range.
__global__ void __launch_bounds__(256) prefill_narrow_kernel(const void *__restrict__ X, int x_dtype, int M, int Mpad, int P,
                                                             __half *__restrict__ X16, __half *__restrict__ X16T,
                                                             float *__restrict__ sumx) {
    __shared__ float part[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * 32 + lane;
    const int nkb = P / PF_BK, ngrp = P / 8;
    const int per = (ngrp + PF_KS - 1) / PF_KS;
    const int g0 = blockIdx.y * per, g1 = min(ngrp, g0 + per);
    float s = 0.f;
    for (int g = g0 + warp; g < g1; g += 8) {
        __half h[8];
        if (n < M) {
            const int64_t i = (int64_t)n * P + g * 8;
            if (x_dtype == QVB8_F32) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(X) + i));
                const float4 b = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(X) + i) + 1);
                h[0] = sat_half(a.x); h[1] = sat_half(a.y); h[2] = sat_half(a.z); h[3] = sat_half(a.w);
                h[4] = sat_half(b.x); h[5] = sat_half(b.y); h[6] = sat_half(b.z); h[7] = sat_half(b.w);
            } else if (x_dtype == QVB8_BF16) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const __nv_bfloat16 *>(X) + i));
                const __nv_bfloat16 *b = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
                for (int k = 0; k < 8; ++k) h[k] = sat_half(__bfloat162float(b[k]));
            } else {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(X) + i));
                const __half *b = reinterpret_cast<const __half *>(&v);
#pragma unroll
                for (int k = 0; k < 8; ++k) h[k] = sat_half(__half2float(b[k]));
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) s += __half2float(h[k]);
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) h[k] = __float2half_rn(0.f);
        }
        {
            const __half t[8] = {h[0], h[2], h[1], h[3], h[4], h[6], h[5], h[7]};       // see pair_order
            *reinterpret_cast<uint4 *>(X16 + x16_index(n, g * 8, nkb)) = *reinterpret_cast<const uint4 *>(t);
        }
        if (X16T) {                                      // column-major copy for the escape pass: tokens contiguous
#pragma unroll
            for (int k = 0; k < 8; ++k) X16T[(int64_t)(g * 8 + k) * Mpad + n] = h[k];
        }
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += part[k][lane];
        sumx[(int64_t)blockIdx.y * Mpad + n] = t;
    }
}

// Y[m, q] += sum over the escapes of row q of x16[m, col] * (exact - band), in stored order.  Block = 32 consecutive
// rows x 256 tokens.  Phase 1: warp w owns rows w, w + 8, w + 16, w + 24; a lane owns eight neighbouring tokens, so an
// escape costs the warp ONE 512-byte read of its column in the column-major copy and eight FMAs per lane.  Phase 2: the
// sums cross shared memory so that a thread owns one token and updates 128 contiguous bytes of Y.
__global__ void __launch_bounds__(256) prefill_escapes_kernel(const int *__restrict__ esc_ptr, const int *__restrict__ esc_col,
                                                              const float *__restrict__ esc_delta, const __half *__restrict__ X16T,
                                                              float *__restrict__ Y, int Q, int M, int Mpad) {
    __shared__ float E[256][33];
    const int q0 = blockIdx.x * 32, n0 = blockIdx.y * 256;
    const int qe = min(Q, q0 + 32);
    if (__ldg(esc_ptr + q0) == __ldg(esc_ptr + qe)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint4 *xt = reinterpret_cast<const uint4 *>(X16T + n0 + 8 * lane);       // Mpad is a multiple of 256
    const int64_t ld = Mpad >> 3;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int q = q0 + warp + 8 * j;
        float acc[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) acc[t] = 0.f;
        if (q < Q) {
            const int e0 = __ldg(esc_ptr + q), e1 = __ldg(esc_ptr + q + 1);
            for (int e = e0; e < e1; e += 2) {           // two at a time: the loads overlap
                const int ee = min(e + 1, e1 - 1);
                const float d0 = __ldg(esc_delta + e), d1 = e + 1 < e1 ? __ldg(esc_delta + ee) : 0.f;
                const uint4 v0 = __ldg(xt + (int64_t)__ldg(esc_col + e) * ld), v1 = __ldg(xt + (int64_t)__ldg(esc_col + ee) * ld);
                const __half2 *h0 = reinterpret_cast<const __half2 *>(&v0), *h1 = reinterpret_cast<const __half2 *>(&v1);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const float2 f = __half22float2(h0[t]);
                    acc[2 * t] = __fmaf_rn(f.x, d0, acc[2 * t]);
                    acc[2 * t + 1] = __fmaf_rn(f.y, d0, acc[2 * t + 1]);
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const float2 f = __half22float2(h1[t]);
                    acc[2 * t] = __fmaf_rn(f.x, d1, acc[2 * t]);
                    acc[2 * t + 1] = __fmaf_rn(f.y, d1, acc[2 * t + 1]);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) E[8 * lane + t][warp + 8 * j] = acc[t];
    }
    __syncthreads();
    const int n = n0 + threadIdx.x;
    if (n >= M) return;
    float *y = Y + (int64_t)n * Q + q0;
    const float *er = E[threadIdx.x];
    if ((Q & 3) == 0 && q0 + 32 <= Q) {
#pragma unroll
        for (int r = 0; r < 32; r += 4) {
            float4 v = *reinterpret_cast<float4 *>(y + r);
            v.x += er[r]; v.y += er[r + 1]; v.z += er[r + 2]; v.w += er[r + 3];
            *reinterpret_cast<float4 *>(y + r) = v;
        }
    } else {
        for (int r = 0; r < 32; ++r)
            if (q0 + r < Q) y[r] += er[r];
    }
}

// Rows wider than 11 bits: their ids are not exact in fp16 (integers above 2048 are not all representable), so the
// tensor-core result of such a row is replaced by an fp32 product over the row.  They are rare (rows dominated by
// outliers).  First a compact list of them, then one warp per (wide row, token).
__global__ void __launch_bounds__(256) prefill_wide_list_kernel(const uint8_t *__restrict__ nbits, int Q, int *__restrict__ list,
                                                                int *__restrict__ count) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < Q && __ldg(nbits + q) > PF_EXACT_BITS) list[atomicAdd(count, 1)] = q;
}
__global__ void __launch_bounds__(256) prefill_wide_rows_kernel(const PrefillParams p, const int *__restrict__ list,
                                                                const int *__restrict__ count) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m = blockIdx.y * 8 + warp;
    if (m >= p.M) return;
    const int n = *count;
    const int nkb = p.P / PF_BK;
    for (int wi = blockIdx.x; wi < n; wi += gridDim.x) {
        const int q = list[wi];
        const int nb = __ldg(p.nbits + q);
        const int64_t bit0 = __ldg(p.bit_off + q);
        const float ts = __ldg(p.tau_s + q), ms = __ldg(p.min_s + q);
        float a = 0.f;
        for (int c = lane; c < p.P; c += 32)
            a = __fmaf_rn(__half2float(p.X16[x16_index(m, c, nkb)]), band(field_bytes(p.ids, bit0 + (int64_t)c * nb, nb), ts, ms), a);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) p.Y[(int64_t)m * p.Q + q] = a;
    }
}

int prefill_error_word(int *out) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_prefill_error, sizeof(int)) != cudaSuccess) return cuda_status("qvb8_device_status");
    *out = v;
    return QVB8_OK;
}

static int g_prefill_debug = 0;

static int launch_prefill(const PrefillParams &prm, cudaStream_t st) {
    static thread_local int granted_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != granted_dev) {
        if (cudaFuncSetAttribute(prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM) != cudaSuccess)
            return cuda_status("qvb8_prefill: shared memory opt-in");
        granted_dev = dev;
    }
    const int slots = prm.max_tiles * 16;
    const dim3 grid((unsigned)((slots + 127) / 128), (unsigned)(prm.Mpad / PF_TOK));
    prefill_kernel<<<grid, PF_THREADS, PF_SMEM, st>>>(prm);
    return cuda_status("qvb8_prefill");
}

// ---------------------------------------------------------------------------------------------------------------
// Middle M (a dozen tokens to a few hundred): the same arithmetic and the same route of the weights -- packed ids ->
// registers -> tensor memory -> tcgen05.mma -- shaped for calls whose time is the weights', not the products'.
//
// What bounds it: the packed ids have to pass the unpack warps once (5 us of integer work per SM for 17408 x 5120) and
// come from HBM (12 us); the products are small.  The kernel above pads every call to 256 tokens and so moves 32 KB of
// activations per 64 columns and CTA through the L2 whatever M is, leaves SMs idle when a weight has fewer than 148 row
// tiles, and holds one buffer of ids per warp in flight.  Here
//   - the token tile is 16, 32, 64, 96 or 128 (one bulk copy per pair of K blocks),
//   - all (row tile, pair of K blocks) units of the product form one sequence that is cut into equal contiguous runs,
//     one per CTA; a tile cut by a run boundary is summed from fp32 partial tiles in scratch, in run order, by whichever
//     CTA finishes it last (a ticket per tile: nobody waits),
//   - two or three buffers of ids per unpack warp are in flight, and four to seven pairs of K blocks fit in tensor memory,
//   - additions inside the tensor cores truncate, so an accumulator sums a chunk of three pairs of K blocks only (384 columns)
//     and the unpack warps add the chunks up in fp32 registers; the operands are id - zero_id, so that the sum is the result
//     and not the larger of two numbers that cancel.  fp32 results over 4096 columns, 48 tokens: 1.3e-7 from 64 bits (2.5e-6
//     with one accumulator per run over plain ids, 6.0e-7 in the streaming kernel); activations of mean 1: 1.9e-7 (1.9e-4,
//     3.9e-5).  It costs 1 to 7 us a call: 17408 x 5120, 16 / 48 / 96 tokens 55 / 60 / 71 -> 57 / 66 / 78 us with the host,
//   - three launches with programmatic dependent launch: narrow (activations to fp16 tiles, sums, x_mode 1 prescale),
//     main, fix (escapes and rows wider than 11 bits).
// Measured against the streaming kernel (which lists its tokens as extra MMA groups and splits K for their activations)
// and the 256-token kernel, 17408 x 5120, us per call: see the dispatch in qvb8_small_m_ex.
constexpr int MD_CTAS = 148;               // runs at most
constexpr int MD_NARROW = 512;             // threads of a narrow block (one token)
constexpr int MD_CHUNK = 3;                // units a tensor-memory accumulator sums (a multiple of PF_G)
static_assert(MD_CHUNK % PF_G == 0, "every unpack group has the same number of units in a chunk");
template <int NTOK> struct MidCfg {
    static constexpr int ACC1 = NTOK <= 32 ? 32 : NTOK;                // columns of an accumulator
    static constexpr int ACC = 2 * ACC1;                               // two accumulators: one is summed while the other is drained
    static constexpr int PIECES = (NTOK / 8 + PF_G - 1) / PF_G;        // pieces of eight tokens that a group drains: g, g + PF_G, ...
    static constexpr int DRAIN_G = NTOK / 8 < PF_G ? NTOK / 8 : PF_G;  // groups with a piece
    static constexpr int NU = (512 - ACC) / 64;                        // weight slots (a pair of K blocks each)
    static constexpr int NBUF = NTOK <= 32 ? 3 : 2;                    // buffers of packed ids per unpack warp
    // activation stages (a pair of K blocks each): a stage's way round -- commit, copy thread, copy from L2, MMA warp --
    // takes 2 us, so few stages pace the kernel (four of them: 0.7 us per pair whatever the token tile)
    static constexpr int NBS = NTOK <= 16 ? 12 : NTOK <= 32 ? 7 : NTOK <= 64 ? 6 : NTOK <= 96 ? 4 : 3;
    static constexpr int B_BYTES = NTOK * 256;
    static constexpr int SMEM = NBS * B_BYTES + PF_UW * NBUF * PF_RAW_BUF + 1024;
};
struct MidParams {
    PrefillParams b;           // (X16: tiles of NTOK tokens; sumx: (Mpad) sums; M: tokens)
    const int *kexp;           // x_mode 1: token n was narrowed as x * 2^-kexp[n]
    int *ticket;               // one counter per (token tile, row tile), zeroed by the narrow kernel
    float *part;               // [CTA][2][NTOK][128] partial tiles: a CTA's first run segment, and its last
    int row_tiles, tok_tiles, units_tile;      // units per tile: pairs of K blocks
    int64_t units;             // all units
};
// A run [lo, hi) of units as segments: segment s covers units [ua, ub) of a tile.
struct MidSeg { int tile, ua, ub; };
__device__ __forceinline__ void mid_run(const MidParams &p, int cta, int64_t &lo, int64_t &hi) {
    lo = (int64_t)cta * p.units / gridDim.x;
    hi = (int64_t)(cta + 1) * p.units / gridDim.x;
}
__device__ __forceinline__ MidSeg mid_seg(const MidParams &p, int64_t at, int64_t hi) {
    MidSeg s;
    s.tile = (int)(at / p.units_tile);
    s.ua = (int)(at - (int64_t)s.tile * p.units_tile);
    s.ub = (int)min((int64_t)p.units_tile, s.ua + (hi - at));
    return s;
}
__device__ __forceinline__ bool mid_empty(const MidParams &p, int tile) {   // a row tile without rows (end of the plan's table)
    const int t16 = (tile % p.row_tiles) * 8;
    return t16 >= p.b.max_tiles || __ldg(&p.b.tiles[t16].cnt) == 0;
}

// Row r of a row tile, from its 16-row descriptor alone (one round trip) unless the row is read element by element.  Returns
// false for a tile without rows.
__device__ __forceinline__ bool mid_row(const MidParams &p, int tile, int r, RowInfo &me, float &ts, float &ms) {
    const int t0 = (tile % p.row_tiles) * 8, t16 = t0 + (r >> 4), s = r & 15;
    const TileDesc *d = p.b.tiles + min(t16, p.b.max_tiles - 1);
    const int cnt0 = t0 < p.b.max_tiles ? __ldg(&p.b.tiles[t0].cnt) : 0;
    const int cnt = __ldg(&d->cnt), nb = __ldg(&d->nb), row = __ldg(&d->row[s]);
    const uint32_t b16 = __ldg(&d->b16[s]);
    ts = __ldg(&d->ts[s]);
    ms = __ldg(&d->ms[s]);
    me.row = t16 < p.b.max_tiles && s < cnt ? row : -1;
    me.nb = me.row >= 0 ? nb : 0;
    me.bit0 = me.row >= 0 ? (int64_t)b16 * 128 : 0;
    if (me.row >= 0 && nb == 0) {                                      // widths outside 3..8, or not on 16 bytes
        me.nb = __ldg(p.b.nbits + me.row);
        me.bit0 = __ldg(p.b.bit_off + me.row);
    }
    const bool bulk_ok = (me.bit0 & 127) == 0 && (reinterpret_cast<uintptr_t>(p.b.ids) & 15) == 0 && me.nb >= 1 && me.nb <= PF_VECS;
    me.mode = (me.row < 0 || me.nb > PF_EXACT_BITS || me.nb < 1) ? 0 : (bulk_ok ? 1 : 2);
    return cnt0 > 0;
}

// X16 position (in halves): [token tile][K block][8-column group][token][8 values in pair order]
template <int NTOK>
__device__ __forceinline__ int64_t mid_x16(int n, int c, int nkb) {
    return ((((int64_t)(n / NTOK) * nkb + (c >> 6)) * 8 + ((c >> 3) & 7)) * NTOK + (n % NTOK)) * 8 + pair_order(c & 7);
}

// One lane of the (converged) warp, in the form that leaves the operands of what it issues in uniform registers.
__device__ __forceinline__ bool pf_elect() {
    uint32_t p;
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
    return p != 0;
}
// One decision for all unpack warps (and a barrier among them).
__device__ __forceinline__ bool mid_all(bool ok) {
    uint32_t all;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.and.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(all) : "r"((uint32_t)ok), "n"(PF_UNPACK) : "memory");
    return all != 0;
}

template <int NTOK>
__global__ void __maxnreg__(128) mid_kernel(const MidParams p) {
    using C = MidCfg<NTOK>;
    extern __shared__ __align__(1024) uint8_t smem[];         // activation stages, then the unpack warps' buffers of ids
    __shared__ alignas(8) uint64_t a_full[C::NU], a_empty[C::NU];     // a weight slot is filled / its MMAs have completed
    __shared__ alignas(8) uint64_t b_full[C::NBS], b_empty[C::NBS];   // an activation stage has landed / been read
    __shared__ alignas(8) uint64_t acc_full[2], acc_empty[2];         // a chunk's sums are complete / have been read
    __shared__ uint32_t tmem_base;
    __shared__ int abort_word, last_part;
    __shared__ PairConst ctab[11];
    __shared__ uint2 s_src[PF_UW][32];                        // an unpack warp's rows: first byte, width (0: not copied)
    volatile int *abort_flag = &abort_word;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int64_t lo, hi;
    mid_run(p, blockIdx.x, lo, hi);
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    if (tid < 32) {                                           // the first tile's descriptors (3.2 KB) travel during the set-up
        const int t16 = (int)(lo / p.units_tile) % p.row_tiles * 8;
        const char *d = reinterpret_cast<const char *>(p.b.tiles + t16) + tid * 128;
        if (d < reinterpret_cast<const char *>(p.b.tiles + min(t16 + 8, p.b.max_tiles)))
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(d));
    }
    if (tid == 0) {
        for (int s = 0; s < C::NU; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;\n" ::"r"(pf_smem(&a_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&a_empty[s])) : "memory");
        }
        for (int s = 0; s < C::NBS; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&b_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&b_empty[s])) : "memory");
        }
        for (int s = 0; s < 2; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(pf_smem(&acc_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(pf_smem(&acc_empty[s])), "r"(4 * C::DRAIN_G) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        abort_word = 0;
        for (int nb = 1; nb <= PF_VECS; ++nb) ctab[nb] = pair_const_of(nb);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(pf_smem(&tmem_base)), "r"((uint32_t)PF_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_base;
    const int nkb = p.b.P / PF_BK;

    if (warp < PF_UW) {
        // ------------------------------------------------------------------------------ unpack warps, then the epilogue
        const int g = warp >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        uint8_t *const mybuf = smem + C::NBS * C::B_BYTES + warp * C::NBUF * PF_RAW_BUF;
        bool alive = true, waited = false;
        int i0 = 0, drained = 0;                         // units of the segments before this one; chunks drained so far
        int slot = g, use = 0;                           // slot of the group's next unit, and its use count
        __shared__ float s_sx[NTOK], s_sc[NTOK];         // the token tile's sums and 2^kexp
        __shared__ float s_ts[128], s_ms[128];           // the row tile's steps, middle values
        __shared__ int s_row[128];                       // ... and output rows
        for (int64_t at = lo; at < hi && alive;) {
            const MidSeg sg = mid_seg(p, at, hi);
            const int which = at > lo ? 1 : 0;           // the run's partial tiles: its first segment, its last
            at += sg.ub - sg.ua;
            RowInfo me;
            float my_ts, my_ms;
            if (!mid_row(p, sg.tile, (warp & 3) * 32 + lane, me, my_ts, my_ms)) continue;
            const int nb1 = me.mode == 1 ? me.nb : 0;
            const int stride = 16 * ((int)__reduce_max_sync(0xffffffffu, nb1) | 1);   // bytes per row of a buffer: an odd multiple of 16
            PairConst pc;
            {
                const volatile PairConst *vc = &ctab[me.mode == 1 ? me.nb : 1];
                pc.mask = vc->mask; pc.mask_hi = vc->mask_hi; pc.k64 = vc->k64; pc.scale = vc->scale; pc.bias = vc->bias;
            }
            // the operands are id - centre (zero_id): the centre joins the bias, exactly
            const int centre = me.mode == 0 ? 0 : (int)zero_id(my_ms, my_ts, me.nb);
            {
                const __half2 bias = __hsub2(*reinterpret_cast<const __half2 *>(&pc.bias), __half2half2(__int2half_rn(centre)));
                pc.bias = *reinterpret_cast<const uint32_t *>(&bias);
            }
            // a pair of K blocks of the warp's 32 rows -> a buffer: eight lanes per row, 16 bytes each
            // (where they come from waits in shared memory: sixteen registers that the sums need)
            s_src[warp][lane] = make_uint2((uint32_t)(me.bit0 >> 3), (uint32_t)nb1);
            __syncwarp();
            const uint32_t dst0 = pf_smem(mybuf) + (uint32_t)((lane >> 3) * stride + (lane & 7) * 16);
            auto fetch = [&](int u_, int b_) {
                if (u_ < sg.ub) {
                    const int nkv = min(2, nkb - 2 * u_);
                    const uint32_t dst = dst0 + (uint32_t)(b_ * PF_RAW_BUF);
#pragma unroll
                    for (int pp = 0; pp < 8; ++pp) {
                        const uint2 from = s_src[warp][pp * 4 + (lane >> 3)];
                        const int nbr = (int)from.y;     // (a last, single K block: 8 nb bytes, rounded up to 16)
                        const int nv = nkv == 2 ? nbr : (8 * nbr + 15) >> 4;
                        const uint8_t *src = p.b.ids + (from.x + (uint32_t)((lane & 7) * 16)) + (int64_t)u_ * (16 * nbr);
                        if ((lane & 7) < nv)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + (uint32_t)(pp * 4 * stride)), "l"(src) : "memory");
                    }
                }
                asm volatile("cp.async.commit_group;\n" ::: "memory");
            };
            const int ufirst = sg.ua + (g + PF_G - i0 % PF_G) % PF_G;              // unit i0 + (u - ua) belongs to group i % PF_G
            // The segment's sums of this thread's row, for the tokens of its group's pieces.  A chunk is drained a chunk late,
            // just before the group unpacks its first unit of the chunk that will overwrite the accumulator: the MMAs are long
            // done then, and nobody waits.
            float sum[C::PIECES][8];
#pragma unroll
            for (int j = 0; j < C::PIECES; ++j)
#pragma unroll
                for (int k = 0; k < 8; ++k) sum[j][k] = 0.f;
            const int chunks = (sg.ub - sg.ua + MD_CHUNK - 1) / MD_CHUNK, chunk0 = drained;
            auto drain = [&]() {
                const int buf = drained & 1, par = (drained >> 1) & 1;
                ++drained;
                if (g >= C::DRAIN_G) return true;
                if (!__all_sync(0xffffffffu, pf_wait(pf_smem(&acc_full[buf]), par, abort_flag, 47))) return false;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
                for (int j = 0; j < C::PIECES; ++j) {
                    const int c0 = (g + j * PF_G) * 8;
                    if (c0 >= NTOK) break;
                    float d[8];
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]), "=f"(d[4]), "=f"(d[5]), "=f"(d[6]), "=f"(d[7])
                                 : "r"(lane_base + (uint32_t)(buf * C::ACC1 + c0)));
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n"
                                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]), "+f"(d[4]), "+f"(d[5]), "+f"(d[6]), "+f"(d[7]) :: "memory");
#pragma unroll
                    for (int k = 0; k < 8; ++k) sum[j][k] += d[k];
                }
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) pf_arrive(pf_smem(&acc_empty[buf]));    // the chunk after next may overwrite the accumulator
                return true;
            };
#pragma unroll
            for (int k = 0; k < C::NBUF - 1; ++k) fetch(ufirst + k * PF_G, k);
            int b = 0, turn = 0;                         // turn: the group's units of this segment so far
            for (int u = ufirst; u < sg.ub; u += PF_G, ++turn) {
                fetch(u + (C::NBUF - 1) * PF_G, b == 0 ? C::NBUF - 1 : b - 1);
                constexpr int PER = MD_CHUNK / PF_G;     // the group's units of a chunk
                if (turn >= 2 * PER && turn % PER == 0 && !drain()) { alive = false; break; }
                asm volatile("cp.async.wait_group %0;\n" ::"n"(C::NBUF - 1) : "memory");
                __syncwarp();
                const uint32_t taddr = lane_base + (uint32_t)(C::ACC + slot * 64);
                const uint4 *src = reinterpret_cast<const uint4 *>(mybuf + b * PF_RAW_BUF + lane * stride);
                uint32_t out[32];
                unpack_half<0>(p.b, me, src, pc, 2 * u, nkb, out, centre);
                bool ok = true;                          // only now is the slot needed: its previous MMAs must have completed
                if (use > 0) ok = pf_wait(pf_smem(&a_empty[slot]), (use - 1) & 1, abort_flag, 42);
                if (!__all_sync(0xffffffffu, ok)) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                tmem_store32(taddr, out);
                unpack_half<1>(p.b, me, src, pc, 2 * u + 1, nkb, out, centre);
                __syncwarp();                            // (rows of different widths diverge in the unpacking)
                tmem_store32(taddr + 32, out);
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) pf_arrive(pf_smem(&a_full[slot]));
                b = b == C::NBUF - 1 ? 0 : b + 1;
                if ((slot += PF_G) >= C::NU) { slot -= C::NU; ++use; }
            }
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
            i0 += sg.ub - sg.ua;
            // ---- the segment's sums: a warp reads its quarter of the rows, the groups share the tokens 16 by 16
            if (!waited) { asm volatile("griddepcontrol.wait;\n" ::: "memory"); waited = true; }
            const bool whole = sg.ua == 0 && sg.ub == p.units_tile;
            const int n0 = (sg.tile / p.row_tiles) * NTOK, rl = (warp & 3) * 32 + lane, row = me.row;
            for (int n = tid; n < NTOK; n += PF_UNPACK) {
                s_sx[n] = __ldcg(p.b.sumx + n0 + n);
                s_sc[n] = __uint_as_float((uint32_t)(127 + __ldcg(p.kexp + n0 + n)) << 23);
            }
            if (g == 0) {
                s_row[rl] = row;
                s_ts[rl] = my_ts;
                s_ms[rl] = __fmaf_rn((float)centre, my_ts, my_ms);   // the band value that the centred ids count from
            }
            while (alive && drained < chunk0 + chunks) alive = drain();
            alive = mid_all(alive);                      // all unpack warps go on, or none (and the tables above are there)
            if (!alive) break;
            {
                const float ts = s_ts[rl], ms = s_ms[rl];
                float *part = p.part + ((int64_t)blockIdx.x * 2 + which) * NTOK * 128 + rl;
#pragma unroll
                for (int j = 0; j < C::PIECES; ++j) {
                    const int c0 = (g + j * PF_G) * 8;
                    if (c0 >= NTOK) break;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int n = n0 + c0 + k;
                        if (n < p.b.M) {
                            if (!whole) part[(int64_t)(c0 + k) * 128] = sum[j][k];
                            else if (row >= 0) p.b.Y[(int64_t)n * p.b.Q + row] = __fmaf_rn(ts, sum[j][k], ms * s_sx[c0 + k]) * s_sc[c0 + k];
                        }
                    }
                }
            }
            if (!whole) {
                // a shared tile: the last of its CTAs to get here adds the parts in run order and writes the results
                __threadfence();
                asm volatile("bar.sync 1, %0;\n" ::"n"(PF_UNPACK) : "memory");
                const int64_t t0 = (int64_t)sg.tile * p.units_tile, t1 = t0 + p.units_tile, G = gridDim.x;
                // the CTAs whose runs touch [t0, t1)
                int ca = (int)(t0 * G / p.units), cb = (int)((t1 - 1) * G / p.units);
                while ((int64_t)(ca + 1) * p.units / G <= t0) ++ca;
                while (ca > 0 && (int64_t)ca * p.units / G > t0) --ca;
                while ((int64_t)(cb + 1) * p.units / G < t1) ++cb;
                while ((int64_t)cb * p.units / G >= t1) --cb;
                if (tid == 0) last_part = atomicAdd(p.ticket + sg.tile, 1) == cb - ca;
                asm volatile("bar.sync 1, %0;\n" ::"n"(PF_UNPACK) : "memory");
                if (last_part) {                         // (written again only behind the next segment's barrier)
                    __threadfence();
                    // a warp takes two tokens, a lane four rows; the loads of eight parts are in flight together
                    const int first = (int64_t)ca * p.units / G < t0 ? 1 : 0;     // run ca holds the tile as its last segment, the others as their first
                    const int live = min(NTOK, p.b.M - n0);
                    for (int c0 = 2 * warp; c0 < live; c0 += 2 * PF_UW) {
                        const float4 *q = reinterpret_cast<const float4 *>(p.part + (int64_t)c0 * 128) + lane;
                        float d[2][4];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float4 v = __ldcg(q + ((int64_t)ca * 2 + first) * (NTOK * 32) + h * 32);
                            d[h][0] = v.x; d[h][1] = v.y; d[h][2] = v.z; d[h][3] = v.w;
                        }
                        for (int c = ca + 1; c <= cb; c += 4) {
                            float4 v[4][2];
#pragma unroll
                            for (int k = 0; k < 4; ++k)
#pragma unroll
                                for (int h = 0; h < 2; ++h)
                                    v[k][h] = c + k <= cb ? __ldcg(q + (int64_t)(c + k) * 2 * (NTOK * 32) + h * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int k = 0; k < 4; ++k)
#pragma unroll
                                for (int h = 0; h < 2; ++h) { d[h][0] += v[k][h].x; d[h][1] += v[k][h].y; d[h][2] += v[k][h].z; d[h][3] += v[k][h].w; }
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const int r = 4 * lane + j;
                                if (c0 + h < live && s_row[r] >= 0)
                                    p.b.Y[(int64_t)(n0 + c0 + h) * p.b.Q + s_row[r]] = __fmaf_rn(s_ts[r], d[h][j], s_ms[r] * s_sx[c0 + h]) * s_sc[c0 + h];
                            }
                    }
                }
            }
            // (the tables are written again only once every warp has read them)
            asm volatile("bar.sync 1, %0;\n" ::"n"(PF_UNPACK) : "memory");
        }
    } else if (warp == PF_UW) {
        // ------------------------------------------------------------------------------------------ activation copies
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;\n" ::: "memory");       // the narrow kernel's tiles
            bool alive = true;
            int i = 0, s = 0;
            uint32_t par = 1;                                          // (the first use of a stage needs no wait)
            for (int64_t at = lo; at < hi && alive;) {
                const MidSeg sg = mid_seg(p, at, hi);
                at += sg.ub - sg.ua;
                if (mid_empty(p, sg.tile)) continue;
                const uint8_t *xsrc = reinterpret_cast<const uint8_t *>(p.b.X16) + (int64_t)(sg.tile / p.row_tiles) * nkb * (C::B_BYTES / 2);
                for (int u = sg.ua; u < sg.ub; ++u, ++i) {
                    if (i >= C::NBS) alive = pf_wait(pf_smem(&b_empty[s]), par, abort_flag, 44);
                    if (!alive) break;
                    const uint32_t bar = pf_smem(&b_full[s]), bytes = (uint32_t)(min(2, nkb - 2 * u) * (C::B_BYTES / 2));
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                                 :: "r"(pf_smem(smem + s * C::B_BYTES)), "l"(xsrc + (int64_t)u * C::B_BYTES), "r"(bytes), "r"(bar)
                                 : "memory");
                    if (++s == C::NBS) { s = 0; par ^= 1u; }
                }
            }
        }
    } else {
        // ------------------------------------------------------------------------------------------ MMA issue
        // The whole warp walks the units (addresses stay in uniform registers), one lane issues; the eight instructions of
        // a pair are unrolled.  With one lane in a rolled loop a pair took 0.77 us, as long as its unpacking.
        constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NTOK >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t dbase = pf_desc(pf_smem(smem), NTOK * 16, 128);
        const uint32_t dlo0 = (uint32_t)dbase, dhi = (uint32_t)(dbase >> 32);
        bool alive = true;
        int begun = 0, slot = 0, s = 0;                  // begun: chunks so far
        uint32_t apar = 0, bpar = 0;
        auto mma = [&](uint32_t acc, uint32_t a_t, uint32_t dlo, bool accumulate) {
            uint64_t db;
            asm volatile("mov.b64 %0, {%1, %2};\n" : "=l"(db) : "r"(dlo), "r"(dhi));
            asm volatile(
                "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                :: "r"(acc), "r"(a_t), "l"(db), "r"(IDESC), "r"((uint32_t)accumulate) : "memory");
        };
        for (int64_t at = lo; at < hi && alive;) {
            const MidSeg sg = mid_seg(p, at, hi);
            at += sg.ub - sg.ua;
            if (mid_empty(p, sg.tile)) continue;
            for (int u = sg.ua, in_chunk = 0; u < sg.ub && alive; ++u) {
                if (in_chunk == 0 && ++begun > 2) alive = pf_wait(pf_smem(&acc_empty[(begun - 1) & 1]), ((begun - 3) >> 1) & 1, abort_flag, 48);
                if (alive) alive = pf_wait(pf_smem(&b_full[s]), bpar, abort_flag, 46);
                if (alive) alive = pf_wait(pf_smem(&a_full[slot]), apar, abort_flag, 45);
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t a_t = tmem + (uint32_t)(C::ACC + slot * 64), dlo = dlo0 + (uint32_t)(s * (C::B_BYTES >> 4));
                const int buf = (begun - 1) & 1;
                const uint32_t acc = tmem + (uint32_t)(buf * C::ACC1);
                const bool first = in_chunk == 0;
                if (++in_chunk == MD_CHUNK || u + 1 == sg.ub) in_chunk = 0;
                if (pf_elect()) {
                    mma(acc, a_t, dlo, !first);
#pragma unroll
                    for (int kk = 1; kk < 4; ++kk) mma(acc, a_t + 8 * kk, dlo + kk * 2 * NTOK, true);
                    if (2 * u + 1 < nkb) {
#pragma unroll
                        for (int kk = 4; kk < 8; ++kk) mma(acc, a_t + 8 * kk, dlo + kk * 2 * NTOK, true);
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(pf_smem(&b_empty[s])) : "memory");
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(pf_smem(&a_empty[slot])) : "memory");
                    if (in_chunk == 0)
                        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(pf_smem(&acc_full[buf])) : "memory");
                }
                __syncwarp();
                if (++slot == C::NU) { slot = 0; apar ^= 1u; }
                if (++s == C::NBS) { s = 0; bpar ^= 1u; }
            }
        }
    }
    __syncwarp();
    if (*abort_flag && warp == PF_UW) {                      // copies may still be in flight: let them land before the CTA goes
        uint64_t t0, t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
        for (int i = 0; i < (1 << 16); ++i) {
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            if (t - t0 > 200000ull) break;
            __nanosleep(1000);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"((uint32_t)PF_TMEM_COLS) : "memory");
}

// One block per token: narrow to saturated fp16 tiles (tokens beyond M become zeros), the sum of the narrowed values and,
// for x_mode 1, the power of two that brings the token's largest magnitude into fp16's range (x * 2^-k, exact).
__device__ __forceinline__ void mid_load8(const void *__restrict__ X, int x_dtype, int64_t i, float (&v)[8]) {
    if (x_dtype == QVB8_F32) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(X) + i));
        const float4 b = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(X) + i) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(X) + i));
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (x_dtype == QVB8_BF16) {
                v[2 * k] = __uint_as_float(w[k] << 16);
                v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
            } else {
                v[2 * k] = __half2float(__ushort_as_half((unsigned short)(w[k] & 0xffffu)));
                v[2 * k + 1] = __half2float(__ushort_as_half((unsigned short)(w[k] >> 16)));
            }
        }
    }
}
template <int NTOK>
__global__ void __launch_bounds__(MD_NARROW) mid_narrow_kernel(const void *__restrict__ X, int x_dtype, int x_mode, int M, int P,
                                                         __half *__restrict__ X16, float *__restrict__ sumx, int *__restrict__ kexp,
                                                         int *__restrict__ ticket, int ntickets) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    __shared__ float part[MD_NARROW / 32];
    __shared__ uint32_t amax_s[MD_NARROW / 32];
    const int n = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int t = n * MD_NARROW + tid; t < ntickets; t += gridDim.x * MD_NARROW) ticket[t] = 0;
    const int nkb = P / PF_BK, ngrp = P / 8;
    float scale = 1.f;
    if (x_mode == 1 && x_dtype != QVB8_F16 && n < M) {
        uint32_t mx = 0u;
#pragma unroll 4
        for (int g = tid; g < ngrp; g += MD_NARROW) {
            float v[8];
            mid_load8(X, x_dtype, (int64_t)n * P + g * 8, v);
#pragma unroll
            for (int k = 0; k < 8; ++k) mx = max(mx, __float_as_uint(v[k]) & 0x7fffffffu);
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) amax_s[warp] = mx;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < MD_NARROW / 32; ++k) mx = max(mx, amax_s[k]);
        const int e = (int)(mx >> 23) - 127, k = e > 15 ? min(e - 15, 112) : 0;
        scale = __uint_as_float((uint32_t)(127 - k) << 23);
        if (tid == 0) kexp[n] = k;
    } else if (tid == 0) kexp[n] = 0;
    float s = 0.f;
#pragma unroll 4
    for (int g = tid; g < ngrp; g += MD_NARROW) {
        uint32_t h[4] = {0u, 0u, 0u, 0u};
        if (n < M) {
            float v[8];
            mid_load8(X, x_dtype, (int64_t)n * P + g * 8, v);
            __half f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                f[k] = sat_half(v[k] * scale);
                s += __half2float(f[k]);
            }
            const __half2 a = __halves2half2(f[0], f[2]), b = __halves2half2(f[1], f[3]), c = __halves2half2(f[4], f[6]), d = __halves2half2(f[5], f[7]);
            h[0] = *reinterpret_cast<const uint32_t *>(&a); h[1] = *reinterpret_cast<const uint32_t *>(&b);   // see pair_order
            h[2] = *reinterpret_cast<const uint32_t *>(&c); h[3] = *reinterpret_cast<const uint32_t *>(&d);
        }
        *reinterpret_cast<uint4 *>(X16 + mid_x16<NTOK>(n, g * 8, nkb)) = make_uint4(h[0], h[1], h[2], h[3]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) part[warp] = s;
    __syncthreads();
    if (tid == 0) {
        for (int k = 1; k < MD_NARROW / 32; ++k) s += part[k];
        sumx[n] = s;
    }
}

// Escapes (Y += sum of x16 * (exact - band) in stored order) and rows wider than 11 bits (their tensor-core sums, over
// zeros, are replaced by an fp32 product).  Block = 16 rows x one token tile; lanes are tokens while a warp walks its
// rows' entries, then rows while it writes Y.  The blocks are small enough to sit beside a main CTA, so the entries (a
// lane each: eight of every row) are in registers by the time the products are done.
constexpr int MD_FIX_ROWS = 16;
template <int NTOK>
__global__ void __launch_bounds__(128) mid_fix_kernel(const MidParams p, const int *__restrict__ esc_ptr, const int *__restrict__ esc_col,
                                                      const float *__restrict__ esc_delta) {
    constexpr int TL = (NTOK + 31) / 32;                               // tokens per lane
    __shared__ float E[NTOK][MD_FIX_ROWS + 1];
    const int q0 = blockIdx.x * MD_FIX_ROWS, n0 = blockIdx.y * NTOK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nkb = p.b.P / PF_BK;
    const uint32_t wide = __ballot_sync(0xffffffffu, lane < MD_FIX_ROWS && q0 + lane < p.b.Q && __ldg(p.b.nbits + min(q0 + lane, p.b.Q - 1)) > PF_EXACT_BITS);
    const int ep = esc_ptr != nullptr ? __ldg(esc_ptr + min(q0 + min(lane, MD_FIX_ROWS), p.b.Q)) : 0;
    const bool escapes = __shfl_sync(0xffffffffu, ep, 0) != __shfl_sync(0xffffffffu, ep, MD_FIX_ROWS);
    // entry lane % 8 of row warp * 4 + lane / 8
    const int my0 = __shfl_sync(0xffffffffu, ep, warp * 4 + (lane >> 3)), my1 = __shfl_sync(0xffffffffu, ep, warp * 4 + (lane >> 3) + 1);
    int col = 0;
    float delta = 0.f;
    if (my0 + (lane & 7) < my1) {
        col = __ldg(esc_col + my0 + (lane & 7));
        delta = __ldg(esc_delta + my0 + (lane & 7));
    }
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    if (!wide && !escapes) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int r = warp * 4 + j, q = q0 + r;
        const int e0 = __shfl_sync(0xffffffffu, ep, r), e1 = __shfl_sync(0xffffffffu, ep, r + 1);
        float a[TL];
#pragma unroll
        for (int t = 0; t < TL; ++t) a[t] = 0.f;
        if ((wide >> r) & 1u) {
            const int nb = __ldg(p.b.nbits + q);
            const int64_t bit0 = __ldg(p.b.bit_off + q);
            const float ts = __ldg(p.b.tau_s + q), ms = __ldg(p.b.min_s + q);
            for (int n = 0; n < NTOK && n0 + n < p.b.M; ++n) {         // lanes take columns here: rare, and long rows
                float s = 0.f;
                for (int c = lane; c < p.b.P; c += 32)
                    s = __fmaf_rn(__half2float(p.b.X16[mid_x16<NTOK>(n0 + n, c, nkb)]), band(field_bytes(p.b.ids, bit0 + (int64_t)c * nb, nb), ts, ms), s);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
#pragma unroll
                for (int t = 0; t < TL; ++t)
                    if (n == t * 32 + lane) a[t] = s;
            }
        }
        // four entries at a time: their loads overlap (an entry beyond the row's last reads the last's column, times zero)
        auto batch = [&](const int (&c)[4], const float (&d)[4], int n) {
            __half x[4][TL];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int t = 0; t < TL; ++t) x[k][t] = p.b.X16[mid_x16<NTOK>(n0 + min(t * 32 + lane, NTOK - 1), c[k], nkb)];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < n) {
#pragma unroll
                    for (int t = 0; t < TL; ++t) a[t] = __fmaf_rn(__half2float(x[k][t]), d[k], a[t]);
                }
        };
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (e0 + 4 * h >= e1) break;
            int c[4];
            float d[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c[k] = __shfl_sync(0xffffffffu, col, j * 8 + h * 4 + k);
                d[k] = __shfl_sync(0xffffffffu, delta, j * 8 + h * 4 + k);
            }
            batch(c, d, e1 - e0 - 4 * h);
        }
        for (int e = e0 + 8; e < e1; e += 4) {
            int c[4];
            float d[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c[k] = __ldg(esc_col + min(e + k, e1 - 1));
                d[k] = __ldg(esc_delta + min(e + k, e1 - 1));
            }
            batch(c, d, e1 - e);
        }
#pragma unroll
        for (int t = 0; t < TL; ++t)
            if (t * 32 + lane < NTOK) E[t * 32 + lane][r] = a[t];
    }
    __syncthreads();
    const int r = lane & (MD_FIX_ROWS - 1);
    if (q0 + r >= p.b.Q) return;
    for (int n = warp * 2 + (lane >> 4); n < NTOK && n0 + n < p.b.M; n += 8) {
        const float v = E[n][r] * __uint_as_float((uint32_t)(127 + __ldcg(p.kexp + n0 + n)) << 23);
        float *y = p.b.Y + (int64_t)(n0 + n) * p.b.Q + q0 + r;
        *y = ((wide >> r) & 1u) ? v : *y + v;
    }
}

// ---- host side of the middle-M path
static int mid_tokens(int64_t M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : M <= 96 ? 96 : 128; }
struct MidScratch { int64_t x16, sumx, kexp, ticket, part, total, tiles; int ntok; };
static MidScratch mid_scratch(int64_t M, int64_t Q, int64_t P) {
    MidScratch s{};
    s.ntok = mid_tokens(M);
    const int64_t tok_tiles = (M + s.ntok - 1) / s.ntok, Mpad = tok_tiles * s.ntok;
    const int64_t rows = ((Q + 15) / 16 + NCLASS - 1) * 16;
    s.tiles = tok_tiles * ((rows + 127) / 128);
    s.x16 = 0;
    s.sumx = s.x16 + up256(Mpad * P * 2);
    s.kexp = s.sumx + up256(Mpad * 4);
    s.ticket = s.kexp + up256(Mpad * 4);
    s.part = s.ticket + up256(s.tiles * 4);
    s.total = s.part + (int64_t)MD_CTAS * 2 * s.ntok * 128 * 4;
    return s;
}
int64_t mid_scratch_bytes(int64_t M, int64_t Q, int64_t P) { return mid_scratch(M, Q, P).total; }

// What the kernels read in place: a plan (for the row order), 16-byte aligned activations, byte offsets within 32 bits.
bool mid_takes(const qvb8_pack *w, const void *plan, const void *X, int64_t M) {
    return plan && aligned(plan, 256) && aligned(X, 16) && w->P % PF_BK == 0 && w->P > 0 && w->ids_bytes < (1ll << 32) && M >= 1 && M <= 65535;
}

// Runs of a product of `tiles` tiles of U units: at most one per SM, at least four units long.  Either every tile is cut
// into the same number S of runs (a CTA then has one segment), or 148 equal runs cut the tiles anywhere (equal shares, but
// a CTA finishes two or three segments, 7 units' time each).  In units (0.47 us): 4096 x 4096, 16 tokens, S = 4: 26.6 us,
// cut anywhere: 29.8; 24576 x 4096 has 193 tiles and no choice.
static int mid_runs(int64_t tiles, int64_t U) {
    const int64_t any = (tiles * U + MD_CTAS - 1) / MD_CTAS + 14;
    int64_t S = MD_CTAS / tiles;
    if (S > U / 4) S = U / 4 > 0 ? U / 4 : 1;
    if (S >= 1 && (U + S - 1) / S + (S > 1 ? 6 : 2) <= any) return (int)(tiles * S);
    const int64_t runs = tiles * U / 4;
    return (int)(runs < 1 ? 1 : runs < MD_CTAS ? runs : MD_CTAS);
}

template <int NTOK>
static int mid_run_kernels(const qvb8_pack *w, const PlanLayout &L, const uint8_t *pb, const MidParams &prm, const void *X, int x_dtype,
                           int x_mode, int Mpad, cudaStream_t st) {
    using C = MidCfg<NTOK>;
    static thread_local int granted_dev = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != granted_dev) {
        if (cudaFuncSetAttribute(mid_kernel<NTOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess)
            return cuda_status("qvb8 middle M: shared memory opt-in");
        granted_dev = dev;
    }
    mid_narrow_kernel<NTOK><<<(unsigned)Mpad, MD_NARROW, 0, st>>>(X, x_dtype, x_mode, prm.b.M, prm.b.P, const_cast<__half *>(prm.b.X16),
                                                            const_cast<float *>(prm.b.sumx), const_cast<int *>(prm.kexp), prm.ticket,
                                                            prm.row_tiles * prm.tok_tiles);
    if (int rc = cuda_status("qvb8 middle M: narrow")) return rc;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.stream = st;
    cfg.gridDim = dim3((unsigned)mid_runs((int64_t)prm.row_tiles * prm.tok_tiles, prm.units_tile));
    cfg.blockDim = dim3(PF_THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    if (cudaLaunchKernelEx(&cfg, mid_kernel<NTOK>, prm) != cudaSuccess) return cuda_status("qvb8 middle M");
    cfg.gridDim = dim3((unsigned)((prm.b.Q + MD_FIX_ROWS - 1) / MD_FIX_ROWS), (unsigned)prm.tok_tiles);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = 0;
    const int *ep = w->n_esc > 0 ? reinterpret_cast<const int *>(pb + L.esc_ptr) : nullptr;
    const int *ec = reinterpret_cast<const int *>(pb + L.esc_col);
    const float *ed = reinterpret_cast<const float *>(pb + L.esc_delta);
    if (cudaLaunchKernelEx(&cfg, mid_fix_kernel<NTOK>, prm, ep, ec, ed) != cudaSuccess) return cuda_status("qvb8 middle M: fix");
    return cuda_status("qvb8 middle M");
}

// scratch: mid_scratch_bytes(M, Q, P) bytes, 256-byte aligned, any contents.
int launch_mid(const qvb8_pack *w, const void *plan, const void *X, int x_dtype, int x_mode, int64_t M, float *Y, void *scratch,
               cudaStream_t st) {
    const MidScratch s = mid_scratch(M, w->Q, w->P);
    uint8_t *sc = reinterpret_cast<uint8_t *>(scratch);
    const PlanLayout L = plan_layout(w->Q, w->n_esc);
    const uint8_t *pb = reinterpret_cast<const uint8_t *>(plan);
    const int tok_tiles = (int)((M + s.ntok - 1) / s.ntok);
    MidParams prm{};
    prm.b = PrefillParams{w->ids, w->min_s, w->tau_s, w->nbits, w->bit_off, reinterpret_cast<const TileDesc *>(pb + L.tiles), L.max_tiles,
                          reinterpret_cast<const __half *>(sc + s.x16), reinterpret_cast<const float *>(sc + s.sumx), Y, (int)w->Q, (int)w->P,
                          (int)M, tok_tiles * s.ntok, 0};
    prm.kexp = reinterpret_cast<const int *>(sc + s.kexp);
    prm.ticket = reinterpret_cast<int *>(sc + s.ticket);
    prm.part = reinterpret_cast<float *>(sc + s.part);
    prm.row_tiles = (L.max_tiles * 16 + 127) / 128;
    prm.tok_tiles = tok_tiles;
    prm.units_tile = (int)((w->P / PF_BK + 1) / 2);
    prm.units = (int64_t)prm.row_tiles * tok_tiles * prm.units_tile;
    switch (s.ntok) {
        case 16: return mid_run_kernels<16>(w, L, pb, prm, X, x_dtype, x_mode, prm.b.Mpad, st);
        case 32: return mid_run_kernels<32>(w, L, pb, prm, X, x_dtype, x_mode, prm.b.Mpad, st);
        case 64: return mid_run_kernels<64>(w, L, pb, prm, X, x_dtype, x_mode, prm.b.Mpad, st);
        case 96: return mid_run_kernels<96>(w, L, pb, prm, X, x_dtype, x_mode, prm.b.Mpad, st);
        default: return mid_run_kernels<128>(w, L, pb, prm, X, x_dtype, x_mode, prm.b.Mpad, st);
    }
}

}  // namespace qv

QV_API void qvb8_prefill_set_tuning(int debug) { qv::g_prefill_debug = debug; }

QV_API int64_t qvb8_prefill_scratch_bytes(int64_t M, int64_t Q, int64_t P) {
    if (M <= 0 || P <= 0 || Q < 0) return 0;
    const int64_t Mpad = (M + qv::PF_TOK - 1) / qv::PF_TOK * qv::PF_TOK;
    return 2 * qv::up256(Mpad * P * 2) + qv::up256(qv::PF_KS * Mpad * 4) + qv::up256((Q + 1) * 4);
}

QV_API int qvb8_prefill(const qvb8_pack *w, const void *plan, const void *X, int x_dtype, int64_t M, float *Y, void *scratch,
                        int64_t scratch_bytes, void *stream) {
    using namespace qv;
    if (int rc = check_pack(w, "qvb8_prefill")) return rc;
    if (int rc = check_device("qvb8_prefill")) return rc;
    if (!X || !Y || M <= 0 || M > 0x7fffff00) return fail(QVB8_ERR_ARG, "qvb8_prefill: bad X / Y / M");
    if (x_dtype != QVB8_F16 && x_dtype != QVB8_BF16 && x_dtype != QVB8_F32) return fail(QVB8_ERR_ARG, "qvb8_prefill: bad X dtype");
    if (w->Q == 0) return QVB8_OK;
    if (w->P % PF_BK != 0) return fail(QVB8_ERR_ARG, "qvb8_prefill: P must be a multiple of %d", PF_BK);
    if (!aligned(X, 16)) return fail(QVB8_ERR_ARG, "qvb8_prefill: X must be 16-byte aligned");
    if (w->ids_bytes >= (1ll << 32)) return fail(QVB8_ERR_ARG, "qvb8_prefill: packs of 4 GiB and more are not supported");
    if (!plan || !aligned(plan, 256)) return fail(QVB8_ERR_ARG, "qvb8_prefill: the pack's plan is needed (qvb8_plan_build), 256-byte aligned");
    const int64_t need = qvb8_prefill_scratch_bytes(M, w->Q, w->P);
    if (!scratch || scratch_bytes < need || !aligned(scratch, 256))
        return fail(QVB8_ERR_SCRATCH, "qvb8_prefill: scratch of %lld bytes (256-byte aligned) needed, %lld given", (long long)need, (long long)scratch_bytes);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int64_t Mpad = (M + PF_TOK - 1) / PF_TOK * PF_TOK;
    uint8_t *sc = reinterpret_cast<uint8_t *>(scratch);
    __half *X16 = reinterpret_cast<__half *>(sc);
    __half *X16T = reinterpret_cast<__half *>(sc + up256(Mpad * w->P * 2));      // written only for packs with escapes
    float *sumx = reinterpret_cast<float *>(sc + 2 * up256(Mpad * w->P * 2));
    int *wide = reinterpret_cast<int *>(reinterpret_cast<uint8_t *>(sumx) + up256(PF_KS * Mpad * 4));      // [0] count, then rows
    prefill_narrow_kernel<<<dim3((unsigned)(Mpad / 32), PF_KS), 256, 0, st>>>(X, x_dtype, (int)M, (int)Mpad, (int)w->P, X16, w->n_esc > 0 ? X16T : nullptr, sumx);
    if (int rc = cuda_status("qvb8_prefill narrow")) return rc;

    const PlanLayout L = plan_layout(w->Q, w->n_esc);
    const uint8_t *pb = reinterpret_cast<const uint8_t *>(plan);
    PrefillParams prm{w->ids, w->min_s, w->tau_s, w->nbits, w->bit_off, reinterpret_cast<const TileDesc *>(pb + L.tiles), L.max_tiles,
                      X16, sumx, Y, (int)w->Q, (int)w->P, (int)M, (int)Mpad, g_prefill_debug};
    if (int rc = launch_prefill(prm, st)) return rc;

    if (cudaMemsetAsync(wide, 0, sizeof(int), st) != cudaSuccess) return cuda_status("qvb8_prefill memset");
    prefill_wide_list_kernel<<<(unsigned)((w->Q + 255) / 256), 256, 0, st>>>(w->nbits, (int)w->Q, wide + 1, wide);
    prefill_wide_rows_kernel<<<dim3(64, (unsigned)((M + 7) / 8)), 256, 0, st>>>(prm, wide + 1, wide);
    if (int rc = cuda_status("qvb8_prefill wide rows")) return rc;
    if (w->n_esc > 0) {
        prefill_escapes_kernel<<<dim3((unsigned)((w->Q + 31) / 32), (unsigned)(Mpad / 256)), 256, 0, st>>>(
            reinterpret_cast<const int *>(pb + L.esc_ptr), reinterpret_cast<const int *>(pb + L.esc_col),
            reinterpret_cast<const float *>(pb + L.esc_delta), X16T, Y, (int)w->Q, (int)M, (int)Mpad);
        if (int rc = cuda_status("qvb8_prefill escapes")) return rc;
    }
    return QVB8_OK;
}

QV_API int64_t qvb8_mid_m_scratch_bytes(int64_t M, int64_t Q, int64_t P) {
    if (M <= 0 || M > 65535 || P <= 0 || Q < 0 || P % qv::PF_BK != 0) return 0;
    return qv::mid_scratch_bytes(M, Q, P);
}

QV_API int qvb8_mid_m(const qvb8_pack *w, const void *plan, const void *X, int x_dtype, int x_mode, int64_t M, float *Y, void *scratch,
                      int64_t scratch_bytes, void *stream) {
    using namespace qv;
    if (int rc = check_pack(w, "qvb8_mid_m")) return rc;
    if (int rc = check_device("qvb8_mid_m")) return rc;
    if (!X || !Y || M <= 0) return fail(QVB8_ERR_ARG, "qvb8_mid_m: bad X / Y / M");
    if (x_dtype != QVB8_F16 && x_dtype != QVB8_BF16 && x_dtype != QVB8_F32) return fail(QVB8_ERR_ARG, "qvb8_mid_m: bad X dtype");
    if (x_mode != 0 && x_mode != 1) return fail(QVB8_ERR_ARG, "qvb8_mid_m: bad x_mode");
    if (w->Q == 0) return QVB8_OK;
    if (!mid_takes(w, plan, X, M))
        return fail(QVB8_ERR_ARG, "qvb8_mid_m: needs the pack's plan (256-byte aligned), 16-byte aligned X, P %% %d == 0, ids below 4 GiB and M <= 65535", PF_BK);
    const int64_t need = mid_scratch_bytes(M, w->Q, w->P);
    if (!scratch || scratch_bytes < need || !aligned(scratch, 16))
        return fail(QVB8_ERR_SCRATCH, "qvb8_mid_m: scratch of %lld bytes (16-byte aligned) needed, %lld given", (long long)need, (long long)scratch_bytes);
    return launch_mid(w, plan, X, x_dtype, x_mode, M, Y, scratch, reinterpret_cast<cudaStream_t>(stream));
}
