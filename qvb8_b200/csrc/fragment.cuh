// From packed ids in shared memory to the operands of mma.sync: what the streaming kernel and the expert layer share.
#pragma once
#include "common.cuh"

namespace qv {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Pairing of a width: ids f and f + D share a register.  E > 0: the low id sits at mantissa bit E and the high id at
// bit 0 of the upper half-word; E < 0: the low id at bit 0, the high id at mantissa bit -E.  (nb * D == 16 - E.)
template <int NB> struct Pairing;
template <> struct Pairing<8> { static constexpr int D = 2, E = 0; };
template <> struct Pairing<7> { static constexpr int D = 2, E = 2; };
template <> struct Pairing<6> { static constexpr int D = 2, E = 4; };
template <> struct Pairing<5> { static constexpr int D = 4, E = -4; };
template <> struct Pairing<4> { static constexpr int D = 4, E = 0; };
template <> struct Pairing<3> { static constexpr int D = 4, E = 4; };

// fp16 bit patterns of 2^-e and -1024 * 2^-e (written as integers: the conversion intrinsics are opaque to constant
// folding and would run on the conversion pipe for every pair).
__host__ __device__ constexpr uint32_t h_pow2(int e) { return (uint32_t)(15 - e) << 10; }
__host__ __device__ constexpr uint32_t h_neg1024_pow2(int e) { return 0x8000u | ((uint32_t)(25 - e) << 10); }

// The four constants of a width, held in registers for a whole tile.  They are read from a small table in shared
// memory with volatile loads: values the compiler can see (literals, or moves of literals) it re-creates next to
// every use -- one extra instruction per pair, measured -- because the fp16 multiply-add takes only one of its two
// constants as an immediate.
struct PairConst { uint32_t mask, magic, scale, bias; };
__host__ __device__ constexpr uint32_t pair_const_word(int nb, int k) {
    const int D = nb >= 6 ? 2 : 4;
    const int E = 16 - nb * D;                                   // Pairing<nb>::E
    const int EL = E > 0 ? E : 0, EH = E < 0 ? -E : 0;
    const uint32_t FM = (1u << nb) - 1u;
    return k == 0 ? ((FM << EL) | (FM << (16 + EH)))
         : k == 1 ? 0x64006400u
         : k == 2 ? (h_pow2(EL) | (h_pow2(EH) << 16))
                  : (h_neg1024_pow2(EL) | (h_neg1024_pow2(EH) << 16));
}
constexpr int PAIR_TABLE_WORDS = 6 * 4;                          // widths 3..8
__device__ __forceinline__ PairConst pair_const(const uint32_t *table, int nb) {
    const uint32_t a = smem_u32(table + (nb - 3) * 4);
    PairConst c;
    asm volatile("ld.volatile.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(c.mask), "=r"(c.magic), "=r"(c.scale), "=r"(c.bias) : "r"(a));
    return c;
}
// The constants of operands id - centre (see zero_id).
__device__ __forceinline__ PairConst centred(PairConst c, float centre) {
    const __half2 b = __hsub2(*reinterpret_cast<const __half2 *>(&c.bias), __float2half2_rn(centre));
    c.bias = *reinterpret_cast<const uint32_t *>(&b);
    return c;
}

// Register holding fp16(id[fa]) in the low half and fp16(id[fa + D]) in the high half, from the nb words W of a
// thread's 32-id block.  All shifts fold to constants after unrolling.
template <int NB, bool CENTRED = false>
__device__ __forceinline__ uint32_t pair_reg(const uint32_t (&W)[NB], int fa, const PairConst &pc) {
    constexpr int D = Pairing<NB>::D, E = Pairing<NB>::E;
    constexpr int EL = E > 0 ? E : 0;            // mantissa shift of the low id
    constexpr int EH = E < 0 ? -E : 0;           // mantissa shift of the high id
    static_assert(NB * D == 16 + EH - EL, "pairing does not line the two ids up");
    static_assert(EL + NB <= 10 && EH + NB <= 10, "id does not fit the fp16 mantissa");
    const int s = NB * fa - EL;                  // bit of the block that must land on bit 0
    uint32_t r;
    if (s < 0) {
        r = W[0] << (-s);
    } else {
        const int wi = s >> 5, sh = s & 31;
        const int top = sh + 16 + EH + NB;       // one past the highest bit needed, relative to W[wi]
        if (sh == 0) r = W[wi];
        else if (top <= 32) r = W[wi] >> sh;
        else asm("shf.r.wrap.b32 %0, %1, %2, %3;\n" : "=r"(r) : "r"(W[wi]), "r"(W[wi + 1 < NB ? wi + 1 : wi]), "r"(sh));
    }
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;\n" : "=r"(r) : "r"(r), "r"(pc.mask), "r"(pc.magic));   // (r & mask) | magic:
    if constexpr (EL == 0 && EH == 0) {                                                         // 1024 + id * 2^shift, twice
        if constexpr (CENTRED) asm("add.f16x2 %0, %1, %2;\n" : "=r"(r) : "r"(r), "r"(pc.bias));
        else asm("sub.f16x2 %0, %1, %2;\n" : "=r"(r) : "r"(r), "r"(pc.magic));
    } else {
        asm("fma.rn.f16x2 %0, %1, %2, %3;\n" : "=r"(r) : "r"(r), "r"(pc.scale), "r"(pc.bias));
    }
    return r;
}

// The nb words of a thread's block, with the widest conflict-free shared-memory loads for that width.
template <int NB>
__device__ __forceinline__ void load_block(uint32_t addr, uint32_t (&W)[NB]) {
    if constexpr (NB == 8) {
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(W[0]), "=r"(W[1]), "=r"(W[2]), "=r"(W[3]) : "r"(addr));
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+16];\n" : "=r"(W[4]), "=r"(W[5]), "=r"(W[6]), "=r"(W[7]) : "r"(addr));
    } else if constexpr (NB == 4) {
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(W[0]), "=r"(W[1]), "=r"(W[2]), "=r"(W[3]) : "r"(addr));
    } else if constexpr (NB == 6) {
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];\n" : "=r"(W[0]), "=r"(W[1]) : "r"(addr));
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+8];\n" : "=r"(W[2]), "=r"(W[3]) : "r"(addr));
        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2+16];\n" : "=r"(W[4]), "=r"(W[5]) : "r"(addr));
    } else {
        static_assert(NB == 8 || NB == 4 || NB == 6, "odd widths are specialised below");
    }
}
// odd widths: nb scalar loads (an odd stride in words spreads the 32 lanes over all banks)
template <>
__device__ __forceinline__ void load_block<7>(uint32_t addr, uint32_t (&W)[7]) {
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(W[0]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+4];\n" : "=r"(W[1]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+8];\n" : "=r"(W[2]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+12];\n" : "=r"(W[3]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+16];\n" : "=r"(W[4]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+20];\n" : "=r"(W[5]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+24];\n" : "=r"(W[6]) : "r"(addr));
}
template <>
__device__ __forceinline__ void load_block<5>(uint32_t addr, uint32_t (&W)[5]) {
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(W[0]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+4];\n" : "=r"(W[1]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+8];\n" : "=r"(W[2]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+12];\n" : "=r"(W[3]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+16];\n" : "=r"(W[4]) : "r"(addr));
}
template <>
__device__ __forceinline__ void load_block<3>(uint32_t addr, uint32_t (&W)[3]) {
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(W[0]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+4];\n" : "=r"(W[1]) : "r"(addr));
    asm volatile("ld.shared.u32 %0, [%1+8];\n" : "=r"(W[2]) : "r"(addr));
}

// Bytes between rows of a stage.  The chunks of a row lie back to back (one contiguous copy per row and stage); the
// stride adds padding so that the 32 lanes of a warp, which read rows g and columns 32 t of ONE chunk, fall on
// distinct banks.
__host__ __device__ constexpr bool stride_ok(int nb, int rs) {
    return nb == 8 ? (rs / 16) % 8 == 1                  // 16-byte loads, quarter warps (rows 2i, 2i+1)
         : nb == 4 ? (rs / 16) % 8 == 4
         : nb == 6 ? (rs / 8) % 16 == 12                 // 8-byte loads, half warps (rows 4i .. 4i+3)
                   : (rs / 4) % 32 == (4 * nb) % 32;     // 4-byte loads, whole warp
}
__host__ __device__ constexpr int stage_row_stride(int nb, int cps) {
    int rs = 16 * nb * cps;
    while (!stride_ok(nb, rs)) rs += 16;
    return rs;
}

// Place of the e-th of eight consecutive activations inside their 16-byte slot, for widths whose ids pair at distance 2:
// x0 x2 x1 x3 x4 x6 x5 x7.
__device__ __forceinline__ int pos_a(int e) { return (e & 4) | ((e & 1) << 1) | ((e >> 1) & 1); }

}  // namespace qv
