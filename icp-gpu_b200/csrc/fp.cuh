// BLS12-381 base field Fp on sm_100a: 381-bit Montgomery arithmetic on twelve
// 32-bit limbs, R = 2^384, every stored value canonical (< p), so a value's
// limbs equal ic_bls12_381's in-memory Montgomery representation.
//
// The multiply is CIOS (Koc, Acar, Kaliski, "Analyzing and comparing Montgomery
// multiplication algorithms", 1996) over paired columns.  A limb product gives
// two words, and the two multiply-adds of one pair of limbs, written next to
// each other (mad.lo.cc then madc.hi.cc on the same operands), issue as one
// 64-bit multiply-add with carry in and out.  So the running value is kept as
// two vectors, E with a word for columns 0..11 and O for columns 1..12: a row
// a * b_i puts the products of a's even limbs on E's pairs and those of its odd
// limbs on O's pairs, two carry chains of six:
//   O  += a_1,3,..,11 * b_i      (the pending word of column 0 carries in)
//   E  += a_0,2,..,10 * b_i,     carry into O's top word
//   m  = E[0] * (-p^-1 mod 2^32)
//   O  += m * p_1,3,..,11;  E  += m * p_0,2,..,10,  carry into O's top word
// and dividing by 2^32 exchanges the vectors: O's columns become E's, E[2..11]
// become O's and E[1] waits as the pending word of column 0.  With a, b < p the
// running value stays below 2^416, so the thirteen columns hold it and no carry
// leaves O's top word.  Per multiply: 24 x 12 / 2 = 288 / 2 paired multiply-adds
// twice (a b and m p) plus 12 mul.lo.
//
// What it is bound by: a paired multiply-add holds the multiply pipe as long as
// mul.hi alone does (4 cycles a warp and scheduler), and mul.lo half of that, so
// rows of separate mul.lo and mul.hi chains cost 6 cycles a limb product where
// the pair costs 4.  The paired columns made every workload 1.24 to 1.52 times as
// fast; the 12 x 12-limb product alone, operands from shared memory, went from 41.4
// to 57.3 G products/s on 148 SMs (bls_limb_layout_rates).
//
// This replaces the reference's vendored sppark fp_t (gpu-crypto/cuda/vendor/
// sppark/mont_t.cuh:381-422, constants bls12-381.hpp:13-33) and is written from
// the algorithm, not from that file.
#pragma once
#include <cstdint>

namespace bls {

struct fp { uint32_t w[12]; };

// p, little-endian 32-bit limbs
#define BLS_P0 0xffffaaabu
#define BLS_P1 0xb9feffffu
#define BLS_P2 0xb153ffffu
#define BLS_P3 0x1eabfffeu
#define BLS_P4 0xf6b0f624u
#define BLS_P5 0x6730d2a0u
#define BLS_P6 0xf38512bfu
#define BLS_P7 0x64774b84u
#define BLS_P8 0x434bacd7u
#define BLS_P9 0x4b1ba7b6u
#define BLS_P10 0x397fe69au
#define BLS_P11 0x1a0111eau
#define BLS_NINV 0xfffcfffdu  // -p^-1 mod 2^32

__host__ __device__ __forceinline__ fp fp_zero() {
    fp r;
    for (int i = 0; i < 12; ++i) r.w[i] = 0;
    return r;
}
// R mod p (Montgomery one)
__host__ __device__ __forceinline__ fp fp_one() {
    fp r;
    r.w[0] = 0x0002fffdu; r.w[1] = 0x76090000u; r.w[2] = 0xc40c0002u; r.w[3] = 0xebf4000bu;
    r.w[4] = 0x53c758bau; r.w[5] = 0x5f489857u; r.w[6] = 0x70525745u; r.w[7] = 0x77ce5853u;
    r.w[8] = 0xa256ec6du; r.w[9] = 0x5c071a97u; r.w[10] = 0xfa80e493u; r.w[11] = 0x15f65ec3u;
    return r;
}
// R^2 mod p
__host__ __device__ __forceinline__ fp fp_rr() {
    fp r;
    r.w[0] = 0x1c341746u; r.w[1] = 0xf4df1f34u; r.w[2] = 0x09d104f1u; r.w[3] = 0x0a76e6a6u;
    r.w[4] = 0x4c95b6d5u; r.w[5] = 0x8de5476cu; r.w[6] = 0x939d83c0u; r.w[7] = 0x67eb88a9u;
    r.w[8] = 0xb519952du; r.w[9] = 0x9a793e85u; r.w[10] = 0x92cae3aau; r.w[11] = 0x11988fe5u;
    return r;
}

__device__ __forceinline__ bool fp_is_zero(const fp& a) {
    uint32_t o = a.w[0];
#pragma unroll
    for (int i = 1; i < 12; ++i) o |= a.w[i];
    return o == 0;
}
__device__ __forceinline__ bool fp_eq(const fp& a, const fp& b) {
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) o |= a.w[i] ^ b.w[i];
    return o == 0;
}

// ---------------------------------------------------------------------------
// carry chains
// ---------------------------------------------------------------------------
// Paired chains: t[0..2N-1] += sum over k < N of x[2k] * b * 2^(64 k), the limbs
// taken from x at stride 2.  mad_pairs: nothing carries out of t[2N-1] (the top
// pair is fresh, or the caller's bound says so); mad_pairs_c returns the carry.
template <int N>
__device__ __forceinline__ void mad_pairs(uint32_t* t, const uint32_t* x, uint32_t b) {
    if constexpr (N == 1)
        asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
            "madc.hi.u32 %1, %2, %3, %1;"
            : "+r"(t[0]), "+r"(t[1])
            : "r"(x[0]), "r"(b));
    if constexpr (N == 2)
        asm("mad.lo.cc.u32 %0, %4, %6, %0;\n\t"
            "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
            "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
            "madc.hi.u32 %3, %5, %6, %3;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3])
            : "r"(x[0]), "r"(x[2]), "r"(b));
    if constexpr (N == 3)
        asm("mad.lo.cc.u32 %0, %6, %9, %0;\n\t"
            "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
            "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
            "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
            "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
            "madc.hi.u32 %5, %8, %9, %5;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5])
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(b));
    if constexpr (N == 4)
        asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
            "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
            "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
            "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
            "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
            "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
            "madc.hi.u32 %7, %11, %12, %7;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7])
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(x[6]), "r"(b));
    if constexpr (N == 5)
        asm("mad.lo.cc.u32 %0, %10, %15, %0;\n\t"
            "madc.hi.cc.u32 %1, %10, %15, %1;\n\t"
            "madc.lo.cc.u32 %2, %11, %15, %2;\n\t"
            "madc.hi.cc.u32 %3, %11, %15, %3;\n\t"
            "madc.lo.cc.u32 %4, %12, %15, %4;\n\t"
            "madc.hi.cc.u32 %5, %12, %15, %5;\n\t"
            "madc.lo.cc.u32 %6, %13, %15, %6;\n\t"
            "madc.hi.cc.u32 %7, %13, %15, %7;\n\t"
            "madc.lo.cc.u32 %8, %14, %15, %8;\n\t"
            "madc.hi.u32 %9, %14, %15, %9;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
              "+r"(t[8]), "+r"(t[9])
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(x[6]), "r"(x[8]), "r"(b));
    if constexpr (N == 6)
        asm("mad.lo.cc.u32 %0, %12, %18, %0;\n\t"
            "madc.hi.cc.u32 %1, %12, %18, %1;\n\t"
            "madc.lo.cc.u32 %2, %13, %18, %2;\n\t"
            "madc.hi.cc.u32 %3, %13, %18, %3;\n\t"
            "madc.lo.cc.u32 %4, %14, %18, %4;\n\t"
            "madc.hi.cc.u32 %5, %14, %18, %5;\n\t"
            "madc.lo.cc.u32 %6, %15, %18, %6;\n\t"
            "madc.hi.cc.u32 %7, %15, %18, %7;\n\t"
            "madc.lo.cc.u32 %8, %16, %18, %8;\n\t"
            "madc.hi.cc.u32 %9, %16, %18, %9;\n\t"
            "madc.lo.cc.u32 %10, %17, %18, %10;\n\t"
            "madc.hi.u32 %11, %17, %18, %11;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
              "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11])
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(x[6]), "r"(x[8]), "r"(x[10]), "r"(b));
}
template <int N>
__device__ __forceinline__ uint32_t mad_pairs_c(uint32_t* t, const uint32_t* x, uint32_t b) {
    uint32_t c = 0;
    if constexpr (N == 1)
        asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
            "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
            "addc.u32 %2, 0, 0;"
            : "+r"(t[0]), "+r"(t[1]), "=r"(c)
            : "r"(x[0]), "r"(b));
    if constexpr (N == 2)
        asm("mad.lo.cc.u32 %0, %5, %7, %0;\n\t"
            "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
            "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
            "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
            "addc.u32 %4, 0, 0;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "=r"(c)
            : "r"(x[0]), "r"(x[2]), "r"(b));
    if constexpr (N == 3)
        asm("mad.lo.cc.u32 %0, %7, %10, %0;\n\t"
            "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
            "addc.u32 %6, 0, 0;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "=r"(c)
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(b));
    if constexpr (N == 4)
        asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
            "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
            "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
            "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
            "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
            "addc.u32 %8, 0, 0;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
              "=r"(c)
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(x[6]), "r"(b));
    if constexpr (N == 5)
        asm("mad.lo.cc.u32 %0, %11, %16, %0;\n\t"
            "madc.hi.cc.u32 %1, %11, %16, %1;\n\t"
            "madc.lo.cc.u32 %2, %12, %16, %2;\n\t"
            "madc.hi.cc.u32 %3, %12, %16, %3;\n\t"
            "madc.lo.cc.u32 %4, %13, %16, %4;\n\t"
            "madc.hi.cc.u32 %5, %13, %16, %5;\n\t"
            "madc.lo.cc.u32 %6, %14, %16, %6;\n\t"
            "madc.hi.cc.u32 %7, %14, %16, %7;\n\t"
            "madc.lo.cc.u32 %8, %15, %16, %8;\n\t"
            "madc.hi.cc.u32 %9, %15, %16, %9;\n\t"
            "addc.u32 %10, 0, 0;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
              "+r"(t[8]), "+r"(t[9]), "=r"(c)
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(x[6]), "r"(x[8]), "r"(b));
    if constexpr (N == 6)
        asm("mad.lo.cc.u32 %0, %13, %19, %0;\n\t"
            "madc.hi.cc.u32 %1, %13, %19, %1;\n\t"
            "madc.lo.cc.u32 %2, %14, %19, %2;\n\t"
            "madc.hi.cc.u32 %3, %14, %19, %3;\n\t"
            "madc.lo.cc.u32 %4, %15, %19, %4;\n\t"
            "madc.hi.cc.u32 %5, %15, %19, %5;\n\t"
            "madc.lo.cc.u32 %6, %16, %19, %6;\n\t"
            "madc.hi.cc.u32 %7, %16, %19, %7;\n\t"
            "madc.lo.cc.u32 %8, %17, %19, %8;\n\t"
            "madc.hi.cc.u32 %9, %17, %19, %9;\n\t"
            "madc.lo.cc.u32 %10, %18, %19, %10;\n\t"
            "madc.hi.cc.u32 %11, %18, %19, %11;\n\t"
            "addc.u32 %12, 0, 0;"
            : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
              "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "=r"(c)
            : "r"(x[0]), "r"(x[2]), "r"(x[4]), "r"(x[6]), "r"(x[8]), "r"(x[10]), "r"(b));
    return c;
}

// t[0..1] = a * b
__device__ __forceinline__ void mul_pair(uint32_t* t, uint32_t a, uint32_t b) {
    const uint64_t p = (uint64_t)a * b;
    t[0] = (uint32_t)p;
    t[1] = (uint32_t)(p >> 32);
}
#define BLS_T13(t) "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), \
    "+r"(t[6]), "+r"(t[7]), "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "+r"(t[12])
#define BLS_T1_12(t) "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), \
    "+r"(t[7]), "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "+r"(t[12])
#define BLS_A12(a) "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), \
    "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11])

// A: t[0..11] += lo(a * b), carry into t[12]
__device__ __forceinline__ void chain_lo(uint32_t* t, const uint32_t* a, uint32_t b) {
    asm("mad.lo.cc.u32 %0, %13, %25, %0;\n\t"
        "madc.lo.cc.u32 %1, %14, %25, %1;\n\t"
        "madc.lo.cc.u32 %2, %15, %25, %2;\n\t"
        "madc.lo.cc.u32 %3, %16, %25, %3;\n\t"
        "madc.lo.cc.u32 %4, %17, %25, %4;\n\t"
        "madc.lo.cc.u32 %5, %18, %25, %5;\n\t"
        "madc.lo.cc.u32 %6, %19, %25, %6;\n\t"
        "madc.lo.cc.u32 %7, %20, %25, %7;\n\t"
        "madc.lo.cc.u32 %8, %21, %25, %8;\n\t"
        "madc.lo.cc.u32 %9, %22, %25, %9;\n\t"
        "madc.lo.cc.u32 %10, %23, %25, %10;\n\t"
        "madc.lo.cc.u32 %11, %24, %25, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : BLS_T13(t) : BLS_A12(a), "r"(b));
}
// B: t[1..12] += hi(a * b); no carry leaves t[12]
__device__ __forceinline__ void chain_hi(uint32_t* t, const uint32_t* a, uint32_t b) {
    asm("mad.hi.cc.u32 %0, %12, %24, %0;\n\t"
        "madc.hi.cc.u32 %1, %13, %24, %1;\n\t"
        "madc.hi.cc.u32 %2, %14, %24, %2;\n\t"
        "madc.hi.cc.u32 %3, %15, %24, %3;\n\t"
        "madc.hi.cc.u32 %4, %16, %24, %4;\n\t"
        "madc.hi.cc.u32 %5, %17, %24, %5;\n\t"
        "madc.hi.cc.u32 %6, %18, %24, %6;\n\t"
        "madc.hi.cc.u32 %7, %19, %24, %7;\n\t"
        "madc.hi.cc.u32 %8, %20, %24, %8;\n\t"
        "madc.hi.cc.u32 %9, %21, %24, %9;\n\t"
        "madc.hi.cc.u32 %10, %22, %24, %10;\n\t"
        "madc.hi.u32 %11, %23, %24, %11;"
        : BLS_T1_12(t) : BLS_A12(a), "r"(b));
}
// C: t[0..11] += lo(m * p), carry into t[12]
__device__ __forceinline__ void chain_lo_p(uint32_t* t, uint32_t m) {
    asm("mad.lo.cc.u32 %0, %13, 0xffffaaab, %0;\n\t"
        "madc.lo.cc.u32 %1, %13, 0xb9feffff, %1;\n\t"
        "madc.lo.cc.u32 %2, %13, 0xb153ffff, %2;\n\t"
        "madc.lo.cc.u32 %3, %13, 0x1eabfffe, %3;\n\t"
        "madc.lo.cc.u32 %4, %13, 0xf6b0f624, %4;\n\t"
        "madc.lo.cc.u32 %5, %13, 0x6730d2a0, %5;\n\t"
        "madc.lo.cc.u32 %6, %13, 0xf38512bf, %6;\n\t"
        "madc.lo.cc.u32 %7, %13, 0x64774b84, %7;\n\t"
        "madc.lo.cc.u32 %8, %13, 0x434bacd7, %8;\n\t"
        "madc.lo.cc.u32 %9, %13, 0x4b1ba7b6, %9;\n\t"
        "madc.lo.cc.u32 %10, %13, 0x397fe69a, %10;\n\t"
        "madc.lo.cc.u32 %11, %13, 0x1a0111ea, %11;\n\t"
        "addc.u32 %12, %12, 0;"
        : BLS_T13(t) : "r"(m));
}
// D: t[1..12] += hi(m * p)
__device__ __forceinline__ void chain_hi_p(uint32_t* t, uint32_t m) {
    asm("mad.hi.cc.u32 %0, %12, 0xffffaaab, %0;\n\t"
        "madc.hi.cc.u32 %1, %12, 0xb9feffff, %1;\n\t"
        "madc.hi.cc.u32 %2, %12, 0xb153ffff, %2;\n\t"
        "madc.hi.cc.u32 %3, %12, 0x1eabfffe, %3;\n\t"
        "madc.hi.cc.u32 %4, %12, 0xf6b0f624, %4;\n\t"
        "madc.hi.cc.u32 %5, %12, 0x6730d2a0, %5;\n\t"
        "madc.hi.cc.u32 %6, %12, 0xf38512bf, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, 0x64774b84, %7;\n\t"
        "madc.hi.cc.u32 %8, %12, 0x434bacd7, %8;\n\t"
        "madc.hi.cc.u32 %9, %12, 0x4b1ba7b6, %9;\n\t"
        "madc.hi.cc.u32 %10, %12, 0x397fe69a, %10;\n\t"
        "madc.hi.u32 %11, %12, 0x1a0111ea, %11;"
        : BLS_T1_12(t) : "r"(m));
}
// d = a - p over 12 limbs; returns the borrow (1 when a < p)
__device__ __forceinline__ uint32_t sub_p(uint32_t* d, const uint32_t* a) {
    uint32_t br;
    asm("sub.cc.u32 %0, %13, 0xffffaaab;\n\t"
        "subc.cc.u32 %1, %14, 0xb9feffff;\n\t"
        "subc.cc.u32 %2, %15, 0xb153ffff;\n\t"
        "subc.cc.u32 %3, %16, 0x1eabfffe;\n\t"
        "subc.cc.u32 %4, %17, 0xf6b0f624;\n\t"
        "subc.cc.u32 %5, %18, 0x6730d2a0;\n\t"
        "subc.cc.u32 %6, %19, 0xf38512bf;\n\t"
        "subc.cc.u32 %7, %20, 0x64774b84;\n\t"
        "subc.cc.u32 %8, %21, 0x434bacd7;\n\t"
        "subc.cc.u32 %9, %22, 0x4b1ba7b6;\n\t"
        "subc.cc.u32 %10, %23, 0x397fe69a;\n\t"
        "subc.cc.u32 %11, %24, 0x1a0111ea;\n\t"
        "subc.u32 %12, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]),
          "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(br)
        : BLS_A12(a));
    return br;  // 0xffffffff on borrow, else 0
}

// keep t if t < p, else t - p
__device__ __forceinline__ void reduce_once(uint32_t* t) {
    uint32_t d[12];
    uint32_t br = sub_p(d, t);
#pragma unroll
    for (int i = 0; i < 12; ++i) t[i] = br ? t[i] : d[i];
}

// ---------------------------------------------------------------------------
// field operations
// ---------------------------------------------------------------------------
#define BLS_T12(t) "+r"((t)[0]), "+r"((t)[1]), "+r"((t)[2]), "+r"((t)[3]), "+r"((t)[4]), "+r"((t)[5]), \
    "+r"((t)[6]), "+r"((t)[7]), "+r"((t)[8]), "+r"((t)[9]), "+r"((t)[10]), "+r"((t)[11])

// one row a * b on the vectors E and O (file comment); prev: the pending word
// of column 0
__device__ __forceinline__ void mont_row_ab(uint32_t* E, uint32_t* O, uint32_t prev, const uint32_t* a, uint32_t b) {
    asm("add.cc.u32 %0, %0, %24;\n\t"
        "madc.lo.cc.u32 %12, %26, %37, %12;\n\t"
        "madc.hi.cc.u32 %13, %26, %37, %13;\n\t"
        "madc.lo.cc.u32 %14, %28, %37, %14;\n\t"
        "madc.hi.cc.u32 %15, %28, %37, %15;\n\t"
        "madc.lo.cc.u32 %16, %30, %37, %16;\n\t"
        "madc.hi.cc.u32 %17, %30, %37, %17;\n\t"
        "madc.lo.cc.u32 %18, %32, %37, %18;\n\t"
        "madc.hi.cc.u32 %19, %32, %37, %19;\n\t"
        "madc.lo.cc.u32 %20, %34, %37, %20;\n\t"
        "madc.hi.cc.u32 %21, %34, %37, %21;\n\t"
        "madc.lo.cc.u32 %22, %36, %37, %22;\n\t"
        "madc.hi.u32 %23, %36, %37, %23;\n\t"
        "mad.lo.cc.u32 %0, %25, %37, %0;\n\t"
        "madc.hi.cc.u32 %1, %25, %37, %1;\n\t"
        "madc.lo.cc.u32 %2, %27, %37, %2;\n\t"
        "madc.hi.cc.u32 %3, %27, %37, %3;\n\t"
        "madc.lo.cc.u32 %4, %29, %37, %4;\n\t"
        "madc.hi.cc.u32 %5, %29, %37, %5;\n\t"
        "madc.lo.cc.u32 %6, %31, %37, %6;\n\t"
        "madc.hi.cc.u32 %7, %31, %37, %7;\n\t"
        "madc.lo.cc.u32 %8, %33, %37, %8;\n\t"
        "madc.hi.cc.u32 %9, %33, %37, %9;\n\t"
        "madc.lo.cc.u32 %10, %35, %37, %10;\n\t"
        "madc.hi.cc.u32 %11, %35, %37, %11;\n\t"
        "addc.u32 %23, %23, 0;"
        : BLS_T12(E), BLS_T12(O)
        : "r"(prev), BLS_A12(a), "r"(b));
}
// one reduction row: m = (E[0] + prev) * (-p^-1), value += m p; column 0 becomes zero
__device__ __forceinline__ void mont_row_mp(uint32_t* E, uint32_t* O, uint32_t prev) {
    uint32_t m;
    asm("add.cc.u32 %0, %0, %25;\n\t"
        "mul.lo.u32 %24, %0, 0xfffcfffd;\n\t"
        "madc.lo.cc.u32 %12, %24, 0xb9feffff, %12;\n\t"
        "madc.hi.cc.u32 %13, %24, 0xb9feffff, %13;\n\t"
        "madc.lo.cc.u32 %14, %24, 0x1eabfffe, %14;\n\t"
        "madc.hi.cc.u32 %15, %24, 0x1eabfffe, %15;\n\t"
        "madc.lo.cc.u32 %16, %24, 0x6730d2a0, %16;\n\t"
        "madc.hi.cc.u32 %17, %24, 0x6730d2a0, %17;\n\t"
        "madc.lo.cc.u32 %18, %24, 0x64774b84, %18;\n\t"
        "madc.hi.cc.u32 %19, %24, 0x64774b84, %19;\n\t"
        "madc.lo.cc.u32 %20, %24, 0x4b1ba7b6, %20;\n\t"
        "madc.hi.cc.u32 %21, %24, 0x4b1ba7b6, %21;\n\t"
        "madc.lo.cc.u32 %22, %24, 0x1a0111ea, %22;\n\t"
        "madc.hi.u32 %23, %24, 0x1a0111ea, %23;\n\t"
        "mad.lo.cc.u32 %0, %24, 0xffffaaab, %0;\n\t"
        "madc.hi.cc.u32 %1, %24, 0xffffaaab, %1;\n\t"
        "madc.lo.cc.u32 %2, %24, 0xb153ffff, %2;\n\t"
        "madc.hi.cc.u32 %3, %24, 0xb153ffff, %3;\n\t"
        "madc.lo.cc.u32 %4, %24, 0xf6b0f624, %4;\n\t"
        "madc.hi.cc.u32 %5, %24, 0xf6b0f624, %5;\n\t"
        "madc.lo.cc.u32 %6, %24, 0xf38512bf, %6;\n\t"
        "madc.hi.cc.u32 %7, %24, 0xf38512bf, %7;\n\t"
        "madc.lo.cc.u32 %8, %24, 0x434bacd7, %8;\n\t"
        "madc.hi.cc.u32 %9, %24, 0x434bacd7, %9;\n\t"
        "madc.lo.cc.u32 %10, %24, 0x397fe69a, %10;\n\t"
        "madc.hi.cc.u32 %11, %24, 0x397fe69a, %11;\n\t"
        "addc.u32 %23, %23, 0;"
        : BLS_T12(E), BLS_T12(O), "=&r"(m)
        : "r"(prev));
    (void)m;
}
// divide by 2^32: exchange the vectors; returns the new pending word
__device__ __forceinline__ uint32_t mont_shift(uint32_t* E, uint32_t* O) {
    const uint32_t prev = E[1];
#pragma unroll
    for (int j = 0; j < 12; ++j) {
        const uint32_t e = j < 10 ? E[j + 2] : 0u;
        E[j] = O[j];
        O[j] = e;
    }
    return prev;
}
// r = E + O 2^32 + prev after the last shift (O[10] = O[11] = 0; the value fits twelve limbs)
__device__ __forceinline__ void mont_merge(uint32_t* r, const uint32_t* E, const uint32_t* O, uint32_t prev) {
    asm("add.cc.u32 %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, %33;\n\t"
        "addc.cc.u32 %10, %22, %34;\n\t"
        "addc.u32 %11, %23, 0;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11])
        : BLS_A12(E), "r"(prev), "r"(O[0]), "r"(O[1]), "r"(O[2]), "r"(O[3]), "r"(O[4]), "r"(O[5]), "r"(O[6]),
          "r"(O[7]), "r"(O[8]), "r"(O[9]));
}

// Montgomery product without the final subtraction.  For a, b < 8p (the
// redundant range of the lane-parallel kernel) the result is below 7.5p and
// every intermediate stays below 2^416, so thirteen columns hold it.
__device__ __forceinline__ fp fp_mul_redundant(const fp& a, const fp& b) {
    uint32_t E[12], O[12], prev = 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) E[i] = O[i] = 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        mont_row_ab(E, O, prev, a.w, b.w[i]);
        mont_row_mp(E, O, 0);
        prev = mont_shift(E, O);
    }
    fp r;
    mont_merge(r.w, E, O, prev);
    return r;
}

__device__ __forceinline__ fp fp_mul(const fp& a, const fp& b) {
    fp r = fp_mul_redundant(a, b);
    reduce_once(r.w);
    return r;
}

// (a b + c d) R^-1 mod p, canonical, by one reduction; a, b, c, d <= p (a row's
// value stays below (a + c + p) 2^32, the result below 1.3p before the subtraction)
__device__ __forceinline__ fp fp_mul2(const fp& a, const fp& b, const fp& c, const fp& d) {
    uint32_t E[12], O[12], prev = 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) E[i] = O[i] = 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        mont_row_ab(E, O, prev, a.w, b.w[i]);
        mont_row_ab(E, O, 0, c.w, d.w[i]);
        mont_row_mp(E, O, 0);
        prev = mont_shift(E, O);
    }
    fp r;
    mont_merge(r.w, E, O, prev);
    reduce_once(r.w);
    return r;
}

// (t + m p) / 2^384 for the m that makes it whole: t[0..11] Montgomery-reduced
// on its own, at most p
__device__ __forceinline__ void mont_reduce12(uint32_t* r, const uint32_t* t) {
    uint32_t E[12], O[12], prev = 0;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        E[i] = t[i];
        O[i] = 0;
    }
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        mont_row_mp(E, O, prev);
        prev = mont_shift(E, O);
    }
    mont_merge(r, E, O, prev);
}

// one row of the square (fp_sqr): a_I times a_I at column 2I and times the
// doubled limbs above it, even columns into A, odd ones into B (B[k]: column k + 1)
template <int I>
__device__ __forceinline__ void sqr_row(uint32_t* A, uint32_t* B, const uint32_t* a, const uint32_t* d) {
    constexpr int NA = 1 + (11 - I) / 2, NB = (12 - I) / 2;   // pairs at even columns, at odd columns
    uint32_t x[12], y[12];
    x[0] = a[I];
#pragma unroll
    for (int k = 1; k < NA; ++k) x[2 * k] = d[I + 2 * k];
#pragma unroll
    for (int k = 0; k < NB; ++k) y[2 * k] = k == 0 ? a[I + 1] << 1 : d[I + 1 + 2 * k];
    if constexpr (I == 0) {
#pragma unroll
        for (int k = 0; k < NA; ++k) mul_pair(A + 2 * k, x[2 * k], a[0]);
#pragma unroll
        for (int k = 0; k < NB; ++k) mul_pair(B + 2 * k, y[2 * k], a[0]);
        A[12] = B[12] = 0;
    } else if constexpr (I & 1) {      // the top pair of A is fresh, B's chain carries out
        A[2 * I + 2 * NA - 1] = 0;
        mad_pairs<NA>(A + 2 * I, x, a[I]);
        if constexpr (NB > 0) B[2 * I + 2 * NB] = mad_pairs_c<NB>(B + 2 * I, y, a[I]);
    } else {
        B[2 * I + 2 * NB - 1] = 0;
        mad_pairs<NB>(B + 2 * I, y, a[I]);
        A[2 * I + 2 * NA] = mad_pairs_c<NA>(A + 2 * I, x, a[I]);
    }
}

// Montgomery square a^2 R^-1 mod p for a <= 3p, canonical (below p): row i takes
// a_i times a_i and times the limbs above it of 2a (whose lowest, a_{i+1}, enters
// without the bit that belongs to a_i), so the 66 cross products are formed once:
// 78 paired multiply-adds, in the two column vectors of the file comment.  Then the
// low twelve limbs are Montgomery-reduced on their own, (t_lo + m p) / R <= p,
// and the high twelve added: a^2 / R + p < 1.92p for a <= 3p (p / R < 0.1017), so one
// conditional subtraction ends it.  222 paired multiply-adds where the general product takes
// 288; the same value as fp_mul(a, a).
__device__ __forceinline__ fp fp_sqr(const fp& a) {
    uint32_t A[24], B[24], d[12];
    d[0] = 0;   // not used: 2a's limbs 2..11 are
#pragma unroll
    for (int j = 1; j < 12; ++j) d[j] = __funnelshift_l(a.w[j - 1], a.w[j], 1);
    sqr_row<0>(A, B, a.w, d);
    sqr_row<1>(A, B, a.w, d);
    sqr_row<2>(A, B, a.w, d);
    sqr_row<3>(A, B, a.w, d);
    sqr_row<4>(A, B, a.w, d);
    sqr_row<5>(A, B, a.w, d);
    sqr_row<6>(A, B, a.w, d);
    sqr_row<7>(A, B, a.w, d);
    sqr_row<8>(A, B, a.w, d);
    sqr_row<9>(A, B, a.w, d);
    sqr_row<10>(A, B, a.w, d);
    sqr_row<11>(A, B, a.w, d);
    B[22] = 0;
    uint32_t t[24];
    t[0] = A[0];
    asm("add.cc.u32 %0, %23, %46;\n\t"
        "addc.cc.u32 %1, %24, %47;\n\t"
        "addc.cc.u32 %2, %25, %48;\n\t"
        "addc.cc.u32 %3, %26, %49;\n\t"
        "addc.cc.u32 %4, %27, %50;\n\t"
        "addc.cc.u32 %5, %28, %51;\n\t"
        "addc.cc.u32 %6, %29, %52;\n\t"
        "addc.cc.u32 %7, %30, %53;\n\t"
        "addc.cc.u32 %8, %31, %54;\n\t"
        "addc.cc.u32 %9, %32, %55;\n\t"
        "addc.cc.u32 %10, %33, %56;\n\t"
        "addc.cc.u32 %11, %34, %57;\n\t"
        "addc.cc.u32 %12, %35, %58;\n\t"
        "addc.cc.u32 %13, %36, %59;\n\t"
        "addc.cc.u32 %14, %37, %60;\n\t"
        "addc.cc.u32 %15, %38, %61;\n\t"
        "addc.cc.u32 %16, %39, %62;\n\t"
        "addc.cc.u32 %17, %40, %63;\n\t"
        "addc.cc.u32 %18, %41, %64;\n\t"
        "addc.cc.u32 %19, %42, %65;\n\t"
        "addc.cc.u32 %20, %43, %66;\n\t"
        "addc.cc.u32 %21, %44, %67;\n\t"
        "addc.u32 %22, %45, %68;"
        : "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]), "=r"(t[8]),
          "=r"(t[9]), "=r"(t[10]), "=r"(t[11]), "=r"(t[12]), "=r"(t[13]), "=r"(t[14]), "=r"(t[15]),
          "=r"(t[16]), "=r"(t[17]), "=r"(t[18]), "=r"(t[19]), "=r"(t[20]), "=r"(t[21]), "=r"(t[22]), "=r"(t[23])
        : "r"(A[1]), "r"(A[2]), "r"(A[3]), "r"(A[4]), "r"(A[5]), "r"(A[6]), "r"(A[7]), "r"(A[8]), "r"(A[9]),
          "r"(A[10]), "r"(A[11]), "r"(A[12]), "r"(A[13]), "r"(A[14]), "r"(A[15]), "r"(A[16]), "r"(A[17]),
          "r"(A[18]), "r"(A[19]), "r"(A[20]), "r"(A[21]), "r"(A[22]), "r"(A[23]), "r"(B[0]), "r"(B[1]),
          "r"(B[2]), "r"(B[3]), "r"(B[4]), "r"(B[5]), "r"(B[6]), "r"(B[7]), "r"(B[8]), "r"(B[9]), "r"(B[10]),
          "r"(B[11]), "r"(B[12]), "r"(B[13]), "r"(B[14]), "r"(B[15]), "r"(B[16]), "r"(B[17]), "r"(B[18]),
          "r"(B[19]), "r"(B[20]), "r"(B[21]), "r"(B[22]));
    uint32_t u[12];
    mont_reduce12(u, t);
    uint32_t s[12];
    asm("add.cc.u32 %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, %33;\n\t"
        "addc.cc.u32 %10, %22, %34;\n\t"
        "addc.u32 %11, %23, %35;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
          "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11])
        : BLS_A12(u), "r"(t[12]), "r"(t[13]), "r"(t[14]), "r"(t[15]), "r"(t[16]), "r"(t[17]),
          "r"(t[18]), "r"(t[19]), "r"(t[20]), "r"(t[21]), "r"(t[22]), "r"(t[23]));
    reduce_once(s);
    fp r;
#pragma unroll
    for (int i = 0; i < 12; ++i) r.w[i] = s[i];
    return r;
}

__device__ __forceinline__ fp fp_add(const fp& a, const fp& b) {
    uint32_t s[12];
    asm("add.cc.u32 %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, %33;\n\t"
        "addc.cc.u32 %10, %22, %34;\n\t"
        "addc.u32 %11, %23, %35;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
          "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11])
        : BLS_A12(a.w), BLS_A12(b.w));
    reduce_once(s);  // a + b < 2p < 2^382: no carry out of limb 11
    fp r;
#pragma unroll
    for (int i = 0; i < 12; ++i) r.w[i] = s[i];
    return r;
}

// a + b without the range reduction: below 2^384 while the sum is below 9p
__device__ __forceinline__ fp fp_add_nr(const fp& a, const fp& b) {
    fp r;
    asm("add.cc.u32 %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, %33;\n\t"
        "addc.cc.u32 %10, %22, %34;\n\t"
        "addc.u32 %11, %23, %35;"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]),
          "=r"(r.w[7]), "=r"(r.w[8]), "=r"(r.w[9]), "=r"(r.w[10]), "=r"(r.w[11])
        : BLS_A12(a.w), BLS_A12(b.w));
    return r;
}

__device__ __forceinline__ fp fp_sub(const fp& a, const fp& b) {
    uint32_t s[12], mask;
    asm("sub.cc.u32 %0, %13, %25;\n\t"
        "subc.cc.u32 %1, %14, %26;\n\t"
        "subc.cc.u32 %2, %15, %27;\n\t"
        "subc.cc.u32 %3, %16, %28;\n\t"
        "subc.cc.u32 %4, %17, %29;\n\t"
        "subc.cc.u32 %5, %18, %30;\n\t"
        "subc.cc.u32 %6, %19, %31;\n\t"
        "subc.cc.u32 %7, %20, %32;\n\t"
        "subc.cc.u32 %8, %21, %33;\n\t"
        "subc.cc.u32 %9, %22, %34;\n\t"
        "subc.cc.u32 %10, %23, %35;\n\t"
        "subc.cc.u32 %11, %24, %36;\n\t"
        "subc.u32 %12, 0, 0;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]),
          "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(mask)
        : BLS_A12(a.w), BLS_A12(b.w));
    fp r;
    asm("add.cc.u32 %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, %33;\n\t"
        "addc.cc.u32 %10, %22, %34;\n\t"
        "addc.u32 %11, %23, %35;"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]),
          "=r"(r.w[6]), "=r"(r.w[7]), "=r"(r.w[8]), "=r"(r.w[9]), "=r"(r.w[10]), "=r"(r.w[11])
        : BLS_A12(s), "r"(BLS_P0 & mask), "r"(BLS_P1 & mask), "r"(BLS_P2 & mask), "r"(BLS_P3 & mask),
          "r"(BLS_P4 & mask), "r"(BLS_P5 & mask), "r"(BLS_P6 & mask), "r"(BLS_P7 & mask),
          "r"(BLS_P8 & mask), "r"(BLS_P9 & mask), "r"(BLS_P10 & mask), "r"(BLS_P11 & mask));
    return r;
}

__device__ __forceinline__ fp fp_neg(const fp& a) { return fp_sub(fp_zero(), a); }

// ---------------------------------------------------------------------------
// conversions
// ---------------------------------------------------------------------------
__device__ __forceinline__ fp fp_load_u64(const uint64_t* v) {
    fp r;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        r.w[2 * i] = (uint32_t)v[i];
        r.w[2 * i + 1] = (uint32_t)(v[i] >> 32);
    }
    return r;
}
__device__ __forceinline__ void fp_store_u64(uint64_t* v, const fp& a) {
#pragma unroll
    for (int i = 0; i < 6; ++i) v[i] = ((uint64_t)a.w[2 * i + 1] << 32) | a.w[2 * i];
}
// Montgomery -> canonical integer limbs (multiply by 1)
__device__ __forceinline__ fp fp_from_mont(const fp& a) {
    fp one_raw = fp_zero();
    one_raw.w[0] = 1;
    return fp_mul(a, one_raw);
}
// canonical integer limbs (< p) -> Montgomery (multiply by R^2)
__device__ __forceinline__ fp fp_to_mont(const fp& a) { return fp_mul(a, fp_rr()); }

// true when the canonical limbs are >= p
__device__ __forceinline__ bool fp_raw_geq_p(const fp& a) {
    uint32_t d[12];
    return sub_p(d, a.w) == 0;
}

// An out-of-line Montgomery multiply and square, and a power over them, for
// code that runs few warps per scheduler (a thread per point, per key or per
// message): there nothing hides a miss in the instruction cache, and a loop
// that inlines a multiply of several hundred instructions at every use misses
// on each pass.
static __device__ __noinline__ fp fp_mul_ool(const fp& a, const fp& b) { return fp_mul(a, b); }
static __device__ __noinline__ fp fp_sqr_ool(const fp& a) { return fp_sqr(a); }

// a^e (e: nbits bits, little-endian u64 words, the same for every thread) by
// a left-to-right sliding window of four bits over the odd powers a, a^3, ...,
// a^15: one squaring per bit and one product per window, about nbits / 5 of
// them, where the bit-by-bit power takes one product per set bit.  a below
// 2p; the result is canonical (a^0 = 1, 0^e = 0 for e > 0).  The squaring is inlined
// at its one place, a loop of its own: a call passes its operands through local
// memory.
__device__ __forceinline__ fp fp_pow_ool(const fp& a, const uint64_t* e, int nbits) {
    fp odd[8];
    odd[0] = a;
    const fp a2 = fp_sqr_ool(a);
    for (int k = 1; k < 8; ++k) odd[k] = fp_mul_ool(odd[k - 1], a2);
    auto bit = [&](int i) { return (int)((e[i >> 6] >> (i & 63)) & 1u); };
    fp r = fp_one();
    bool started = false;
#pragma unroll 1
    for (int i = nbits - 1; i >= 0;) {
        int j = i;                                   // squarings down to bit j, and the window's value
        while (j >= 0 && !bit(j)) --j;
        int v = 0;
        if (j >= 0) {                                // the window [w, j] ends on a set bit
            int w = j >= 3 ? j - 3 : 0;
            while (!bit(w)) ++w;
            for (int k = j; k >= w; --k) v = (v << 1) | bit(k);
            j = w;
        } else {
            j = 0;
        }
        if (started) {
#pragma unroll 1
            for (int k = i; k >= j; --k) r = fp_sqr(r);
            if (v) r = fp_mul(r, odd[v >> 1]);
        } else if (v) {
            r = odd[v >> 1];
            started = true;
        }
        i = j - 1;
    }
    return r;
}

}  // namespace bls
