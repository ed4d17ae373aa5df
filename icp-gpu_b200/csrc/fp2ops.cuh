// Device arithmetic of the Fp2-lane verify kernel (verify_fp2.cu): products
// into double-width accumulators, one Montgomery reduction per output, and
// the QP reduction that keeps every slot below 2^381 + p.  The generator's
// emulator (gen_fp2ops.py) models each routine here bit for bit.
#pragma once
#include "fp.cuh"
#include "fp2ops.inc"
#include "fp_inv.cuh"

namespace bls {
namespace f2 {

#define BLS_SUB13_12(m, s)                                                                                 \
    asm("sub.cc.u32 %0, %0, %13;\n\t"                                                                     \
        "subc.cc.u32 %1, %1, %14;\n\t"                                                                    \
        "subc.cc.u32 %2, %2, %15;\n\t"                                                                    \
        "subc.cc.u32 %3, %3, %16;\n\t"                                                                    \
        "subc.cc.u32 %4, %4, %17;\n\t"                                                                    \
        "subc.cc.u32 %5, %5, %18;\n\t"                                                                    \
        "subc.cc.u32 %6, %6, %19;\n\t"                                                                    \
        "subc.cc.u32 %7, %7, %20;\n\t"                                                                    \
        "subc.cc.u32 %8, %8, %21;\n\t"                                                                    \
        "subc.cc.u32 %9, %9, %22;\n\t"                                                                    \
        "subc.cc.u32 %10, %10, %23;\n\t"                                                                  \
        "subc.cc.u32 %11, %11, %24;\n\t"                                                                  \
        "subc.u32 %12, %12, 0;"                                                                          \
        : "+r"(m[0]), "+r"(m[1]), "+r"(m[2]), "+r"(m[3]), "+r"(m[4]), "+r"(m[5]), "+r"(m[6]), "+r"(m[7]),  \
          "+r"(m[8]), "+r"(m[9]), "+r"(m[10]), "+r"(m[11]), "+r"(m[12])                                  \
        : "r"((s)[0]), "r"((s)[1]), "r"((s)[2]), "r"((s)[3]), "r"((s)[4]), "r"((s)[5]), "r"((s)[6]),       \
          "r"((s)[7]), "r"((s)[8]), "r"((s)[9]), "r"((s)[10]), "r"((s)[11]))
#define BLS_ADD_MID(p, m)                                                                                    \
    asm("add.cc.u32 %0, %0, %18;\n\t"                                                                     \
        "addc.cc.u32 %1, %1, %19;\n\t"                                                                    \
        "addc.cc.u32 %2, %2, %20;\n\t"                                                                    \
        "addc.cc.u32 %3, %3, %21;\n\t"                                                                    \
        "addc.cc.u32 %4, %4, %22;\n\t"                                                                    \
        "addc.cc.u32 %5, %5, %23;\n\t"                                                                    \
        "addc.cc.u32 %6, %6, %24;\n\t"                                                                    \
        "addc.cc.u32 %7, %7, %25;\n\t"                                                                    \
        "addc.cc.u32 %8, %8, %26;\n\t"                                                                    \
        "addc.cc.u32 %9, %9, %27;\n\t"                                                                    \
        "addc.cc.u32 %10, %10, %28;\n\t"                                                                  \
        "addc.cc.u32 %11, %11, %29;\n\t"                                                                  \
        "addc.cc.u32 %12, %12, %30;\n\t"                                                                  \
        "addc.cc.u32 %13, %13, 0;\n\t"                                                                    \
        "addc.cc.u32 %14, %14, 0;\n\t"                                                                    \
        "addc.cc.u32 %15, %15, 0;\n\t"                                                                    \
        "addc.cc.u32 %16, %16, 0;\n\t"                                                                    \
        "addc.u32 %17, %17, 0;"                                                                          \
        : "+r"((p)[6]), "+r"((p)[7]), "+r"((p)[8]), "+r"((p)[9]), "+r"((p)[10]), "+r"((p)[11]),            \
          "+r"((p)[12]), "+r"((p)[13]), "+r"((p)[14]), "+r"((p)[15]), "+r"((p)[16]), "+r"((p)[17]),        \
          "+r"((p)[18]), "+r"((p)[19]), "+r"((p)[20]), "+r"((p)[21]), "+r"((p)[22]), "+r"((p)[23])         \
        : "r"(m[0]), "r"(m[1]), "r"(m[2]), "r"(m[3]), "r"(m[4]), "r"(m[5]), "r"(m[6]), "r"(m[7]),         \
          "r"(m[8]), "r"(m[9]), "r"(m[10]), "r"(m[11]), "r"(m[12]))

// r[0..11] = a[0..5] * b[0..5]: row i puts the products of a's even limbs and
// of its odd limbs on the pairs of two vectors, A for even columns and B for odd
// ones (B[k]: column k + 1), as in fp.cuh; one add chain joins them
__device__ __forceinline__ void mul6(uint32_t* r, const uint32_t* a, const uint32_t* b) {
    uint32_t A[12], B[12];
#pragma unroll
    for (int k = 0; k < 6; k += 2) {
        mul_pair(A + k, a[k], b[0]);
        mul_pair(B + k, a[k + 1], b[0]);
    }
#pragma unroll
    for (int i = 1; i < 6; ++i) {
        uint32_t* X = (i & 1) ? B + (i - 1) : A + i;   // even limbs: columns i, i + 2, i + 4, carry to i + 6
        uint32_t* Y = (i & 1) ? A + (i + 1) : B + i;   // odd limbs: columns i + 1, .., i + 6, the top pair fresh
        if (i == 1) Y[4] = 0;
        Y[5] = 0;
        mad_pairs<3>(Y, a + 1, b[i]);
        X[6] = mad_pairs_c<3>(X, a, b[i]);
    }
    r[0] = A[0];
    asm("add.cc.u32 %0, %11, %22;\n\t"
        "addc.cc.u32 %1, %12, %23;\n\t"
        "addc.cc.u32 %2, %13, %24;\n\t"
        "addc.cc.u32 %3, %14, %25;\n\t"
        "addc.cc.u32 %4, %15, %26;\n\t"
        "addc.cc.u32 %5, %16, %27;\n\t"
        "addc.cc.u32 %6, %17, %28;\n\t"
        "addc.cc.u32 %7, %18, %29;\n\t"
        "addc.cc.u32 %8, %19, %30;\n\t"
        "addc.cc.u32 %9, %20, %31;\n\t"
        "addc.u32 %10, %21, %32;"
        : "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11])
        : "r"(A[1]), "r"(A[2]), "r"(A[3]), "r"(A[4]), "r"(A[5]), "r"(A[6]), "r"(A[7]), "r"(A[8]), "r"(A[9]),
          "r"(A[10]), "r"(A[11]), "r"(B[0]), "r"(B[1]), "r"(B[2]), "r"(B[3]), "r"(B[4]), "r"(B[5]), "r"(B[6]),
          "r"(B[7]), "r"(B[8]), "r"(B[9]), "r"(B[10]));
}

// p[0..23] = a * b, schoolbook: mul6's rows over all twelve limbs (144 pairs).
// The measured ceiling of the verify kernels' multiply form runs it
// (k_imad_chain); the kernels' own products are prod24k's.
__device__ __forceinline__ void prod24(uint32_t* p, const uint32_t* a, const uint32_t* b) {
    uint32_t A[24], B[24];
#pragma unroll
    for (int k = 0; k < 12; k += 2) {
        mul_pair(A + k, a[k], b[0]);
        mul_pair(B + k, a[k + 1], b[0]);
    }
#pragma unroll
    for (int i = 1; i < 12; ++i) {
        uint32_t* X = (i & 1) ? B + (i - 1) : A + i;
        uint32_t* Y = (i & 1) ? A + (i + 1) : B + i;
        if (i == 1) Y[10] = 0;
        Y[11] = 0;
        mad_pairs<6>(Y, a + 1, b[i]);
        X[12] = mad_pairs_c<6>(X, a, b[i]);
    }
    uint32_t c;
    p[0] = A[0];
    asm("add.cc.u32 %0, %13, %25;\n\t"
        "addc.cc.u32 %1, %14, %26;\n\t"
        "addc.cc.u32 %2, %15, %27;\n\t"
        "addc.cc.u32 %3, %16, %28;\n\t"
        "addc.cc.u32 %4, %17, %29;\n\t"
        "addc.cc.u32 %5, %18, %30;\n\t"
        "addc.cc.u32 %6, %19, %31;\n\t"
        "addc.cc.u32 %7, %20, %32;\n\t"
        "addc.cc.u32 %8, %21, %33;\n\t"
        "addc.cc.u32 %9, %22, %34;\n\t"
        "addc.cc.u32 %10, %23, %35;\n\t"
        "addc.cc.u32 %11, %24, %36;\n\t"
        "addc.u32 %12, 0, 0;"
        : "=r"(p[1]), "=r"(p[2]), "=r"(p[3]), "=r"(p[4]), "=r"(p[5]), "=r"(p[6]), "=r"(p[7]), "=r"(p[8]),
          "=r"(p[9]), "=r"(p[10]), "=r"(p[11]), "=r"(p[12]), "=r"(c)
        : "r"(A[1]), "r"(A[2]), "r"(A[3]), "r"(A[4]), "r"(A[5]), "r"(A[6]), "r"(A[7]), "r"(A[8]), "r"(A[9]),
          "r"(A[10]), "r"(A[11]), "r"(A[12]), "r"(B[0]), "r"(B[1]), "r"(B[2]), "r"(B[3]), "r"(B[4]), "r"(B[5]),
          "r"(B[6]), "r"(B[7]), "r"(B[8]), "r"(B[9]), "r"(B[10]), "r"(B[11]));
    asm("add.cc.u32 %11, %11, 0xffffffff;\n\t"
        "addc.cc.u32 %0, %12, %23;\n\t"
        "addc.cc.u32 %1, %13, %24;\n\t"
        "addc.cc.u32 %2, %14, %25;\n\t"
        "addc.cc.u32 %3, %15, %26;\n\t"
        "addc.cc.u32 %4, %16, %27;\n\t"
        "addc.cc.u32 %5, %17, %28;\n\t"
        "addc.cc.u32 %6, %18, %29;\n\t"
        "addc.cc.u32 %7, %19, %30;\n\t"
        "addc.cc.u32 %8, %20, %31;\n\t"
        "addc.cc.u32 %9, %21, %32;\n\t"
        "addc.u32 %10, %22, %33;"
        : "=r"(p[13]), "=r"(p[14]), "=r"(p[15]), "=r"(p[16]), "=r"(p[17]), "=r"(p[18]), "=r"(p[19]),
          "=r"(p[20]), "=r"(p[21]), "=r"(p[22]), "=r"(p[23]), "+r"(c)
        : "r"(A[13]), "r"(A[14]), "r"(A[15]), "r"(A[16]), "r"(A[17]), "r"(A[18]), "r"(A[19]), "r"(A[20]),
          "r"(A[21]), "r"(A[22]), "r"(A[23]), "r"(B[12]), "r"(B[13]), "r"(B[14]), "r"(B[15]), "r"(B[16]),
          "r"(B[17]), "r"(B[18]), "r"(B[19]), "r"(B[20]), "r"(B[21]), "r"(B[22]));
}

// p[0..23] = a * b by one level of Karatsuba on 6-limb halves: L = a0 b0,
// H = a1 b1, M = (a0 + a1)(b0 + b1) with the halves' carry bits folded in,
// p = L + (M - L - H) 2^192 + H 2^384.  Three 6 x 6 products (108 paired
// multiply-adds) instead of 144; the sums and corrections are plain adds, on
// the pipe that the multiplies leave free.  Twelve warps an SM, operands from
// shared memory and the product accumulated: 57.3 G products/s on 148 SMs
// (bls_limb_layout_rates), against 41.4 G over separate mul.lo and mul.hi rows.
__device__ __forceinline__ void prod24k(uint32_t* p, const uint32_t* a, const uint32_t* b) {
    uint32_t sa[6], sb[6], ca, cb;
    asm("add.cc.u32 %0, %7, %13;\n\t"
        "addc.cc.u32 %1, %8, %14;\n\t"
        "addc.cc.u32 %2, %9, %15;\n\t"
        "addc.cc.u32 %3, %10, %16;\n\t"
        "addc.cc.u32 %4, %11, %17;\n\t"
        "addc.cc.u32 %5, %12, %18;\n\t"
        "addc.u32 %6, 0, 0;"
        : "=r"(sa[0]), "=r"(sa[1]), "=r"(sa[2]), "=r"(sa[3]), "=r"(sa[4]), "=r"(sa[5]), "=r"(ca)
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]),
          "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]));
    asm("add.cc.u32 %0, %7, %13;\n\t"
        "addc.cc.u32 %1, %8, %14;\n\t"
        "addc.cc.u32 %2, %9, %15;\n\t"
        "addc.cc.u32 %3, %10, %16;\n\t"
        "addc.cc.u32 %4, %11, %17;\n\t"
        "addc.cc.u32 %5, %12, %18;\n\t"
        "addc.u32 %6, 0, 0;"
        : "=r"(sb[0]), "=r"(sb[1]), "=r"(sb[2]), "=r"(sb[3]), "=r"(sb[4]), "=r"(sb[5]), "=r"(cb)
        : "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]),
          "r"(b[6]), "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]), "r"(b[11]));
    uint32_t m[13];
    mul6(p, a, b);
    mul6(p + 12, a + 6, b + 6);
    mul6(m, sa, sb);
    // + ca sb 2^192 + cb sa 2^192 + ca cb 2^384 (m stays below 2^386)
    const uint32_t ma = 0u - ca, mb = 0u - cb;
    asm("add.cc.u32 %0, %0, %7;\n\t"
        "addc.cc.u32 %1, %1, %8;\n\t"
        "addc.cc.u32 %2, %2, %9;\n\t"
        "addc.cc.u32 %3, %3, %10;\n\t"
        "addc.cc.u32 %4, %4, %11;\n\t"
        "addc.cc.u32 %5, %5, %12;\n\t"
        "addc.u32 %6, %13, 0;"
        : "+r"(m[6]), "+r"(m[7]), "+r"(m[8]), "+r"(m[9]), "+r"(m[10]), "+r"(m[11]), "=r"(m[12])
        : "r"(sb[0] & ma), "r"(sb[1] & ma), "r"(sb[2] & ma), "r"(sb[3] & ma), "r"(sb[4] & ma), "r"(sb[5] & ma),
          "r"(ca & cb));
    asm("add.cc.u32 %0, %0, %7;\n\t"
        "addc.cc.u32 %1, %1, %8;\n\t"
        "addc.cc.u32 %2, %2, %9;\n\t"
        "addc.cc.u32 %3, %3, %10;\n\t"
        "addc.cc.u32 %4, %4, %11;\n\t"
        "addc.cc.u32 %5, %5, %12;\n\t"
        "addc.u32 %6, %6, 0;"
        : "+r"(m[6]), "+r"(m[7]), "+r"(m[8]), "+r"(m[9]), "+r"(m[10]), "+r"(m[11]), "+r"(m[12])
        : "r"(sa[0] & mb), "r"(sa[1] & mb), "r"(sa[2] & mb), "r"(sa[3] & mb), "r"(sa[4] & mb), "r"(sa[5] & mb));
    // m -= L, m -= H: a0 b1 + a1 b0, below 2^385
    BLS_SUB13_12(m, p);
    BLS_SUB13_12(m, p + 12);
    // p[6..23] += m[0..12]
    BLS_ADD_MID(p, m);
}

// acc[12..25] += x (neg = 0) or -= x (neg = 1): acc += +-x 2^384, modulo 2^832
__device__ __forceinline__ void acc_add_hi(uint32_t* acc, const uint32_t* x, uint32_t neg) {
    uint32_t c = neg, m = 0u - neg;
#pragma unroll
    for (int i = 0; i < 14; ++i) {
        const uint64_t s = (uint64_t)acc[12 + i] + ((i < 12 ? x[i] : 0u) ^ m) + c;
        acc[12 + i] = (uint32_t)s;
        c = (uint32_t)(s >> 32);
    }
}

// acc[0..25] -= p (24 limbs), modulo 2^832
__device__ __forceinline__ void acc_sub(uint32_t* acc, const uint32_t* p) {
    asm("sub.cc.u32 %0, %0, %26;\n\t"
        "subc.cc.u32 %1, %1, %27;\n\t"
        "subc.cc.u32 %2, %2, %28;\n\t"
        "subc.cc.u32 %3, %3, %29;\n\t"
        "subc.cc.u32 %4, %4, %30;\n\t"
        "subc.cc.u32 %5, %5, %31;\n\t"
        "subc.cc.u32 %6, %6, %32;\n\t"
        "subc.cc.u32 %7, %7, %33;\n\t"
        "subc.cc.u32 %8, %8, %34;\n\t"
        "subc.cc.u32 %9, %9, %35;\n\t"
        "subc.cc.u32 %10, %10, %36;\n\t"
        "subc.cc.u32 %11, %11, %37;\n\t"
        "subc.cc.u32 %12, %12, %38;\n\t"
        "subc.cc.u32 %13, %13, %39;\n\t"
        "subc.cc.u32 %14, %14, %40;\n\t"
        "subc.cc.u32 %15, %15, %41;\n\t"
        "subc.cc.u32 %16, %16, %42;\n\t"
        "subc.cc.u32 %17, %17, %43;\n\t"
        "subc.cc.u32 %18, %18, %44;\n\t"
        "subc.cc.u32 %19, %19, %45;\n\t"
        "subc.cc.u32 %20, %20, %46;\n\t"
        "subc.cc.u32 %21, %21, %47;\n\t"
        "subc.cc.u32 %22, %22, %48;\n\t"
        "subc.cc.u32 %23, %23, %49;\n\t"
        "subc.cc.u32 %24, %24, 0;\n\t"
        "subc.u32 %25, %25, 0;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]),
          "+r"(acc[7]), "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]),
          "+r"(acc[14]), "+r"(acc[15]), "+r"(acc[16]), "+r"(acc[17]), "+r"(acc[18]), "+r"(acc[19]),
          "+r"(acc[20]), "+r"(acc[21]), "+r"(acc[22]), "+r"(acc[23]), "+r"(acc[24]), "+r"(acc[25])
        : "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]), "r"(p[8]),
          "r"(p[9]), "r"(p[10]), "r"(p[11]), "r"(p[12]), "r"(p[13]), "r"(p[14]), "r"(p[15]), "r"(p[16]),
          "r"(p[17]), "r"(p[18]), "r"(p[19]), "r"(p[20]), "r"(p[21]), "r"(p[22]), "r"(p[23]));
}

// acc[0..25] += p[0..25], modulo 2^832
__device__ __forceinline__ void add26(uint32_t* acc, const uint32_t* p) {
    asm("add.cc.u32 %0, %0, %26;\n\t"
        "addc.cc.u32 %1, %1, %27;\n\t"
        "addc.cc.u32 %2, %2, %28;\n\t"
        "addc.cc.u32 %3, %3, %29;\n\t"
        "addc.cc.u32 %4, %4, %30;\n\t"
        "addc.cc.u32 %5, %5, %31;\n\t"
        "addc.cc.u32 %6, %6, %32;\n\t"
        "addc.cc.u32 %7, %7, %33;\n\t"
        "addc.cc.u32 %8, %8, %34;\n\t"
        "addc.cc.u32 %9, %9, %35;\n\t"
        "addc.cc.u32 %10, %10, %36;\n\t"
        "addc.cc.u32 %11, %11, %37;\n\t"
        "addc.cc.u32 %12, %12, %38;\n\t"
        "addc.cc.u32 %13, %13, %39;\n\t"
        "addc.cc.u32 %14, %14, %40;\n\t"
        "addc.cc.u32 %15, %15, %41;\n\t"
        "addc.cc.u32 %16, %16, %42;\n\t"
        "addc.cc.u32 %17, %17, %43;\n\t"
        "addc.cc.u32 %18, %18, %44;\n\t"
        "addc.cc.u32 %19, %19, %45;\n\t"
        "addc.cc.u32 %20, %20, %46;\n\t"
        "addc.cc.u32 %21, %21, %47;\n\t"
        "addc.cc.u32 %22, %22, %48;\n\t"
        "addc.cc.u32 %23, %23, %49;\n\t"
        "addc.cc.u32 %24, %24, %50;\n\t"
        "addc.u32 %25, %25, %51;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]), "+r"(acc[7]), "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]), "+r"(acc[14]), "+r"(acc[15]), "+r"(acc[16]), "+r"(acc[17]), "+r"(acc[18]), "+r"(acc[19]), "+r"(acc[20]), "+r"(acc[21]), "+r"(acc[22]), "+r"(acc[23]), "+r"(acc[24]), "+r"(acc[25])
        : "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]), "r"(p[8]), "r"(p[9]), "r"(p[10]), "r"(p[11]), "r"(p[12]), "r"(p[13]), "r"(p[14]), "r"(p[15]), "r"(p[16]), "r"(p[17]), "r"(p[18]), "r"(p[19]), "r"(p[20]), "r"(p[21]), "r"(p[22]), "r"(p[23]), "r"(p[24]), "r"(p[25]));
}

// acc[0..25] += p (24 limbs), modulo 2^832
__device__ __forceinline__ void acc_plus(uint32_t* acc, const uint32_t* p) {
    asm("add.cc.u32 %0, %0, %26;\n\t"
        "addc.cc.u32 %1, %1, %27;\n\t"
        "addc.cc.u32 %2, %2, %28;\n\t"
        "addc.cc.u32 %3, %3, %29;\n\t"
        "addc.cc.u32 %4, %4, %30;\n\t"
        "addc.cc.u32 %5, %5, %31;\n\t"
        "addc.cc.u32 %6, %6, %32;\n\t"
        "addc.cc.u32 %7, %7, %33;\n\t"
        "addc.cc.u32 %8, %8, %34;\n\t"
        "addc.cc.u32 %9, %9, %35;\n\t"
        "addc.cc.u32 %10, %10, %36;\n\t"
        "addc.cc.u32 %11, %11, %37;\n\t"
        "addc.cc.u32 %12, %12, %38;\n\t"
        "addc.cc.u32 %13, %13, %39;\n\t"
        "addc.cc.u32 %14, %14, %40;\n\t"
        "addc.cc.u32 %15, %15, %41;\n\t"
        "addc.cc.u32 %16, %16, %42;\n\t"
        "addc.cc.u32 %17, %17, %43;\n\t"
        "addc.cc.u32 %18, %18, %44;\n\t"
        "addc.cc.u32 %19, %19, %45;\n\t"
        "addc.cc.u32 %20, %20, %46;\n\t"
        "addc.cc.u32 %21, %21, %47;\n\t"
        "addc.cc.u32 %22, %22, %48;\n\t"
        "addc.cc.u32 %23, %23, %49;\n\t"
        "addc.cc.u32 %24, %24, 0;\n\t"
        "addc.u32 %25, %25, 0;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]),
          "+r"(acc[7]), "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]),
          "+r"(acc[14]), "+r"(acc[15]), "+r"(acc[16]), "+r"(acc[17]), "+r"(acc[18]), "+r"(acc[19]),
          "+r"(acc[20]), "+r"(acc[21]), "+r"(acc[22]), "+r"(acc[23]), "+r"(acc[24]), "+r"(acc[25])
        : "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]), "r"(p[8]),
          "r"(p[9]), "r"(p[10]), "r"(p[11]), "r"(p[12]), "r"(p[13]), "r"(p[14]), "r"(p[15]), "r"(p[16]),
          "r"(p[17]), "r"(p[18]), "r"(p[19]), "r"(p[20]), "r"(p[21]), "r"(p[22]), "r"(p[23]));
}

// x = 2 x (12 limbs; x below 2^383)
__device__ __forceinline__ void dbl12(uint32_t* x) {
#pragma unroll
    for (int i = 11; i > 0; --i) x[i] = __funnelshift_l(x[i - 1], x[i], 1);
    x[0] <<= 1;
}

// t[0..12] = k * p for a small k (k < 2^32)
__device__ __forceinline__ void set_kp(uint32_t* t, uint32_t k) {
#pragma unroll
    for (int i = 0; i < 13; ++i) t[i] = 0;
    chain_lo_p(t, k);
    chain_hi_p(t, k);
}

// Montgomery reduction of a 26-limb accumulator (value below 2^771):
// r[0..12] = acc / 2^384 mod p, as acc_hi + (acc_lo + M p) / 2^384 (below 2^388).
// The low half is reduced in twelve rows on paired columns (mont_reduce12).
__device__ __forceinline__ void redc26(uint32_t* r, const uint32_t* acc) {
    uint32_t t[12];
    mont_reduce12(t, acc);
    asm("add.cc.u32 %0, %13, %26;\n\t"
        "addc.cc.u32 %1, %14, %27;\n\t"
        "addc.cc.u32 %2, %15, %28;\n\t"
        "addc.cc.u32 %3, %16, %29;\n\t"
        "addc.cc.u32 %4, %17, %30;\n\t"
        "addc.cc.u32 %5, %18, %31;\n\t"
        "addc.cc.u32 %6, %19, %32;\n\t"
        "addc.cc.u32 %7, %20, %33;\n\t"
        "addc.cc.u32 %8, %21, %34;\n\t"
        "addc.cc.u32 %9, %22, %35;\n\t"
        "addc.cc.u32 %10, %23, %36;\n\t"
        "addc.cc.u32 %11, %24, %37;\n\t"
        "addc.u32 %12, %25, 0;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12])
        : "r"(acc[12]), "r"(acc[13]), "r"(acc[14]), "r"(acc[15]), "r"(acc[16]), "r"(acc[17]), "r"(acc[18]),
          "r"(acc[19]), "r"(acc[20]), "r"(acc[21]), "r"(acc[22]), "r"(acc[23]), "r"(acc[24]),
          "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]), "r"(t[8]),
          "r"(t[9]), "r"(t[10]), "r"(t[11]));
}

// out = v - q (12 limbs; q = QP[v >> 381] in four 16-byte units)
__device__ __forceinline__ void qp_subtract(uint32_t* out, const uint32_t* v, const uint4& q0, const uint4& q1,
                                            const uint4& q2, const uint4& q3) {
    uint32_t top;
    asm("sub.cc.u32 %0, %13, %26;\n\t"
        "subc.cc.u32 %1, %14, %27;\n\t"
        "subc.cc.u32 %2, %15, %28;\n\t"
        "subc.cc.u32 %3, %16, %29;\n\t"
        "subc.cc.u32 %4, %17, %30;\n\t"
        "subc.cc.u32 %5, %18, %31;\n\t"
        "subc.cc.u32 %6, %19, %32;\n\t"
        "subc.cc.u32 %7, %20, %33;\n\t"
        "subc.cc.u32 %8, %21, %34;\n\t"
        "subc.cc.u32 %9, %22, %35;\n\t"
        "subc.cc.u32 %10, %23, %36;\n\t"
        "subc.cc.u32 %11, %24, %37;\n\t"
        "subc.u32 %12, %25, %38;"
        : "=r"(out[0]), "=r"(out[1]), "=r"(out[2]), "=r"(out[3]), "=r"(out[4]), "=r"(out[5]), "=r"(out[6]),
          "=r"(out[7]), "=r"(out[8]), "=r"(out[9]), "=r"(out[10]), "=r"(out[11]), "=r"(top)
        : "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(q0.x), "r"(q0.y), "r"(q0.z), "r"(q0.w), "r"(q1.x),
          "r"(q1.y), "r"(q1.z), "r"(q1.w), "r"(q2.x), "r"(q2.y), "r"(q2.z), "r"(q2.w), "r"(q3.x));
    (void)top;  // zero: v - QP[h] < 2^384
}

// v (13 limbs, below 2^388) -> v - QP[v >> 381], below 2^381 + p (12 limbs)
__device__ __forceinline__ void qp_reduce(uint32_t* out, const uint32_t* v) {
    const uint32_t h = (v[12] << 3) | (v[11] >> 29);
    const uint4* q = reinterpret_cast<const uint4*>(kQP2[h & 127]);
    qp_subtract(out, v, __ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
}

// the same with the QP table copied into shared memory, unit j of entry e at
// tab[128 j + e] (lanes reading different entries then spread over the banks)
__device__ __forceinline__ void qp_reduce_tab(uint32_t* out, const uint32_t* v, const uint4* tab) {
    const uint32_t h = ((v[12] << 3) | (v[11] >> 29)) & 127u;
    qp_subtract(out, v, tab[h], tab[128 + h], tab[256 + h], tab[384 + h]);
}

// r[0..12] += x[0..12]
__device__ __forceinline__ void add13(uint32_t* r, const uint32_t* x) {
    asm("add.cc.u32 %0, %0, %13;\n\t"
        "addc.cc.u32 %1, %1, %14;\n\t"
        "addc.cc.u32 %2, %2, %15;\n\t"
        "addc.cc.u32 %3, %3, %16;\n\t"
        "addc.cc.u32 %4, %4, %17;\n\t"
        "addc.cc.u32 %5, %5, %18;\n\t"
        "addc.cc.u32 %6, %6, %19;\n\t"
        "addc.cc.u32 %7, %7, %20;\n\t"
        "addc.cc.u32 %8, %8, %21;\n\t"
        "addc.cc.u32 %9, %9, %22;\n\t"
        "addc.cc.u32 %10, %10, %23;\n\t"
        "addc.cc.u32 %11, %11, %24;\n\t"
        "addc.u32 %12, %12, %25;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
          "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(x[8]),
          "r"(x[9]), "r"(x[10]), "r"(x[11]), "r"(x[12]));
}
// r[0..12] += x and r[0..12] -= x (12 limbs), modulo 2^416
__device__ __forceinline__ void add13_12(uint32_t* r, const uint32_t* x) {
    asm("add.cc.u32 %0, %0, %13;\n\t"
        "addc.cc.u32 %1, %1, %14;\n\t"
        "addc.cc.u32 %2, %2, %15;\n\t"
        "addc.cc.u32 %3, %3, %16;\n\t"
        "addc.cc.u32 %4, %4, %17;\n\t"
        "addc.cc.u32 %5, %5, %18;\n\t"
        "addc.cc.u32 %6, %6, %19;\n\t"
        "addc.cc.u32 %7, %7, %20;\n\t"
        "addc.cc.u32 %8, %8, %21;\n\t"
        "addc.cc.u32 %9, %9, %22;\n\t"
        "addc.cc.u32 %10, %10, %23;\n\t"
        "addc.cc.u32 %11, %11, %24;\n\t"
        "addc.u32 %12, %12, %25;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
          "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(x[8]),
          "r"(x[9]), "r"(x[10]), "r"(x[11]), "r"(0u));
}
__device__ __forceinline__ void sub13_12(uint32_t* r, const uint32_t* x) {
    asm("sub.cc.u32 %0, %0, %13;\n\t"
        "subc.cc.u32 %1, %1, %14;\n\t"
        "subc.cc.u32 %2, %2, %15;\n\t"
        "subc.cc.u32 %3, %3, %16;\n\t"
        "subc.cc.u32 %4, %4, %17;\n\t"
        "subc.cc.u32 %5, %5, %18;\n\t"
        "subc.cc.u32 %6, %6, %19;\n\t"
        "subc.cc.u32 %7, %7, %20;\n\t"
        "subc.cc.u32 %8, %8, %21;\n\t"
        "subc.cc.u32 %9, %9, %22;\n\t"
        "subc.cc.u32 %10, %10, %23;\n\t"
        "subc.cc.u32 %11, %11, %24;\n\t"
        "subc.u32 %12, %12, %25;"
        : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
          "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(x[8]),
          "r"(x[9]), "r"(x[10]), "r"(x[11]), "r"(0u));
}

// x = 2 x (13 limbs)
__device__ __forceinline__ void dbl13(uint32_t* x) {
#pragma unroll
    for (int i = 12; i > 0; --i) x[i] = __funnelshift_l(x[i - 1], x[i], 1);
    x[0] <<= 1;
}

// t[0..12] += c x (x: 12 limbs, |c| < 2^31), modulo 2^416: y = |c| x by
// shifts for |c| <= 2 (the common 1 and 2 of the programs' linear terms) or
// by one multiply chain, then one add chain of y or of its complement (no
// branch on the sign, which differs between lanes)
__device__ __forceinline__ void madd13(uint32_t* t, const uint32_t* x, int c) {
    const uint32_t a = (uint32_t)(c < 0 ? -c : c), m = c < 0 ? 0xffffffffu : 0u;
    uint32_t y[13];
    if (a <= 2u) {
#pragma unroll
        for (int i = 0; i < 12; ++i) y[i] = x[i];
        y[12] = 0;
        if (a == 2u) {
            y[12] = x[11] >> 31;
#pragma unroll
            for (int i = 11; i > 0; --i) y[i] = __funnelshift_l(x[i - 1], x[i], 1);
            y[0] = x[0] << 1;
        } else if (a == 0u) {
            return;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 13; ++i) y[i] = 0;
        chain_lo(y, x, a);
        chain_hi(y, x, a);
    }
    uint32_t cf;   // carry in = 1 for a subtraction: m + m carries out exactly when m is all ones
    asm("add.cc.u32 %13, %27, %27;\n\t"
        "addc.cc.u32 %0, %0, %14;\n\t"
        "addc.cc.u32 %1, %1, %15;\n\t"
        "addc.cc.u32 %2, %2, %16;\n\t"
        "addc.cc.u32 %3, %3, %17;\n\t"
        "addc.cc.u32 %4, %4, %18;\n\t"
        "addc.cc.u32 %5, %5, %19;\n\t"
        "addc.cc.u32 %6, %6, %20;\n\t"
        "addc.cc.u32 %7, %7, %21;\n\t"
        "addc.cc.u32 %8, %8, %22;\n\t"
        "addc.cc.u32 %9, %9, %23;\n\t"
        "addc.cc.u32 %10, %10, %24;\n\t"
        "addc.cc.u32 %11, %11, %25;\n\t"
        "addc.u32 %12, %12, %26;"
        : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
          "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "+r"(t[12]), "=r"(cf)
        : "r"(y[0] ^ m), "r"(y[1] ^ m), "r"(y[2] ^ m), "r"(y[3] ^ m), "r"(y[4] ^ m), "r"(y[5] ^ m), "r"(y[6] ^ m),
          "r"(y[7] ^ m), "r"(y[8] ^ m), "r"(y[9] ^ m), "r"(y[10] ^ m), "r"(y[11] ^ m), "r"(y[12] ^ m), "r"(m));
    (void)cf;
}

// acc[0..24] += p (24 limbs), modulo 2^800
__device__ __forceinline__ void add25(uint32_t* acc, const uint32_t* p) {
    asm("add.cc.u32 %0, %0, %25;\n\t"
        "addc.cc.u32 %1, %1, %26;\n\t"
        "addc.cc.u32 %2, %2, %27;\n\t"
        "addc.cc.u32 %3, %3, %28;\n\t"
        "addc.cc.u32 %4, %4, %29;\n\t"
        "addc.cc.u32 %5, %5, %30;\n\t"
        "addc.cc.u32 %6, %6, %31;\n\t"
        "addc.cc.u32 %7, %7, %32;\n\t"
        "addc.cc.u32 %8, %8, %33;\n\t"
        "addc.cc.u32 %9, %9, %34;\n\t"
        "addc.cc.u32 %10, %10, %35;\n\t"
        "addc.cc.u32 %11, %11, %36;\n\t"
        "addc.cc.u32 %12, %12, %37;\n\t"
        "addc.cc.u32 %13, %13, %38;\n\t"
        "addc.cc.u32 %14, %14, %39;\n\t"
        "addc.cc.u32 %15, %15, %40;\n\t"
        "addc.cc.u32 %16, %16, %41;\n\t"
        "addc.cc.u32 %17, %17, %42;\n\t"
        "addc.cc.u32 %18, %18, %43;\n\t"
        "addc.cc.u32 %19, %19, %44;\n\t"
        "addc.cc.u32 %20, %20, %45;\n\t"
        "addc.cc.u32 %21, %21, %46;\n\t"
        "addc.cc.u32 %22, %22, %47;\n\t"
        "addc.cc.u32 %23, %23, %48;\n\t"
        "addc.u32 %24, %24, %49;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]),
          "+r"(acc[7]), "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]),
          "+r"(acc[14]), "+r"(acc[15]), "+r"(acc[16]), "+r"(acc[17]), "+r"(acc[18]), "+r"(acc[19]),
          "+r"(acc[20]), "+r"(acc[21]), "+r"(acc[22]), "+r"(acc[23]), "+r"(acc[24])
        : "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]), "r"(p[8]),
          "r"(p[9]), "r"(p[10]), "r"(p[11]), "r"(p[12]), "r"(p[13]), "r"(p[14]), "r"(p[15]), "r"(p[16]),
          "r"(p[17]), "r"(p[18]), "r"(p[19]), "r"(p[20]), "r"(p[21]), "r"(p[22]), "r"(p[23]), "r"(0u));
}
// acc[0..24] += p[0..24] and acc[0..24] -= p[0..24], modulo 2^800
__device__ __forceinline__ void add25_25(uint32_t* acc, const uint32_t* p) {
    asm("add.cc.u32 %0, %0, %25;\n\t"
        "addc.cc.u32 %1, %1, %26;\n\t"
        "addc.cc.u32 %2, %2, %27;\n\t"
        "addc.cc.u32 %3, %3, %28;\n\t"
        "addc.cc.u32 %4, %4, %29;\n\t"
        "addc.cc.u32 %5, %5, %30;\n\t"
        "addc.cc.u32 %6, %6, %31;\n\t"
        "addc.cc.u32 %7, %7, %32;\n\t"
        "addc.cc.u32 %8, %8, %33;\n\t"
        "addc.cc.u32 %9, %9, %34;\n\t"
        "addc.cc.u32 %10, %10, %35;\n\t"
        "addc.cc.u32 %11, %11, %36;\n\t"
        "addc.cc.u32 %12, %12, %37;\n\t"
        "addc.cc.u32 %13, %13, %38;\n\t"
        "addc.cc.u32 %14, %14, %39;\n\t"
        "addc.cc.u32 %15, %15, %40;\n\t"
        "addc.cc.u32 %16, %16, %41;\n\t"
        "addc.cc.u32 %17, %17, %42;\n\t"
        "addc.cc.u32 %18, %18, %43;\n\t"
        "addc.cc.u32 %19, %19, %44;\n\t"
        "addc.cc.u32 %20, %20, %45;\n\t"
        "addc.cc.u32 %21, %21, %46;\n\t"
        "addc.cc.u32 %22, %22, %47;\n\t"
        "addc.cc.u32 %23, %23, %48;\n\t"
        "addc.u32 %24, %24, %49;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]),
          "+r"(acc[7]), "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]),
          "+r"(acc[14]), "+r"(acc[15]), "+r"(acc[16]), "+r"(acc[17]), "+r"(acc[18]), "+r"(acc[19]),
          "+r"(acc[20]), "+r"(acc[21]), "+r"(acc[22]), "+r"(acc[23]), "+r"(acc[24])
        : "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]), "r"(p[8]),
          "r"(p[9]), "r"(p[10]), "r"(p[11]), "r"(p[12]), "r"(p[13]), "r"(p[14]), "r"(p[15]), "r"(p[16]),
          "r"(p[17]), "r"(p[18]), "r"(p[19]), "r"(p[20]), "r"(p[21]), "r"(p[22]), "r"(p[23]), "r"(p[24]));
}
__device__ __forceinline__ void sub25_25(uint32_t* acc, const uint32_t* p) {
    asm("sub.cc.u32 %0, %0, %25;\n\t"
        "subc.cc.u32 %1, %1, %26;\n\t"
        "subc.cc.u32 %2, %2, %27;\n\t"
        "subc.cc.u32 %3, %3, %28;\n\t"
        "subc.cc.u32 %4, %4, %29;\n\t"
        "subc.cc.u32 %5, %5, %30;\n\t"
        "subc.cc.u32 %6, %6, %31;\n\t"
        "subc.cc.u32 %7, %7, %32;\n\t"
        "subc.cc.u32 %8, %8, %33;\n\t"
        "subc.cc.u32 %9, %9, %34;\n\t"
        "subc.cc.u32 %10, %10, %35;\n\t"
        "subc.cc.u32 %11, %11, %36;\n\t"
        "subc.cc.u32 %12, %12, %37;\n\t"
        "subc.cc.u32 %13, %13, %38;\n\t"
        "subc.cc.u32 %14, %14, %39;\n\t"
        "subc.cc.u32 %15, %15, %40;\n\t"
        "subc.cc.u32 %16, %16, %41;\n\t"
        "subc.cc.u32 %17, %17, %42;\n\t"
        "subc.cc.u32 %18, %18, %43;\n\t"
        "subc.cc.u32 %19, %19, %44;\n\t"
        "subc.cc.u32 %20, %20, %45;\n\t"
        "subc.cc.u32 %21, %21, %46;\n\t"
        "subc.cc.u32 %22, %22, %47;\n\t"
        "subc.cc.u32 %23, %23, %48;\n\t"
        "subc.u32 %24, %24, %49;"
        : "+r"(acc[0]), "+r"(acc[1]), "+r"(acc[2]), "+r"(acc[3]), "+r"(acc[4]), "+r"(acc[5]), "+r"(acc[6]),
          "+r"(acc[7]), "+r"(acc[8]), "+r"(acc[9]), "+r"(acc[10]), "+r"(acc[11]), "+r"(acc[12]), "+r"(acc[13]),
          "+r"(acc[14]), "+r"(acc[15]), "+r"(acc[16]), "+r"(acc[17]), "+r"(acc[18]), "+r"(acc[19]),
          "+r"(acc[20]), "+r"(acc[21]), "+r"(acc[22]), "+r"(acc[23]), "+r"(acc[24])
        : "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(p[4]), "r"(p[5]), "r"(p[6]), "r"(p[7]), "r"(p[8]),
          "r"(p[9]), "r"(p[10]), "r"(p[11]), "r"(p[12]), "r"(p[13]), "r"(p[14]), "r"(p[15]), "r"(p[16]),
          "r"(p[17]), "r"(p[18]), "r"(p[19]), "r"(p[20]), "r"(p[21]), "r"(p[22]), "r"(p[23]), "r"(p[24]));
}

// r = a + b (12 limbs, no carry out: both below 2^383)
__device__ __forceinline__ void add12(uint32_t* r, const uint32_t* a, const uint32_t* b) {
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
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11])
        : BLS_A12(a), BLS_A12(b));
}

// x = 3p - x and x = 5p - x (12 limbs), the multiples as immediates (reading them
// from constant memory is slower)
__device__ __forceinline__ void sub_from_3p(uint32_t* x) {
    asm("sub.cc.u32 %0, 0xffff0001, %0;\n\t"
        "subc.cc.u32 %1, 0x2dfcffff, %1;\n\t"
        "subc.cc.u32 %2, 0x13fbffff, %2;\n\t"
        "subc.cc.u32 %3, 0x5c03fffc, %3;\n\t"
        "subc.cc.u32 %4, 0xe412e26c, %4;\n\t"
        "subc.cc.u32 %5, 0x359277e2, %5;\n\t"
        "subc.cc.u32 %6, 0xda8f383e, %6;\n\t"
        "subc.cc.u32 %7, 0x2d65e28e, %7;\n\t"
        "subc.cc.u32 %8, 0xc9e30686, %8;\n\t"
        "subc.cc.u32 %9, 0xe152f722, %9;\n\t"
        "subc.cc.u32 %10, 0xac7fb3ce, %10;\n\t"
        "subc.u32 %11, 0x4e0335be, %11;"
        : BLS_T12(x));
}
__device__ __forceinline__ void sub_from_5p(uint32_t* x) {
    asm("sub.cc.u32 %0, 0xfffe5557, %0;\n\t"
        "subc.cc.u32 %1, 0xa1faffff, %1;\n\t"
        "subc.cc.u32 %2, 0x76a3fffe, %2;\n\t"
        "subc.cc.u32 %3, 0x995bfff9, %3;\n\t"
        "subc.cc.u32 %4, 0xd174ceb4, %4;\n\t"
        "subc.cc.u32 %5, 0x03f41d24, %5;\n\t"
        "subc.cc.u32 %6, 0xc1995dbd, %6;\n\t"
        "subc.cc.u32 %7, 0xf6547998, %7;\n\t"
        "subc.cc.u32 %8, 0x507a6034, %8;\n\t"
        "subc.cc.u32 %9, 0x778a468f, %9;\n\t"
        "subc.cc.u32 %10, 0x1f7f8103, %10;\n\t"
        "subc.u32 %11, 0x82055993, %11;"
        : BLS_T12(x));
}

// r = a + 3p - b (12 limbs; a, b below 2^381 + p, result below 2^384)
__device__ __forceinline__ void add3p_sub(uint32_t* r, const uint32_t* a, const uint32_t* b) {
    uint32_t t[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) t[i] = b[i];
    sub_from_3p(t);
    add12(r, t, a);
}

}  // namespace f2
}  // namespace bls
