// Fp inverse by Bernstein and Yang's division steps ("Fast constant-time gcd
// computation and modular inversion", CHES 2019), counting delta in halves and in
// thirty-bit limbs as in the public description of libsecp256k1's inverse (Dettman,
// Wuille: doc/safegcd_implementation.md of that project), shared by the verify kernels
// (the final exponentiation's one inversion), the line tables and the hash to G1.
//
// One step takes (delta, f, g), f odd, to
//   (2 - delta, g, (g - f) / 2)             when delta > 0 and g is odd,
//   (2 + delta, f, (g + (g mod 2) f) / 2)   otherwise
// (delta counted in halves, from 1), and after enough steps g = 0 and f = +-gcd.
// Thirty steps look at no more than the low thirty bits of f and g, so they run on
// one word each and leave a 2 x 2 matrix of words, which is then applied to the
// whole of f and g (an exact division by 2^30) and, with a multiple of p added to
// make the division exact, to d and e, where f = d x and g = e x modulo p.
//
// Values are signed, in thirteen limbs of thirty bits, so that a limb product is
// one signed wide multiply-add and there are no carry chains.  Nothing branches
// on the value but the end of the loop (26 or 27 rounds for 381 bits), so the
// lanes of a warp invert different values side by side, bound by one warp's
// dependent chain.  A binary Euclid diverges; with one on the product of the warp's
// values (prefix and suffix products by shuffles), which avoids that, the verify
// kernel took 3.60 instead of 3.50 ms.
#pragma once
#include "fp.cuh"

namespace bls {

constexpr int kInvLimbs = 13, kInvBits = 30;
constexpr int32_t kInvMask = (1 << kInvBits) - 1;
// Theorem 11.2 of the paper: (49 * 381 + 57) / 17 = 1,101 steps suffice from delta = 1
// (741 for 256 bits).  From 1/2 fewer do: 590 for 256 bits in the description named
// above.  The loop ends when g is zero, after at most 1,110 steps.
constexpr int kInvMaxRounds = 37;

__device__ __forceinline__ void inv_limbs(int32_t* r, const uint32_t* w) {
#pragma unroll
    for (int i = 0; i < kInvLimbs; ++i) {
        const int b = kInvBits * i, k = b >> 5, s = b & 31;
        const uint32_t lo = w[k], hi = k + 1 < 12 ? w[k + 1] : 0u;
        r[i] = (int32_t)(__funnelshift_r(lo, hi, s) & (uint32_t)kInvMask);
    }
}

// x: Montgomery form of a (any value below 2^381 + p); a^-1 in Montgomery form,
// 0 for 0.  kR3: R^3 mod p, which takes the plain inverse x^-1 there.
static __device__ __noinline__ fp fp_inverse_mont(fp x, const uint32_t* kR3) {
    // canonical representative (x < 2^381 + p < 3p)
    reduce_once(x.w);
    reduce_once(x.w);
    uint32_t t[13];
    const uint32_t P_[12] = {BLS_P0, BLS_P1, BLS_P2, BLS_P3, BLS_P4, BLS_P5,
                             BLS_P6, BLS_P7, BLS_P8, BLS_P9, BLS_P10, BLS_P11};
    int32_t P30[kInvLimbs], f[kInvLimbs], g[kInvLimbs], d[kInvLimbs], e[kInvLimbs];
    inv_limbs(P30, P_);
    inv_limbs(g, x.w);
#pragma unroll
    for (int i = 0; i < kInvLimbs; ++i) {
        f[i] = P30[i];
        d[i] = 0;
        e[i] = i == 0 ? 1 : 0;
    }
    int delta = 1;
#pragma unroll 1
    for (int round = 0; round < kInvMaxRounds; ++round) {
        int32_t any = 0;
#pragma unroll
        for (int i = 0; i < kInvLimbs; ++i) any |= g[i];
        if (any == 0) break;
        // thirty steps on the low words: 2^i f_i = u f + v g, 2^i g_i = q f + r g
        int32_t u = 1, v = 0, q = 0, r = 1;
        uint32_t f0 = (uint32_t)f[0] | ((uint32_t)f[1] << kInvBits), g0 = (uint32_t)g[0] | ((uint32_t)g[1] << kInvBits);
#pragma unroll 6
        for (int i = 0; i < kInvBits; ++i) {
            const bool odd = g0 & 1u, swap = odd && delta > 0;
            const uint32_t af = odd ? (swap ? 0u - f0 : f0) : 0u;
            const int32_t au = odd ? (swap ? -u : u) : 0, av = odd ? (swap ? -v : v) : 0;
            delta = 2 + (swap ? -delta : delta);
            f0 = swap ? g0 : f0;
            u = (swap ? q : u) << 1;
            v = (swap ? r : v) << 1;
            g0 = (g0 + af) >> 1;
            q += au;
            r += av;
        }
        // f, g = (u f + v g) / 2^30, (q f + r g) / 2^30: the low thirty bits are zero
        int64_t cf = (int64_t)u * f[0] + (int64_t)v * g[0], cg = (int64_t)q * f[0] + (int64_t)r * g[0];
        // d, e likewise, with m p added for the m < 2^30 that clears the low limb:
        // |u| + |v| <= 2^30, so |d| and |e| grow by less than p a round
        int64_t cd = (int64_t)u * d[0] + (int64_t)v * e[0], ce = (int64_t)q * d[0] + (int64_t)r * e[0];
        const int32_t md = (int32_t)((uint32_t)cd * BLS_NINV) & kInvMask, me = (int32_t)((uint32_t)ce * BLS_NINV) & kInvMask;
        cd += (int64_t)md * P30[0];
        ce += (int64_t)me * P30[0];
        cf >>= kInvBits;
        cg >>= kInvBits;
        cd >>= kInvBits;
        ce >>= kInvBits;
#pragma unroll
        for (int i = 1; i < kInvLimbs; ++i) {
            cf += (int64_t)u * f[i] + (int64_t)v * g[i];
            cg += (int64_t)q * f[i] + (int64_t)r * g[i];
            cd += (int64_t)u * d[i] + (int64_t)v * e[i] + (int64_t)md * P30[i];
            ce += (int64_t)q * d[i] + (int64_t)r * e[i] + (int64_t)me * P30[i];
            f[i - 1] = (int32_t)cf & kInvMask;
            g[i - 1] = (int32_t)cg & kInvMask;
            d[i - 1] = (int32_t)cd & kInvMask;
            e[i - 1] = (int32_t)ce & kInvMask;
            cf >>= kInvBits;
            cg >>= kInvBits;
            cd >>= kInvBits;
            ce >>= kInvBits;
        }
        f[kInvLimbs - 1] = (int32_t)cf;
        g[kInvLimbs - 1] = (int32_t)cg;
        d[kInvLimbs - 1] = (int32_t)cd;
        e[kInvLimbs - 1] = (int32_t)ce;
    }
    // f = +-1 and d x = f: |d| < 37 p, the limbs below the top one nonnegative.
    // +-d + 64 p, in 32-bit words, then the multiples of p off.
    const bool neg = f[kInvLimbs - 1] < 0;
    int64_t c = 0;
    uint64_t acc = 0;
    int bits = 0, k = 0;
#pragma unroll
    for (int i = 0; i < kInvLimbs; ++i) {
        c += (neg ? -(int64_t)d[i] : (int64_t)d[i]) + 64 * (int64_t)P30[i];
        const uint64_t limb = i == kInvLimbs - 1 ? (uint64_t)c : (uint64_t)(c & kInvMask);
        c >>= kInvBits;
        acc |= limb << bits;
        bits += kInvBits;
        if (bits >= 32) {
            t[k++] = (uint32_t)acc;
            acc >>= 32;
            bits -= 32;
        }
    }
    t[12] = (uint32_t)acc;
#pragma unroll
    for (int j = 6; j >= 0; --j) {      // below 2^(j+1) p: 2^j p off when it fits
        uint32_t w[13], br = 0;
#pragma unroll
        for (int i = 0; i < 13; ++i) {
            const uint32_t lo = i < 12 ? P_[i] << j : 0u, hi = (i > 0 && j > 0) ? P_[i - 1] >> (32 - j) : 0u;
            const uint64_t y = (uint64_t)t[i] - (lo | hi) - br;
            w[i] = (uint32_t)y;
            br = (uint32_t)(y >> 63);
        }
#pragma unroll
        for (int i = 0; i < 13; ++i) t[i] = br ? t[i] : w[i];
    }
    fp inv, r3;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        inv.w[i] = t[i];
        r3.w[i] = kR3[i];
    }
    return fp_mul(inv, r3);             // x^-1 R^3 / R: the Montgomery form of a^-1
}

}  // namespace bls
