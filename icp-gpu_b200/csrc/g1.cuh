// G1 point decoding on the device: 48-byte compressed points (ZCash BLS12-381
// format, big-endian x with three flag bits in the top of byte 0) to affine
// Montgomery (x, y), with every check ic_bls12_381's G1Affine::from_compressed
// makes.  The value path follows the reference decoder (cuda/decompress.cu:
// 44-187: y = (x^3 + 4)^((p+1)/4), sign chosen by "lexicographically largest");
// the reference performs none of the checks, which are added here:
//   compression flag set; infinity flag only with an all-zero payload and no
//   sort flag; x < p; x^3 + 4 a square; the point in the order-r subgroup.
// The subgroup test is phi(P) == -[x^2] P with phi(x, y) = (beta x, y),
// beta the cube root of unity whose eigenvalue on G1 is -x^2 (Scott, eprint
// 2021/1130 section 6; correctness proof eprint 2022/352).
#pragma once
#include "fp.cuh"

namespace bls {

enum : int32_t {
    ST_OK = 0,
    ST_BAD_FLAGS = 1,
    ST_X_NOT_CANONICAL = 2,
    ST_NOT_ON_CURVE = 3,
    ST_NOT_IN_SUBGROUP = 4,
    ST_BAD_KEY_INDEX = 5,     // not a decode status: a key id outside the tables
};

// a key id the verify kernels may read (VerifyArgs::check_keys, n_keys)
__device__ __forceinline__ bool key_index_ok(int64_t id, int check, int n_keys) {
    return !check || (id >= 0 && id < (int64_t)n_keys);
}

__device__ __forceinline__ fp fp_four() {
    fp one = fp_one();
    fp two = fp_add(one, one);
    return fp_add(two, two);
}

// a^((p+1)/4); a square root whenever one exists (p = 3 mod 4)
static __device__ __noinline__ fp fp_sqrt_candidate(const fp& a) {
    const uint64_t e[6] = {0xee7fbfffffffeaabULL, 0x07aaffffac54ffffULL, 0xd9cc34a83dac3d89ULL,
                           0xd91dd2e13ce144afULL, 0x92c6e9ed90d2eb35ULL, 0x0680447a8e5ff9a6ULL};
    return fp_pow_ool(a, e, 379);
}

// canonical value > (p - 1) / 2
__device__ __forceinline__ bool fp_lex_largest(const fp& a) {
    fp v = fp_from_mont(a);
    // (p-1)/2 = 0x0d0088f51cbff34d 258dd3db21a5d66b b23ba5c279c2895f b39869507b587b12 0f55ffff58a9ffff dcff7fffffffd555
    const uint32_t h[12] = {0xffffd555u, 0xdcff7fffu, 0x58a9ffffu, 0x0f55ffffu, 0x7b587b12u, 0xb3986950u,
                            0x79c2895fu, 0xb23ba5c2u, 0x21a5d66bu, 0x258dd3dbu, 0x1cbff34du, 0x0d0088f5u};
    int res = 0;  // 1 greater, -1 less, 0 equal (most significant difference wins)
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        if (v.w[i] > h[i]) res = 1;
        else if (v.w[i] < h[i]) res = -1;
    }
    return res > 0;
}

// Jacobian coordinates on y^2 = x^3 + 4
struct g1j { fp X, Y, Z; };

// The Jacobian routines run one thread per point, a few warps per scheduler:
// their products are the out-of-line multiply of fp.cuh, and a sum that is squared
// (below 3p) or multiplied (below 8p) next is left unreduced.
// dbl-2009-l (a = 0)
static __device__ __noinline__ g1j g1j_dbl(const g1j& p) {
    fp A = fp_sqr_ool(p.X), B = fp_sqr_ool(p.Y), C = fp_sqr_ool(B);
    fp D = fp_sub(fp_sub(fp_sqr_ool(fp_add_nr(p.X, B)), A), C);
    D = fp_add(D, D);
    fp E = fp_add_nr(fp_add_nr(A, A), A);
    fp F = fp_sqr_ool(E);
    g1j r;
    r.X = fp_sub(F, fp_add(D, D));
    fp C8 = fp_add(C, C);
    C8 = fp_add(C8, C8);
    C8 = fp_add(C8, C8);
    r.Y = fp_sub(fp_mul_ool(E, fp_sub(D, r.X)), C8);
    r.Z = fp_mul_ool(fp_add_nr(p.Y, p.Y), p.Z);
    return r;
}

// p + (qx, qy) with q affine (madd-2007-bl), exceptional cases handled
static __device__ __noinline__ g1j g1j_add_affine(const g1j& p, const fp& qx, const fp& qy) {
    if (fp_is_zero(p.Z)) return {qx, qy, fp_one()};
    fp Z1Z1 = fp_sqr_ool(p.Z);
    fp U2 = fp_mul_ool(qx, Z1Z1);
    fp S2 = fp_mul_ool(fp_mul_ool(qy, p.Z), Z1Z1);
    fp H = fp_sub(U2, p.X);
    fp rr = fp_sub(S2, p.Y);
    if (fp_is_zero(H)) {
        if (fp_is_zero(rr)) return g1j_dbl(p);
        return {fp_one(), fp_one(), fp_zero()};
    }
    rr = fp_add_nr(rr, rr);
    fp HH = fp_sqr_ool(H);
    fp I = fp_add_nr(HH, HH);
    I = fp_add_nr(I, I);
    fp J = fp_mul_ool(H, I);
    fp V = fp_mul_ool(p.X, I);
    g1j r;
    r.X = fp_sub(fp_sub(fp_sqr_ool(rr), J), fp_add(V, V));
    fp YJ = fp_mul_ool(p.Y, J);
    r.Y = fp_sub(fp_mul_ool(rr, fp_sub(V, r.X)), fp_add(YJ, YJ));
    r.Z = fp_sub(fp_sub(fp_sqr_ool(fp_add_nr(p.Z, H)), Z1Z1), HH);
    return r;
}

// p + q, both Jacobian (add-2007-bl), exceptional cases handled
static __device__ __noinline__ g1j g1j_add(const g1j& p, const g1j& q) {
    if (fp_is_zero(p.Z)) return q;
    if (fp_is_zero(q.Z)) return p;
    const fp Z1Z1 = fp_sqr_ool(p.Z), Z2Z2 = fp_sqr_ool(q.Z);
    const fp U1 = fp_mul_ool(p.X, Z2Z2), U2 = fp_mul_ool(q.X, Z1Z1);
    const fp S1 = fp_mul_ool(fp_mul_ool(p.Y, q.Z), Z2Z2), S2 = fp_mul_ool(fp_mul_ool(q.Y, p.Z), Z1Z1);
    const fp H = fp_sub(U2, U1);
    fp rr = fp_sub(S2, S1);
    if (fp_is_zero(H)) {
        if (fp_is_zero(rr)) return g1j_dbl(p);
        return {fp_one(), fp_one(), fp_zero()};
    }
    fp I = fp_add_nr(H, H);
    I = fp_sqr_ool(I);
    const fp J = fp_mul_ool(H, I);
    rr = fp_add_nr(rr, rr);
    const fp V = fp_mul_ool(U1, I);
    g1j r;
    r.X = fp_sub(fp_sub(fp_sqr_ool(rr), J), fp_add(V, V));
    const fp SJ = fp_mul_ool(S1, J);
    r.Y = fp_sub(fp_mul_ool(rr, fp_sub(V, r.X)), fp_add(SJ, SJ));
    r.Z = fp_mul_ool(fp_sub(fp_sub(fp_sqr_ool(fp_add_nr(p.Z, q.Z)), Z1Z1), Z2Z2), H);
    return r;
}

// phi(P) == -[x^2] P for an affine curve point P (not the identity)
static __device__ __noinline__ bool g1_in_subgroup(const fp& x, const fp& y) {
    // x^2 = 0xac45a4010001a402_0000000100000000 (128 bits, 17 set)
    const uint64_t k[2] = {0x0000000100000000ULL, 0xac45a4010001a402ULL};
    g1j acc = {x, y, fp_one()};
    for (int i = 126; i >= 0; --i) {
        acc = g1j_dbl(acc);
        if ((k[i >> 6] >> (i & 63)) & 1) acc = g1j_add_affine(acc, x, y);
    }
    if (fp_is_zero(acc.Z)) return false;
    // beta, Montgomery form
    const uint64_t bv[6] = {0x30f1361b798a64e8ULL, 0xf3b8ddab7ece5a2aULL, 0x16a8ca3ac61577f7ULL,
                            0xc26a2ff874fd029bULL, 0x3636b76660701c6eULL, 0x051ba4ab241b6160ULL};
    fp beta = fp_load_u64(bv);
    fp Z2 = fp_sqr(acc.Z), Z3 = fp_mul(Z2, acc.Z);
    // X/Z^2 == beta x  and  Y/Z^3 == -y
    bool ex = fp_eq(acc.X, fp_mul(fp_mul(beta, x), Z2));
    bool ey = fp_eq(fp_add(acc.Y, fp_mul(y, Z3)), fp_zero());
    return ex && ey;
}

// ---------------------------------------------------------------------------
// Four lanes to a point, for batches too small to fill the chip with a lane each:
// the squares of one level of a doubling (and the products of one level of an
// addition) run side by side, one to a lane, and are handed round by shuffles, so
// a doubling takes two squares and a product one after another where a lane alone
// takes five squares and two products.  Every lane of the quad holds the point.
// All 32 lanes of a warp call these together.
// ---------------------------------------------------------------------------
__device__ __forceinline__ fp quad_get(const fp& v, int l) {
    fp r;
#pragma unroll
    for (int i = 0; i < 12; ++i) r.w[i] = __shfl_sync(0xffffffffu, v.w[i], l, 4);
    return r;
}
__device__ __forceinline__ fp fp_sel(bool c, const fp& a, const fp& b) {
    fp r;
#pragma unroll
    for (int i = 0; i < 12; ++i) r.w[i] = c ? a.w[i] : b.w[i];
    return r;
}

// dbl-2009-l, with Z3 = (Y + Z)^2 - Y^2 - Z^2 to make its first level four squares
// and (2B)^2 beside B^2 in the second; sums that are squared or multiplied next
// are left unreduced (fp_sqr takes values below 3p).
__device__ __forceinline__ g1j quad_dbl(const g1j& p) {
    const int l = threadIdx.x & 3;
    fp s = fp_sqr(fp_sel(l < 2, fp_sel(l == 0, p.X, p.Y), fp_sel(l == 2, fp_add_nr(p.Y, p.Z), p.Z)));
    const fp A = quad_get(s, 0), B = quad_get(s, 1);
    g1j r;
    r.Z = fp_sub(fp_sub(quad_get(s, 2), B), quad_get(s, 3));
    const fp E = fp_add_nr(fp_add_nr(A, A), A);
    s = fp_sqr(fp_sel(l < 2, fp_sel(l == 0, E, B), fp_add_nr(fp_sel(l == 2, p.X, B), B)));
    const fp F = quad_get(s, 0);
    fp D = fp_sub(fp_sub(quad_get(s, 2), A), quad_get(s, 1));   // 2 X B
    D = fp_add(D, D);
    r.X = fp_sub(fp_sub(F, D), D);
    const fp C4 = quad_get(s, 3);
    r.Y = fp_sub(fp_mul(E, fp_sub(D, r.X)), fp_add(C4, C4));
    return r;
}

// p + (qx, qy), q affine (madd-2007-bl with Z3 = 2 Z1 H).  *bad is set, and the
// result of no use, when p is the identity or +-q; the caller then takes the
// one-lane path.
static __device__ __noinline__ g1j quad_add_affine(const g1j& p, const fp& qx, const fp& qy, bool* bad) {
    const int l = threadIdx.x & 3;
    fp s = fp_mul_ool(fp_sel(l == 0, p.Z, qy), p.Z);                                        // Z^2, qy Z
    const fp ZZ = quad_get(s, 0);
    s = fp_mul_ool(fp_sel(l == 0, qx, quad_get(s, 1)), ZZ);                                 // U2, S2
    const fp H = fp_sub(quad_get(s, 0), p.X);
    fp rr = fp_sub(quad_get(s, 1), p.Y);
    rr = fp_add(rr, rr);
    if (fp_is_zero(p.Z) || fp_is_zero(H)) *bad = true;
    s = fp_mul_ool(fp_sel(l == 1, rr, H), fp_sel(l == 0, H, fp_sel(l == 1, rr, p.Z)));      // H^2, rr^2, H Z
    fp I = quad_get(s, 0);
    I = fp_add(I, I);
    I = fp_add(I, I);
    g1j r;
    r.Z = quad_get(s, 2);
    r.Z = fp_add(r.Z, r.Z);
    const fp rr2 = quad_get(s, 1);
    s = fp_mul_ool(fp_sel(l == 0, H, p.X), I);                                              // J, V
    const fp J = quad_get(s, 0), V = quad_get(s, 1);
    r.X = fp_sub(fp_sub(rr2, J), fp_add(V, V));
    s = fp_mul_ool(fp_sel(l == 0, rr, p.Y), fp_sel(l == 0, fp_sub(V, r.X), J));             // rr (V - X3), Y J
    const fp YJ = quad_get(s, 1);
    r.Y = fp_sub(quad_get(s, 0), fp_add(YJ, YJ));
    return r;
}

// p + q, both Jacobian (add-2007-bl with Z3 = 2 Z1 Z2 H); *bad as for quad_add_affine
static __device__ __noinline__ g1j quad_add(const g1j& p, const g1j& q, bool* bad) {
    const int l = threadIdx.x & 3;
    const bool odd = l & 1, high = l >> 1;
    // Z1^2, Z2^2, Y1 Z2, Y2 Z1
    fp s = fp_mul_ool(fp_sel(high, fp_sel(odd, q.Y, p.Y), fp_sel(odd, q.Z, p.Z)), fp_sel(l == 0 || l == 3, p.Z, q.Z));
    const fp ZZ1 = quad_get(s, 0), ZZ2 = quad_get(s, 1), YZ1 = quad_get(s, 2), YZ2 = quad_get(s, 3);
    // U1, U2, S1, S2
    s = fp_mul_ool(fp_sel(high, fp_sel(odd, YZ2, YZ1), fp_sel(odd, q.X, p.X)), fp_sel(odd, ZZ1, ZZ2));
    const fp U1 = quad_get(s, 0), S1 = quad_get(s, 2);
    const fp H = fp_sub(quad_get(s, 1), U1);
    fp rr = fp_sub(quad_get(s, 3), S1);
    rr = fp_add(rr, rr);
    if (fp_is_zero(p.Z) || fp_is_zero(q.Z) || fp_is_zero(H)) *bad = true;
    // (2H)^2, rr^2, Z1 Z2
    fp I = fp_add(H, H);
    s = fp_mul_ool(fp_sel(high, p.Z, fp_sel(odd, rr, I)), fp_sel(high, q.Z, fp_sel(odd, rr, I)));
    I = quad_get(s, 0);
    const fp rr2 = quad_get(s, 1), zz = quad_get(s, 2);
    // J = H I, V = U1 I, Z1 Z2 H
    s = fp_mul_ool(fp_sel(high, zz, fp_sel(odd, U1, H)), fp_sel(high, H, I));
    const fp J = quad_get(s, 0), V = quad_get(s, 1);
    g1j r;
    r.Z = quad_get(s, 2);
    r.Z = fp_add(r.Z, r.Z);
    r.X = fp_sub(fp_sub(rr2, J), fp_add(V, V));
    // rr (V - X3), S1 J
    s = fp_mul_ool(fp_sel(odd, S1, rr), fp_sel(odd, J, fp_sub(V, r.X)));
    const fp SJ = quad_get(s, 1);
    r.Y = fp_sub(quad_get(s, 0), fp_add(SJ, SJ));
    return r;
}

// g1_in_subgroup with four lanes to the point
static __device__ __noinline__ bool quad_in_subgroup(const fp& x, const fp& y) {
    const uint64_t k[2] = {0x0000000100000000ULL, 0xac45a4010001a402ULL};
    g1j acc = {x, y, fp_one()};
    bool bad = false;
#pragma unroll 1
    for (int i = 126; i >= 0; --i) {
        acc = quad_dbl(acc);
        if ((k[i >> 6] >> (i & 63)) & 1) acc = quad_add_affine(acc, x, y, &bad);
    }
    const uint64_t bv[6] = {0x30f1361b798a64e8ULL, 0xf3b8ddab7ece5a2aULL, 0x16a8ca3ac61577f7ULL,
                            0xc26a2ff874fd029bULL, 0x3636b76660701c6eULL, 0x051ba4ab241b6160ULL};
    const int l = threadIdx.x & 3;
    fp s = fp_mul_ool(fp_sel(l == 0, acc.Z, fp_load_u64(bv)), fp_sel(l == 0, acc.Z, x));    // Z^2, beta x
    const fp Z2 = quad_get(s, 0);
    s = fp_mul_ool(Z2, fp_sel(l == 0, acc.Z, quad_get(s, 1)));                              // Z^3, beta x Z^2
    const fp Z3 = quad_get(s, 0), bx = quad_get(s, 1);
    const bool ok = fp_eq(acc.X, bx) && fp_is_zero(fp_add(acc.Y, fp_mul_ool(y, Z3)));
    // a point of small order met an exceptional addition: one lane, all cases handled.
    // x = 0, the identity's encoding among them, is a point of order 3, outside without
    // that second chain of 1 ms.
    return bad ? (!fp_is_zero(x) && g1_in_subgroup(x, y)) : (ok && !fp_is_zero(acc.Z));
}

// x of a 48-byte encoding as an integer, the flag bits off
__device__ __forceinline__ fp g1_raw_x(const uint8_t* in) {
    fp raw;
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        // limb i (little-endian) = big-endian bytes [44 - 4i, 48 - 4i)
        const uint8_t* b = in + 44 - 4 * i;
        uint32_t b0 = b[0];
        if (i == 11) b0 &= 0x1f;
        raw.w[i] = (b0 << 24) | ((uint32_t)b[1] << 16) | ((uint32_t)b[2] << 8) | b[3];
    }
    return raw;
}

// Decode one 48-byte point.  On success writes Montgomery (x, y) and sets
// *identity for the point at infinity (x = 0, y = R mod p, the ic_bls12_381
// identity limbs).  Returns a status code.
__device__ __forceinline__ int32_t g1_decode(const uint8_t* in, fp& x, fp& y, bool& identity,
                                             bool check_subgroup) {
    identity = false;
    x = fp_zero();
    y = fp_zero();
    uint32_t top = in[0];
    bool comp = (top >> 7) & 1, inf = (top >> 6) & 1, sort = (top >> 5) & 1;
    const fp raw = g1_raw_x(in);
    if (!comp) return ST_BAD_FLAGS;
    if (inf) {
        if (sort || !fp_is_zero(raw)) return ST_BAD_FLAGS;
        identity = true;
        y = fp_one();
        return ST_OK;
    }
    if (fp_raw_geq_p(raw)) return ST_X_NOT_CANONICAL;
    fp xm = fp_to_mont(raw);
    fp y2 = fp_add(fp_mul(fp_sqr(xm), xm), fp_four());
    fp yy = fp_sqrt_candidate(y2);
    if (!fp_eq(fp_sqr(yy), y2)) return ST_NOT_ON_CURVE;
    if (fp_lex_largest(yy) != sort) yy = fp_neg(yy);
    if (check_subgroup && !g1_in_subgroup(xm, yy)) return ST_NOT_IN_SUBGROUP;
    x = xm;
    y = yy;
    return ST_OK;
}

// the raw-ABI identity convention: x = 0 and y in {0, R mod p}
__device__ __forceinline__ bool g1_limbs_identity(const fp& x, const fp& y) {
    return fp_is_zero(x) && (fp_is_zero(y) || fp_eq(y, fp_one()));
}

// point i, decoded by one thread with every check
__device__ __forceinline__ void g1_decode_store(const uint8_t* in, int i, uint64_t* xy, int32_t* status) {
    fp x, y;
    bool id;
    const int32_t st = g1_decode(in + 48 * (size_t)i, x, y, id, true);
    status[i] = st;
    fp_store_u64(xy + 12 * (size_t)i, x);
    fp_store_u64(xy + 12 * (size_t)i + 6, y);
}

// Points base .. base + 15 of n by a block of three warps; inside: 16 bytes of
// shared memory.  Warp 0 takes the square roots, a lane to a point; warps 1 and
// 2 run the subgroup test, four lanes to a point (quad_in_subgroup), at the same
// time.  The test does not need the root: with d = x^3 + 4 the point (d x, d^2)
// lies on y^2 = x^3 + 4 d^3, and when d = y^2 the map (x, y) -> (y^2 x, y^3 y) takes the
// curve to that one, (x, +-y) to (d x, d^2), and commutes with (x, y) -> (beta x, y),
// while the doubling and addition formulas do not use the constant term.  When d
// is not a square the point is off the curve and the test's answer is dropped.
constexpr int kQuadPoints = 16, kQuadThreads = 96;
__device__ __forceinline__ void g1_decode_quad(int base, const uint8_t* in, int n, uint64_t* xy, int32_t* status,
                                               uint8_t* inside) {
    const int t = threadIdx.x;
    fp x, y;
    bool id = false;
    int32_t st = ST_OK;
    const bool have = t < kQuadPoints && base + t < n;
    if (t < 32) {
        if (have) st = g1_decode(in + 48 * (size_t)(base + t), x, y, id, false);
    } else {
        const int j = (t - 32) >> 2;
        // past the end: the last point again, so that the warp stays together
        const int i = base + j < n ? base + j : n - 1;
        const fp xm = fp_to_mont(g1_raw_x(in + 48 * (size_t)i));
        const fp d = fp_add(fp_mul_ool(fp_sqr_ool(xm), xm), fp_four());
        const bool ok = quad_in_subgroup(fp_mul_ool(d, xm), fp_sqr_ool(d));
        if ((t & 3) == 0) inside[j] = ok ? 1 : 0;
    }
    __syncthreads();
    if (!have) return;
    if (st == ST_OK && !id && !inside[t]) {
        st = ST_NOT_IN_SUBGROUP;
        x = y = fp_zero();
    }
    status[base + t] = st;
    fp_store_u64(xy + 12 * (size_t)(base + t), x);
    fp_store_u64(xy + 12 * (size_t)(base + t) + 6, y);
}

}  // namespace bls
