// k_neg_hash_to_g1: -H(m) for a batch of messages (h2c.cuh), two threads per
// message: both expand the message (SHA-256 is cheap next to the field work),
// thread 2i maps u0 and thread 2i + 1 maps u1 at the same time (SSWU to E',
// then the isogeny to E), then thread 2i adds the two points, clears the
// cofactor and writes the result.  The output
// is the verify kernels' neg_hms layout, so a verify from message bytes hashes
// straight into the verify launch's input buffer.
#include <cuda_runtime.h>

#include "h2c.cuh"
#include "internal.h"

namespace bls {

constexpr int kHashThreads = 64;

__global__ void __launch_bounds__(kHashThreads) k_neg_hash_to_g1(const uint8_t* msgs, const uint32_t* offsets,
                                                                 int n, const uint8_t* dst, int dst_len,
                                                                 uint64_t* out) {
    __shared__ uint4 xch[kHashThreads / 2][9];   // the odd thread's mapped point (Jacobian X, Y, Z)
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = t >> 1, which = t & 1;
    const bool live = i < n;
    g1j pt;
    if (live) {
        const uint32_t a = offsets[i], b = offsets[i + 1];
        uint32_t ub[32];
        h2c::expand_xmd_128(msgs + a, b - a, dst, (uint32_t)dst_len, ub);
        fp xn, xd, ys;
        h2c::map_sswu(h2c::field_from_be64(ub + 16 * which), xn, xd, ys);
        pt = h2c::iso_map(xn, xd, ys);
        if (which) {
            uint4* d = xch[threadIdx.x >> 1];
            const fp* c[3] = {&pt.X, &pt.Y, &pt.Z};
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    d[3 * k + j] = make_uint4(c[k]->w[4 * j], c[k]->w[4 * j + 1], c[k]->w[4 * j + 2], c[k]->w[4 * j + 3]);
        }
    }
    __syncthreads();
    // the even thread of a live message adds the points, clears the cofactor
    // and inverts the result's Z
    if (!live || which) return;
    g1j r;
    {
        const uint4* d = xch[threadIdx.x >> 1];
        g1j p1;
        fp* c[3] = {&p1.X, &p1.Y, &p1.Z};
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const uint4 q = d[3 * k + j];
                c[k]->w[4 * j] = q.x; c[k]->w[4 * j + 1] = q.y; c[k]->w[4 * j + 2] = q.z; c[k]->w[4 * j + 3] = q.w;
            }
        r = h2c::clear_sum(pt, p1);
    }
    const fp zi = fp_inverse_mont(r.Z, h2c::kR3);
    fp ox, oy;
    h2c::neg_affine(r, zi, ox, oy);
    fp_store_u64(out + 12 * (size_t)i, ox);
    fp_store_u64(out + 12 * (size_t)i + 6, oy);
}

// The same for batches too small to fill the chip: eight lanes to a message, a
// quad of four to each of its two field elements.  The quad's lanes map the element
// together (the power is a chain that all four repeat), evaluate one polynomial of
// the isogeny each, and the two quads exchange their points and clear the cofactor
// with the products of a level side by side (quad_add, quad_dbl).
// Bound by one dependent chain, for a 32-byte message in cycles: expansion 101 k,
// the map with its power of 379 squarings 818 k, isogeny 108 k, sum and cofactor
// 479 k, inverse 78 k.
constexpr int kHashQuadThreads = 32;

__global__ void __launch_bounds__(kHashQuadThreads) k_neg_hash_to_g1_quad(const uint8_t* msgs, const uint32_t* offsets,
                                                                         int n, const uint8_t* dst, int dst_len,
                                                                         uint64_t* out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int which = (t >> 2) & 1;
    const int i = t >> 3, m = i < n ? i : n - 1;     // past the end: the last message again, the warp stays together
    const uint32_t a = offsets[m], b = offsets[m + 1];
    uint32_t ub[32];
    h2c::expand_xmd_128(msgs + a, b - a, dst, (uint32_t)dst_len, ub);
    __syncwarp();
    fp xn, xd, ys;
    h2c::map_sswu(h2c::field_from_be64(ub + 16 * which), xn, xd, ys);
    __syncwarp();
    const g1j pt = h2c::quad_iso_map(xn, xd, ys);
    g1j other;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        other.X.w[k] = __shfl_xor_sync(0xffffffffu, pt.X.w[k], 4);
        other.Y.w[k] = __shfl_xor_sync(0xffffffffu, pt.Y.w[k], 4);
        other.Z.w[k] = __shfl_xor_sync(0xffffffffu, pt.Z.w[k], 4);
    }
    bool bad = false;
    g1j r = h2c::quad_clear_sum(pt, other, &bad);
    if (bad) r = h2c::clear_sum(pt, other);          // all cases, each lane for itself
    const fp zi = fp_inverse_mont(r.Z, h2c::kR3);
    if (i >= n || (t & 7)) return;
    fp ox, oy;
    h2c::neg_affine(r, zi, ox, oy);
    fp_store_u64(out + 12 * (size_t)i, ox);
    fp_store_u64(out + 12 * (size_t)i + 6, oy);
}

// bls_neg_hash_to_g1 from host buffers, eight lanes against two: 1 message 0.84 and
// 1.34 ms, 1,000 messages 0.87 and 1.37 ms, 2,368 (a warp on every scheduler) 0.88 and
// 1.37 ms, 4,736 (two) 1.21 and 1.40 ms; 7,104 messages 1.87 against 1.42 ms.
constexpr int kHashQuadMax = 4736;

cudaError_t launch_neg_hash_to_g1(const uint8_t* msgs, const uint32_t* offsets, int n, const uint8_t* dst,
                                  int dst_len, uint64_t* out, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (n <= kHashQuadMax) {
        k_neg_hash_to_g1_quad<<<(unsigned)((8LL * n + kHashQuadThreads - 1) / kHashQuadThreads), kHashQuadThreads, 0, s>>>(
            msgs, offsets, n, dst, dst_len, out);
        return cudaGetLastError();
    }
    const long long threads = 2LL * n;
    k_neg_hash_to_g1<<<(unsigned)((threads + kHashThreads - 1) / kHashThreads), kHashThreads, 0, s>>>(
        msgs, offsets, n, dst, dst_len, out);
    return cudaGetLastError();
}

}  // namespace bls
