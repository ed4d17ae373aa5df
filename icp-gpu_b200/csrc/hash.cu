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

// xch: the odd threads' mapped points (Jacobian X, Y, Z)
__device__ __forceinline__ void neg_hash_block(int base, const uint8_t* msgs, const uint32_t* offsets, int n,
                                               const uint8_t* dst, int dst_len, uint64_t* out, uint4 (*xch)[9]) {
    const int t = 2 * base + threadIdx.x;
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

__global__ void __launch_bounds__(kHashThreads) k_neg_hash_to_g1(const uint8_t* msgs, const uint32_t* offsets,
                                                                 int n, const uint8_t* dst, int dst_len,
                                                                 uint64_t* out) {
    __shared__ uint4 xch[kHashThreads / 2][9];
    neg_hash_block(blockIdx.x * (kHashThreads / 2), msgs, offsets, n, dst, dst_len, out, xch);
}

// The hashes of n messages and the decoded points of as many signatures in one
// launch: blocks 0 .. hash_blocks - 1 hash, the others decode, a thread a point.  Two
// latency chains of which neither reads what the other writes, on three warps an SM
// for 4,736 of each.
__global__ void __launch_bounds__(kHashThreads) k_neg_hash_decode_wide(const uint8_t* msgs, const uint32_t* offsets,
                                                                      int n, const uint8_t* dst, int dst_len,
                                                                      uint64_t* out, int hash_blocks,
                                                                      const uint8_t* sigs, uint64_t* xy,
                                                                      int32_t* status) {
    __shared__ uint4 xch[kHashThreads / 2][9];
    const int b = blockIdx.x;
    if (b < hash_blocks) {
        neg_hash_block(b * (kHashThreads / 2), msgs, offsets, n, dst, dst_len, out, xch);
        return;
    }
    const int i = (b - hash_blocks) * kHashThreads + threadIdx.x;
    if (i < n) g1_decode_store(sigs, i, xy, status);
}

// The hash for batches too small to fill the chip: eight lanes to a message, a
// quad of four to each of its two field elements.  The quad's lanes map the element
// together (the power is a chain that all four repeat), evaluate one polynomial of
// the isogeny each, and the two quads exchange their points and clear the cofactor
// with the products of a level side by side (quad_add, quad_dbl).
// Bound by one dependent chain, half of it the map's power of 379 squarings, most of the
// rest the sum and the cofactor's 63 doublings.
__device__ __forceinline__ void neg_hash_quad(int t, const uint8_t* msgs, const uint32_t* offsets, int n,
                                              const uint8_t* dst, int dst_len, uint64_t* out) {
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

constexpr int kHashQuadThreads = 32;
__global__ void __launch_bounds__(kHashQuadThreads) k_neg_hash_to_g1_quad(const uint8_t* msgs, const uint32_t* offsets,
                                                                         int n, const uint8_t* dst, int dst_len,
                                                                         uint64_t* out) {
    neg_hash_quad(blockIdx.x * blockDim.x + threadIdx.x, msgs, offsets, n, dst, dst_len, out);
}

// The hashes and the decoded points of k_neg_hash_decode_wide in the small-batch forms:
// hash blocks of three warps, four messages each, and g1_decode_quad's.
__global__ void __launch_bounds__(kQuadThreads) k_neg_hash_decode(const uint8_t* msgs, const uint32_t* offsets, int n,
                                                                 const uint8_t* dst, int dst_len, uint64_t* out,
                                                                 int hash_blocks, const uint8_t* sigs, uint64_t* xy,
                                                                 int32_t* status) {
    __shared__ uint8_t inside[kQuadPoints];
    const int b = blockIdx.x;
    if (b >= hash_blocks)
        g1_decode_quad((b - hash_blocks) * kQuadPoints, sigs, n, xy, status, inside);
    else if (b * (kQuadThreads / 8) + (int)(threadIdx.x >> 5) * 4 < n)     // the warp has a message
        neg_hash_quad(b * kQuadThreads + threadIdx.x, msgs, offsets, n, dst, dst_len, out);
}

// bls_neg_hash_to_g1 from host buffers, eight lanes against two: 1 message 0.84 and
// 1.34 ms, 1,000 messages 0.87 and 1.37 ms, 2,368 (a warp on every scheduler) 0.88 and
// 1.37 ms, 4,736 (two) 1.21 and 1.40 ms; 7,104 messages 1.87 against 1.42 ms.
constexpr int kHashQuadMax = 4736;    // 32 an SM

cudaError_t launch_neg_hash_to_g1(const uint8_t* msgs, const uint32_t* offsets, int n, const uint8_t* dst,
                                  int dst_len, uint64_t* out, int sms, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (small_batch(n, kHashQuadMax, sms)) {
        k_neg_hash_to_g1_quad<<<(unsigned)((8LL * n + kHashQuadThreads - 1) / kHashQuadThreads), kHashQuadThreads, 0, s>>>(
            msgs, offsets, n, dst, dst_len, out);
        return cudaGetLastError();
    }
    const long long threads = 2LL * n;
    k_neg_hash_to_g1<<<(unsigned)((threads + kHashThreads - 1) / kHashThreads), kHashThreads, 0, s>>>(
        msgs, offsets, n, dst, dst_len, out);
    return cudaGetLastError();
}

// bls_verify_messages of compressed signatures from host buffers: the small-batch forms
// in two launches, in one, and the thread-a-point forms in one.  1,000 items 3.94, 3.40
// and 4.07 ms; 2,000 items 4.17, 3.95, 4.29 ms; 2,368 items, where the hash alone has a
// warp on every scheduler, 4.18, 4.26, 4.29 ms; 3,000 items 5.37, 5.12, 5.01 ms; 4,736
// items 5.44, 6.03, 5.04 ms (the eight- and four-lane forms repeat work, and side by side
// that fills the chip).  Two launches of the thread-a-point forms, for more items than
// the small-batch forms take: 14,208 items 13.69, in one 13.30 ms; 40,000 37.9 and 37.2 ms.
constexpr int kHashDecodeQuadMax = 2072;    // 14 of each an SM
constexpr int kHashDecodeTwoMax = 2368;     // 16

cudaError_t launch_neg_hash_decode(const uint8_t* msgs, const uint32_t* offsets, int n, const uint8_t* dst,
                                   int dst_len, uint64_t* out, const uint8_t* sigs, uint64_t* xy, int32_t* status,
                                   int sms, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (small_batch(n, kHashDecodeQuadMax, sms)) {
        const int hash_blocks = (8 * n + kQuadThreads - 1) / kQuadThreads;
        k_neg_hash_decode<<<hash_blocks + (n + kQuadPoints - 1) / kQuadPoints, kQuadThreads, 0, s>>>(
            msgs, offsets, n, dst, dst_len, out, hash_blocks, sigs, xy, status);
        return cudaGetLastError();
    }
    if (small_batch(n, kHashDecodeTwoMax, sms)) {
        const cudaError_t e = launch_neg_hash_to_g1(msgs, offsets, n, dst, dst_len, out, sms, s);
        return e != cudaSuccess ? e : launch_g1_decompress(sigs, n, xy, status, sms, s);
    }
    const int hash_blocks = (n + kHashThreads / 2 - 1) / (kHashThreads / 2);
    k_neg_hash_decode_wide<<<hash_blocks + (n + kHashThreads - 1) / kHashThreads, kHashThreads, 0, s>>>(
        msgs, offsets, n, dst, dst_len, out, hash_blocks, sigs, xy, status);
    return cudaGetLastError();
}

}  // namespace bls
