// Warp-uniform Fp2-lane verify kernel.  The tower programs of gen_fp2ops.py in
// their paired-warp form (fp2ops.inc): a block of twelve warps verifies 32 items,
// one per lane.  The two warps of coefficient k (k = w % 6, w the warp) each
// produce one component of the k-th Fp2 coefficient of every Fp12 result (half
// h = w / 6: real, imaginary).  Every lane of a warp runs the same descriptor:
// descriptor reads are constant-memory broadcasts, control flow never diverges,
// and the only per-lane difference is which item's slots a lane reads and writes.
//
// Per verification (gpu-crypto/cuda/api.cu:80-91, api.cu:30-52, api.cu:65-78):
// the Miller loop over both pairs with the lines of the generator's and the
// key's tables, the reference's final-exponentiation chain, the canonical Gt
// compared with one; optional Miller / Gt outputs.
//
// What bounds it: instruction throughput of three warps a scheduler.  Warps of
// paired multiply-adds and warps of carry adds, run beside one another, slow each
// other as if a paired multiply-add took 3.7 and an add 1.5 cycles of one shared
// resource, and the kernel's time is its instructions at those rates (a product of
// 108 pairs and about 150 adds: 657 cycles a warp and scheduler).  So every add
// counts.  Against the form in which the two warps of a coefficient each added
// every product into two accumulators (verify_fp2.cu's): one accumulator, no bias
// to preload, one range reduction per component instead of two: 3.92 -> 3.60 ms
// per 4,096 verifications (3.42 with what came after it).  Also measured, and
// slower: one warp a component with no partial sums and a third more products,
// accumulated in place; eighteen warps, three to a coefficient, at the 96 registers
// that leaves; operands of the next product loaded ahead.
//
// Shared memory (16-byte units): the items' Fp2 slots interleaved by item
// (unit ((s * 2 + c) * 3 + q) * 32 + v holds words 4q..4q+3 of component c of
// slot s of item v, so a warp's load of one component is three conflict-free
// 512-byte rows), then the block-shared constant slots, the partial sums that
// the warps of a coefficient hand each other (25 words, same interleaving), the
// per-item flags and the tables of k p (the components' bias multiples) and of
// the reduction.
#include <cuda_runtime.h>

#include "fp2ops.cuh"
#include "g1.cuh"
#include "internal.h"

namespace bls {
namespace {

constexpr int kV = kBlockItems;                  // items a block holds at most, one per lane
constexpr int kRoles = 12;                       // warps per block
constexpr int kThreads = 32 * kRoles;
constexpr int kGroups = f2::kGroupsUsed;
constexpr int kKSlots = f2::kKSlotCount;         // block-shared constant slots (absolute 0 .. kKSlots - 1)
constexpr int kCOff = 6 * kGroups;               // C area after the groups
constexpr int kItemSlots = kCOff + 12;           // Fp2 slots per item
constexpr int kSlotU4 = kItemSlots * 6 * kV;     // 16-byte units of the item slots
constexpr int kKU4 = kKSlots * 6;                // constant slots, not interleaved
constexpr int kXchU4 = 6 * 2 * 7 * kV;           // partial sums: 25 words (7 units) per coefficient, half, item
constexpr int kXchAntiU4 = 3 * 7 * kV;           // and the square's subtracted sums, of three coefficients
static_assert((kXchU4 + kXchAntiU4) / (7 * kV) == f2::kPartSlots, "a slot of 7 units per partial sum and item");
constexpr int kKpCount = f2::kMaxBias + 1;       // k p, 16 words each
constexpr int kInfoWords = 4 * kV;               // per item: key index, flags, status, result flags
constexpr int kFlagBytes = 16 * kV;              // per item and role: "not the expected value" bytes
constexpr int kQpU4 = 128 * 4;                   // the QP table (128 entries of 16 words)
constexpr size_t kSmemBytes = (size_t)(kSlotU4 + kKU4 + kXchU4 + kXchAntiU4 + kQpU4) * 16 + (size_t)kKpCount * 64 +
                              (size_t)kInfoWords * 4 + kFlagBytes + 16;
static_assert(kKSlots + kItemSlots <= 256, "slot indices must fit a byte");
static_assert(kKpCount <= kThreads, "one thread per table entry at start-up");
static_assert(kSmemBytes <= 227 * 1024, "one block per SM");

struct Sm {
    uint4* slots;      // item slots
    uint4* kslots;     // constant slots
    uint4* xch;        // partial sums
    uint4* qp;         // QP table (qp_reduce_tab)
    uint32_t* kp;      // k p table
    uint32_t* info;    // per item: [0] key index, [1] skip bits, [2] status, [3] spare
    uint8_t* flags;    // per item, 16 bytes: role r's "not expected" byte at r
    uint32_t* bcast;   // claim broadcast (4 words)
    int v;             // this lane's item
};

// D, A, B, C, K, T: absolute slot of index 0, one byte each
struct Bases { uint64_t b; };

__device__ __forceinline__ uint32_t slot_addr(const Bases& bs, uint32_t ref) {
    return (uint32_t)(bs.b >> (8u * (ref >> 4))) % 256u + (ref & 15u);
}

// the three 16-byte units of component `comp` of absolute slot `slot` for this lane
__device__ __forceinline__ const uint4* unit_ptr(const Sm& s, uint32_t slot, int comp) {
    if (slot < (uint32_t)kKSlots) return s.kslots + (slot * 2 + comp) * 3;
    return s.slots + ((slot - kKSlots) * 2 + comp) * 3 * kV + s.v;
}
__device__ __forceinline__ uint32_t unit_stride(uint32_t slot) { return slot < (uint32_t)kKSlots ? 1u : (uint32_t)kV; }

__device__ __forceinline__ void load_fp(uint32_t* x, const Sm& s, uint32_t slot, int comp) {
    const uint4* p = unit_ptr(s, slot, comp);
    const uint32_t st = unit_stride(slot);
    const uint4 a = p[0], b = p[st], c = p[2 * st];
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    x[8] = c.x; x[9] = c.y; x[10] = c.z; x[11] = c.w;
}
// stores go to item slots only (the constant slots are written at start-up)
__device__ __forceinline__ void store_fp(const Sm& s, uint32_t slot, int comp, const uint32_t* x) {
    uint4* p = s.slots + ((slot - kKSlots) * 2 + comp) * 3 * kV + s.v;
    p[0] = make_uint4(x[0], x[1], x[2], x[3]);
    p[kV] = make_uint4(x[4], x[5], x[6], x[7]);
    p[2 * kV] = make_uint4(x[8], x[9], x[10], x[11]);
}

// t[0..12] = k p from the block's table (k <= kMaxBias for every descriptor)
__device__ __forceinline__ void load_kp(uint32_t* t, const Sm& s, uint32_t k) {
    const uint32_t* e = s.kp + 16 * k;
    const uint4* v = reinterpret_cast<const uint4*>(e);
    const uint4 a = v[0], b = v[1], c = v[2];
    t[0] = a.x; t[1] = a.y; t[2] = a.z; t[3] = a.w;
    t[4] = b.x; t[5] = b.y; t[6] = b.z; t[7] = b.w;
    t[8] = c.x; t[9] = c.y; t[10] = c.z; t[11] = c.w;
    t[12] = e[12];
}

__device__ __forceinline__ int sext4(uint32_t v) { return (int)(v << 28) >> 28; }

// An operand: the linear form `f` of a slot's two components (gen_fp2ops.py)
__device__ __forceinline__ void load_form(uint32_t* x, const Sm& s, uint32_t f, uint32_t slot) {
    const int c = f & 1u;
    if (f >= 8u && f < 12u) {                       // x0 + x1, 5p - x0 - x1, 2 (x0 + x1)
        uint32_t y[12];
        load_fp(x, s, slot, 0);
        load_fp(y, s, slot, 1);
        f2::add12(x, x, y);
        if (f == 9u) f2::sub_from_5p(x);
        if (f == 10u) f2::dbl12(x);
        return;
    }
    load_fp(x, s, slot, c);
    if (f < 2u) return;                             // x_c
    if (f >= 6u && f < 8u) {                        // x_c - x_(1-c) + 3p
        uint32_t y[12];
        load_fp(y, s, slot, 1 - c);
        f2::add3p_sub(x, x, y);
        return;
    }
    if (f >= 4u) f2::sub_from_3p(x);          // 3p - x_c
    if ((f & 4u) == 0u || f >= 12u) f2::dbl12(x);   // 2 x_c, 2 (3p - x_c)
}

// The operands U, V of the product described by w (gen_fp2ops.py: COMBOS).  The
// pairs of forms that the hot programs use have a case each, with all loads
// ahead of the arithmetic, where two calls of load_form wait for each of theirs.
__device__ __forceinline__ void load_operands(uint32_t* U, uint32_t* V, const Sm& s, uint32_t w, const Bases& bs,
                                              const uint32_t* line) {
    const uint32_t xs = slot_addr(bs, (w >> 8) & 0x7fu), ys = slot_addr(bs, (w >> 16) & 0x7fu);
    uint32_t T[12];
    switch (w & 15u) {
        case 0:     // x0 + x1, y0
            load_fp(U, s, xs, 0); load_fp(T, s, xs, 1); load_fp(V, s, ys, 0);
            f2::add12(U, U, T);
            break;
        case 1:     // 3p - x1, y0 + y1
            load_fp(U, s, xs, 1); load_fp(V, s, ys, 0); load_fp(T, s, ys, 1);
            f2::sub_from_3p(U);
            f2::add12(V, V, T);
            break;
        case 2:     // x0, y1 - y0 + 3p
            load_fp(U, s, xs, 0); load_fp(T, s, ys, 0); load_fp(V, s, ys, 1);
            f2::add3p_sub(V, V, T);
            break;
        case 3:     // 2 x0, y1
            load_fp(U, s, xs, 0); load_fp(V, s, ys, 1);
            f2::dbl12(U);
            break;
        case 4:     // x0 + x1, x0 - x1 + 3p
            load_fp(V, s, xs, 0); load_fp(T, s, xs, 1);
            f2::add12(U, V, T);
            f2::add3p_sub(V, V, T);
            break;
        case 5: {   // x0 - x1 + 3p, y0 + y1
            uint32_t S[12];
            load_fp(U, s, xs, 0); load_fp(T, s, xs, 1); load_fp(V, s, ys, 0); load_fp(S, s, ys, 1);
            f2::add3p_sub(U, U, T);
            f2::add12(V, V, S);
            break;
        }
        case 6:     // 2 x0, 3p - y1
            load_fp(U, s, xs, 0); load_fp(V, s, ys, 1);
            f2::dbl12(U);
            f2::sub_from_3p(V);
            break;
        case 7:     // 2 x1, y0
            load_fp(U, s, xs, 1); load_fp(V, s, ys, 0);
            f2::dbl12(U);
            break;
        case 8:     // x0 + x1, 2 y0
            load_fp(U, s, xs, 0); load_fp(T, s, xs, 1); load_fp(V, s, ys, 0);
            f2::add12(U, U, T);
            f2::dbl12(V);
            break;
        case 9:     // 2 (3p - x1), y0 + y1
            load_fp(U, s, xs, 1); load_fp(V, s, ys, 0); load_fp(T, s, ys, 1);
            f2::sub_from_3p(U);
            f2::dbl12(U);
            f2::add12(V, V, T);
            break;
        case 10:    // 2 x0, y1 - y0 + 3p
            load_fp(U, s, xs, 0); load_fp(T, s, ys, 0); load_fp(V, s, ys, 1);
            f2::dbl12(U);
            f2::add3p_sub(V, V, T);
            break;
        case 11: {  // x0 - x1 + 3p, 2 (y0 + y1)
            uint32_t S[12];
            load_fp(U, s, xs, 0); load_fp(T, s, xs, 1); load_fp(V, s, ys, 0); load_fp(S, s, ys, 1);
            f2::add3p_sub(U, U, T);
            f2::add12(V, V, S);
            f2::dbl12(V);
            break;
        }
        case 12:    // 2 x0, 2 (3p - y1)
            load_fp(U, s, xs, 0); load_fp(V, s, ys, 1);
            f2::dbl12(U);
            f2::sub_from_3p(V);
            f2::dbl12(V);
            break;
        case 13:    // 2 x1, 2 y0
            load_fp(U, s, xs, 1); load_fp(V, s, ys, 0);
            f2::dbl12(U);
            f2::dbl12(V);
            break;
        case 14:
            load_form(U, s, ((w >> 15) & 1u) | ((w >> 22) & 2u) | ((w >> 28) & 12u), xs);
            load_form(V, s, (w >> 4) & 15u, ys);
            break;
        default:    // the line coefficient, the point's coordinate
#pragma unroll
            for (int i = 0; i < 12; ++i) U[i] = line[i];
            load_fp(V, s, ys, (w >> 4) & 1u);
    }
}

// a partial sum (25 words) of this lane into its slot, and back
__device__ __forceinline__ uint4* part_row(const Sm& s, uint32_t slot) { return s.xch + slot * 7 * kV + s.v; }
__device__ __forceinline__ void part_store(uint4* row, const uint32_t* p, uint32_t top) {
#pragma unroll
    for (int q = 0; q < 6; ++q) row[q * kV] = make_uint4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
    reinterpret_cast<uint32_t*>(row + 6 * kV)[0] = top;
}
__device__ __forceinline__ void part_load(uint32_t* p, const uint4* row) {
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const uint4 u = row[q * kV];
        p[4 * q] = u.x; p[4 * q + 1] = u.y; p[4 * q + 2] = u.z; p[4 * q + 3] = u.w;
    }
    p[24] = reinterpret_cast<const uint32_t*>(row + 6 * kV)[0];
}

// acc (25 words) = the sum of the np > 0 products described at `prod`, partial
// sums stored on the way.  line: the key-table coefficient this warp has read,
// for the line load's products.
__device__ __forceinline__ void sum_products(uint32_t* acc, const uint32_t* prod, uint32_t np, const Sm& s,
                                             const Bases& bs, const uint32_t* line) {
#pragma unroll 1
    for (uint32_t j = 0; j < np; ++j) {
        const uint32_t w = prod[j];
        uint32_t U[12], V[12], P[24];
        load_operands(U, V, s, w, bs, line);
        f2::prod24k(P, U, V);
        if (j == 0) {
#pragma unroll
            for (int i = 0; i < 24; ++i) acc[i] = P[i];
            acc[24] = 0;
        } else {
            f2::add25(acc, P);
        }
        const uint32_t store = (w >> 24) & 3u;
        if (store == 1u) part_store(part_row(s, (w >> 26) & 15u), acc, acc[24]);
        if (store == 2u) part_store(part_row(s, (w >> 26) & 15u), P, 0u);
    }
}

// The same with kSplit lanes to an item: each lane sums its list of the products
// (gen_fp2ops.py: split_products), and the lanes' sums are added at the end, in
// every lane.
template <int kSplit>
__device__ __forceinline__ void sum_products_split(uint32_t* acc, const uint32_t* list, const Sm& s, const Bases& bs,
                                                   const uint32_t* line) {
    constexpr int kItems = kV / kSplit;
    const int sub = (threadIdx.x & 31) / kItems;
    const uint32_t steps = list[0];
#pragma unroll
    for (int i = 0; i < 25; ++i) acc[i] = 0;
#pragma unroll 1
    for (uint32_t j = 0; j < steps; ++j) {
        const uint32_t w = list[1 + kSplit * j + sub];
        if (w != f2::kNoProduct) {
            uint32_t U[12], V[12], P[24];
            load_operands(U, V, s, w, bs, line);
            f2::prod24k(P, U, V);
            f2::add25(acc, P);
            if ((w >> 24) & 3u) part_store(part_row(s, (w >> 26) & 15u), acc, acc[24]);
        }
        __syncwarp();
    }
#pragma unroll
    for (int d = kItems; d < kV; d *= 2) {
        uint32_t p[25];
#pragma unroll
        for (int i = 0; i < 25; ++i) p[i] = __shfl_xor_sync(0xffffffffu, acc[i], d);
        f2::add25_25(acc, p);
    }
}

// Warp (k, half) on program `pid` for every item of the block.  No program of
// the generated sequences writes a slot that any warp of it reads (the
// generator places a result that would overwrite an operand in an unused group,
// and refuses to emit a sequence where it cannot), so a warp stores its
// component as soon as it has it: one block-wide meeting per program, after the
// stores, and one of a coefficient's two warps when the partial sums are there.
template <int kSplit>
__device__ __forceinline__ void run(int pid, const Sm& s, int k, int half, const Bases& bs, const uint32_t* line) {
    const uint32_t off = f2::kPairIndex[pid][6 * half + k];
    const uint32_t hdr = off != 0xffffu ? f2::kPair[off] : 0u, adds = off != 0xffffu ? f2::kPair[off + 1] : 0u;
    const uint32_t np = hdr & 15u;
    uint32_t acc[25];
    if (np) {
        if constexpr (kSplit == 1)
            sum_products(acc, f2::kPair + off + 2, np, s, bs, line);
        else if constexpr (kSplit == 2)
            sum_products_split<2>(acc, f2::kSplit2 + f2::kSplit2Index[pid][6 * half + k], s, bs, line);
        else
            sum_products_split<4>(acc, f2::kSplit4 + f2::kSplit4Index[pid][6 * half + k], s, bs, line);
    }
    // a named barrier (id 1 + k) over the 64 threads of coefficient k; both
    // warps reach it on every program, whether or not they have an output
    asm volatile("bar.sync %0, 64;" ::"r"(1 + k) : "memory");
    if (off != 0xffffu) {
        const uint32_t nl = (hdr >> 4) & 3u, scale = (hdr >> 6) & 3u, bias = (hdr >> 16) & 0xffu;
        const uint32_t* lin = f2::kPair + off + 2 + np;
        uint32_t o[12];
        if ((hdr >> 24) & 1u) {                     // the one Fp inverse
            fp r = fp_zero();
            if (half == 0) {
                fp z;
                load_fp(z.w, s, slot_addr(bs, lin[0] >> 8), 0);
                r = fp_inverse_mont(z, f2::kR3);
            }
#pragma unroll
            for (int i = 0; i < 12; ++i) o[i] = r.w[i];
        } else {
            uint32_t r[13];
            if (np) {
#pragma unroll 1
                for (int i = 0; i < 2; ++i) {
                    const uint32_t a = (adds >> (8 * i)) & 31u;
                    if (a == 15u) break;
                    uint32_t p[25];
                    part_load(p, part_row(s, a & 15u));
                    if (a & 16u) f2::sub25_25(acc, p);
                    else f2::add25_25(acc, p);
                }
                f2::redc26(r, acc);
                if (scale) {                        // 3 r
                    uint32_t d[13];
#pragma unroll
                    for (int i = 0; i < 13; ++i) d[i] = r[i];
                    f2::dbl13(d);
                    f2::add13(r, d);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 13; ++i) r[i] = 0;
            }
            if (bias) {
                uint32_t b[13];
                load_kp(b, s, bias);
                f2::add13(r, b);
            }
#pragma unroll 1
            for (uint32_t j = 0; j < nl; ++j) {
                uint32_t z[12];
                load_fp(z, s, slot_addr(bs, lin[j] >> 8), half);
                const int c = sext4(lin[j]);
                if (c & 1) {
                    if (c < 0) f2::sub13_12(r, z);
                    else f2::add13_12(r, z);
                } else {
                    f2::dbl12(z);
                    if (c < 0) f2::sub13_12(r, z);
                    else f2::add13_12(r, z);
                }
            }
            if (scale == 2u) f2::dbl13(r);          // 2 (3 REDC + ..)
            f2::qp_reduce_tab(o, r, s.qp);
        }
        store_fp(s, slot_addr(bs, (hdr >> 8) & 0x7fu), half, o);
    }
}

// The meeting after the op `e`: the block's warps, or, where the generator has proved
// that they touch nothing of each other's (gen_fp2ops.py: check_meetings), only those of
// a set of coefficients, or none.
__device__ __forceinline__ void meet(uint32_t e, int k) {
    const uint32_t kind = (e >> f2::kMeetShift) & 3u;
    if (kind == f2::kMeetSets) {
        if ((f2::kMeetSet >> k) & 1u) asm volatile("bar.sync 7, %0;" ::"n"(64 * f2::kMeetSetSize) : "memory");
        else asm volatile("bar.sync 8, %0;" ::"n"(64 * (6 - f2::kMeetSetSize)) : "memory");
    } else if (kind == f2::kMeetAll) {
        __syncthreads();
    }
}

__device__ __forceinline__ uint32_t grp(int g) { return kKSlots + 6 * g; }

__device__ __forceinline__ void copy_fp_from_global(const Sm& s, uint32_t slot, int comp, const uint64_t* src) {
    const uint4* g = reinterpret_cast<const uint4*>(src);
    uint4* p = s.slots + ((slot - kKSlots) * 2 + comp) * 3 * kV + s.v;
    p[0] = __ldg(g);
    p[kV] = __ldg(g + 1);
    p[2 * kV] = __ldg(g + 2);
}

// 6 x u64 read at L2 (not L1): a serving ring rewrites its slots by copies
__device__ __forceinline__ fp fp_load_u64_cg(const uint64_t* v) {
    fp r;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const unsigned long long x = __ldcg(reinterpret_cast<const unsigned long long*>(v) + i);
        r.w[2 * i] = (uint32_t)x;
        r.w[2 * i + 1] = (uint32_t)(x >> 32);
    }
    return r;
}

// canonical form of a slot value (below 2^381 + p < 3p)
__device__ __forceinline__ fp canonical(fp v) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        uint32_t d[12];
        uint32_t br = sub_p(d, v.w);
#pragma unroll
        for (int i = 0; i < 12; ++i) v.w[i] = br ? v.w[i] : d[i];
    }
    return v;
}

// canonical group `g` -> out (72 u64 per item, NULL: not wanted) and the
// "is one" test of every item over the twelve roles
__device__ __forceinline__ bool emit_group(const Sm& s, int g, int k, int half, uint64_t* out) {
    fp v;
    load_fp(v.w, s, grp(g) + k, half);
    v = canonical(v);
    if (out) fp_store_u64(out + 12 * k + 6 * half, v);
    const bool ok = (k == 0 && half == 0) ? fp_eq(v, fp_one()) : fp_is_zero(v);
    s.flags[16 * s.v + 8 * half + k] = ok ? 0 : 1;
    __syncthreads();
    const uint4 f = reinterpret_cast<const uint4*>(s.flags)[s.v];
    __syncthreads();
    return (f.x | f.y | f.z | f.w) == 0;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t ld_acquire_gpu(const volatile uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Ring serving, thread 0 of a block: claim up to 32 published items (all in
// device memory); *count gets how many.  False when the block should leave:
// the stop flag, serve_idle_ns in which the published count did not move,
// or serve_max_ns after the launch; the loop also has an iteration cap, so
// every wait ends.  The published count is read with acquire semantics and a
// fence follows the claim, so the claimed items' loads come after the copies
// that published them.
__device__ bool serve_claim(const VerifyArgs& a, uint64_t t_launch, uint32_t* base, uint32_t* count) {
    uint64_t t_moved = globaltimer_ns();
    uint32_t seen = ld_acquire_gpu(a.serve_avail);
    for (uint32_t it = 0; it < (1u << 26); ++it) {
        const uint32_t cur = *reinterpret_cast<volatile uint32_t*>(a.serve_claimed);
        const uint32_t av = ld_acquire_gpu(a.serve_avail);
        const int32_t ready = (int32_t)(av - cur);
        if (ready > 0) {
            const uint32_t n = ready < kV ? (uint32_t)ready : (uint32_t)kV;
            if (atomicCAS(a.serve_claimed, cur, cur + n) == cur) {
                __threadfence();
                *base = cur;
                *count = n;
                return true;
            }
            continue;
        }
        const uint64_t now = globaltimer_ns();
        if (av != seen) {
            seen = av;
            t_moved = now;
        }
        if (*a.serve_stop || now - t_moved > a.serve_idle_ns || now - t_launch > a.serve_max_ns) return false;
        __nanosleep(500);
    }
    return false;
}

// kSplit lanes work on each item, 32 / kSplit items a block.  What a block does
// takes the same time whether its lanes hold 32 items or one, so a batch that
// would leave lanes empty gives them a share of the products instead.
template <int kSplit>
__global__ void __launch_bounds__(kThreads, 1) k_verify_w(VerifyArgs a, const uint32_t* __restrict__ in_status) {
    constexpr int kItems = kV / kSplit;
    extern __shared__ uint4 smem4[];
    Sm s;
    s.slots = smem4;
    s.kslots = smem4 + kSlotU4;
    s.xch = s.kslots + kKU4;
    s.qp = s.xch + kXchU4 + kXchAntiU4;
    s.kp = reinterpret_cast<uint32_t*>(s.qp + kQpU4);
    s.info = s.kp + 16 * kKpCount;
    s.flags = reinterpret_cast<uint8_t*>(s.info + kInfoWords);
    s.bcast = reinterpret_cast<uint32_t*>(s.flags + kFlagBytes);
    // from a shuffle, so that the compiler knows it to be uniform in the warp:
    // descriptor decoding and branches on uniform registers
    const int role = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const int half = role / 6, k = role % 6;
    s.v = threadIdx.x & (kItems - 1);
    const bool lead = (threadIdx.x & 31) < kItems;   // of an item's lanes, the one that writes results

    {
        uint32_t* kw = reinterpret_cast<uint32_t*>(s.kslots);
        for (int i = threadIdx.x; i < kKSlots * 24; i += blockDim.x) kw[i] = f2::kKSlots[i / 24][i % 24];
    }
    if (threadIdx.x < kKpCount) {
        uint32_t t[13];
        f2::set_kp(t, threadIdx.x);
#pragma unroll
        for (int i = 0; i < 13; ++i) s.kp[16 * threadIdx.x + i] = t[i];
    }
    {
        // unit j of entry e at 128 j + e (qp_reduce_tab)
        uint32_t* qw = reinterpret_cast<uint32_t*>(s.qp);
        for (int i = threadIdx.x; i < 128 * 16; i += blockDim.x) {
            const int e = i / 16, w = i % 16;
            qw[4 * (128 * (w / 4) + e) + w % 4] = f2::kQP2[e][w];
        }
    }
    // the flag bytes no role writes (6, 7, 14, 15 of each item) stay zero
    for (int i = threadIdx.x; i < kFlagBytes / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(s.flags)[i] = 0;
    __syncthreads();

    const int norm = a.pk_norm != nullptr ? 1 : 0;
    const uint64_t* g2_lines = norm ? a.g2_norm : a.g2;
    const bool serving = a.serve_avail != nullptr;
    const uint64_t t_launch = serving ? globaltimer_ns() : 0;
    int next = blockIdx.x * kItems;
    const int stride = gridDim.x * kItems;
    uint32_t* info = s.info + 4 * s.v;

    for (;;) {
        int base, count;
        if (serving) {
            if (threadIdx.x == 0) {
                uint32_t b = 0, n = 0;
                const bool go = serve_claim(a, t_launch, &b, &n);
                s.bcast[0] = b;
                s.bcast[1] = go ? n : 0u;
            }
            __syncthreads();
            base = (int)s.bcast[0];
            count = (int)s.bcast[1];
            __syncthreads();
            if (count == 0) break;
        } else {
            if (a.work_counter) {
                if (threadIdx.x == 0) s.bcast[0] = (uint32_t)atomicAdd(a.work_counter, kItems);
                __syncthreads();
                base = (int)s.bcast[0];
                __syncthreads();
            } else {
                base = next;
                next += stride;
            }
            if (base >= a.n) break;
            count = a.n - base < kItems ? a.n - base : kItems;
        }
        const bool have = s.v < count;
        // item = ring slot (serving) or batch index
        const uint32_t item = serving ? (uint32_t)(base + s.v) % a.serve_cap : (uint32_t)(base + s.v);

        // warp 0 reads the item's points, status and key; the others wait for its
        // per-item record
        if (role == 0) {
            uint32_t skip = 3u, pki = 0, status = 0;
            fp sx = fp_zero(), sy = fp_zero(), hx = fp_zero(), hy = fp_zero();
            if (have) {
                const uint64_t* sp = a.sig_xy ? a.sig_xy + 12 * (size_t)item : (const uint64_t*)a.sigs + 12 * (size_t)item;
                const uint64_t* hp = a.nhms + 12 * (size_t)item;
                if (in_status) status = __ldcg(in_status + item);
                sx = fp_load_u64_cg(sp);
                sy = fp_load_u64_cg(sp + 6);
                hx = fp_load_u64_cg(hp);
                hy = fp_load_u64_cg(hp + 6);
                pki = a.pk_index ? (uint32_t)__ldcg(a.pk_index + item) : item;
                if (!key_index_ok((int64_t)(int32_t)pki, a.check_keys, a.n_keys)) {   // no table read for it
                    if (status == 0) status = ST_BAD_KEY_INDEX;
                    pki = 0;
                }
                const bool s1 = status != 0 || g1_limbs_identity(sx, sy);
                const bool s2 = status != 0 || g1_limbs_identity(hx, hy) || (a.pk_identity && a.pk_identity[pki]);
                skip = (s1 ? 1u : 0u) | (s2 ? 2u : 0u);
            }
            const uint32_t C = kKSlots + kCOff;
            store_fp(s, C + 0 * 6 + 3, 0, (skip & 1u) ? fp_zero().w : sx.w);
            store_fp(s, C + 0 * 6 + 3, 1, (skip & 1u) ? fp_zero().w : sy.w);
            store_fp(s, C + 1 * 6 + 3, 0, (skip & 2u) ? fp_zero().w : hx.w);
            store_fp(s, C + 1 * 6 + 3, 1, (skip & 2u) ? fp_zero().w : hy.w);
            info[0] = pki;
            info[1] = skip;
            info[2] = status;
        }
        // f = 1
        store_fp(s, grp(0) + k, half, (k == 0 && half == 0) ? fp_one().w : fp_zero().w);
        __syncthreads();
        const uint32_t pki = info[0], skip = info[1];
        const uint64_t* pk = (norm ? a.pk_norm : a.pk_tables) + (size_t)kCoeffU64 * pki;
        const uint64_t* pk_cf = norm ? a.pk_corr + 12 * (size_t)pki : a.g2_corr;

        const int seq_len = norm ? f2::kSeqLenNorm : f2::kSeqLenRaw;
        for (int st = 0; st < seq_len; ++st) {
            const uint32_t e = f2::kSeq[norm][st];
            const uint32_t code = e & 31u;
            if ((e & f2::kCondMl) && !a.ml_out) continue;
            Bases bs;
            bs.b = (uint64_t)grp((e >> 5) & 7u) | (uint64_t)grp((e >> 8) & 7u) << 8 |
                   (uint64_t)grp((e >> 11) & 7u) << 16 | (uint64_t)(kKSlots + kCOff) << 24 |
                   (uint64_t)grp(f2::kTGroup) << 40;
            int pid = (int)code;
            uint32_t line[12];
            if (code == f2::kOpLoadLines) {
                // role (k, h): pair k / 3, coefficient k % 3, component h; a
                // skipped pair gets the line (0, 0, 1), which leaves f unchanged.
                // The roles holding c1 and c0 form their component of l2 = c1 P.x
                // and l3 = c0 P.y (the LSCALE op that follows, and is skipped).
                const int pair = k / 3, c = k % 3;
                if ((skip >> pair) & 1u) {
                    const fp v = (c == 2 && half == 0) ? fp_one() : fp_zero();
#pragma unroll
                    for (int i = 0; i < 12; ++i) line[i] = v.w[i];
                } else {
                    const uint64_t* q = pair ? pk : g2_lines;
                    const uint4* g = reinterpret_cast<const uint4*>(q + 36 * ((e >> 14) & 127u) + 12 * c + 6 * half);
                    const uint4 a0 = __ldg(g), a1 = __ldg(g + 1), a2 = __ldg(g + 2);
                    line[0] = a0.x; line[1] = a0.y; line[2] = a0.z; line[3] = a0.w;
                    line[4] = a1.x; line[5] = a1.y; line[6] = a1.z; line[7] = a1.w;
                    line[8] = a2.x; line[9] = a2.y; line[10] = a2.z; line[11] = a2.w;
                }
                if (c == 2) store_fp(s, kKSlots + kCOff + 6 * pair + 2, half, line);
                pid = f2::kNumPrograms;             // the line load's row of the descriptor index
                ++st;
            }
            if (code < (uint32_t)f2::kNumPrograms || code == f2::kOpLoadLines) {
                run<kSplit>(pid, s, k, half, bs, line);
                meet(e, k);
            } else if (code == f2::kOpLoadCorr) {
                // the generator's and the key's Miller correction factors into the c2 slots
                if (k < 2) {
                    const uint32_t slot = kKSlots + kCOff + 6 * k + 2;
                    if ((skip >> k) & 1u) store_fp(s, slot, half, half ? fp_zero().w : fp_one().w);
                    else copy_fp_from_global(s, slot, half, (k ? pk_cf : a.g2_corr) + 6 * half);
                }
                __syncthreads();
            } else if (code == f2::kOpMillerDone) {
                if (a.ml_out) emit_group(s, (e >> 5) & 7u, k, half, have && lead ? a.ml_out + 72 * (size_t)item : nullptr);
            }
        }
        const bool one = emit_group(s, (int)f2::kGtGroup[norm], k, half,
                                    (have && lead && a.gt_out) ? a.gt_out + 72 * (size_t)item : nullptr);
        if (have && lead && role == 0) {
            const int32_t status = (int32_t)info[2];
            a.results[item] = status != 0 ? -status : (one ? 1 : 0);
        }
        __syncthreads();
    }
}

cudaError_t configure() {
    static cudaError_t done = [] {
        cudaError_t e = cudaSuccess;
        for (const void* f : {(const void*)k_verify_w<1>, (const void*)k_verify_w<2>, (const void*)k_verify_w<4>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
        return e;
    }();
    return done;
}

}  // namespace

size_t verify_w_smem_bytes() { return kSmemBytes; }

int verify_w_blocks_per_sm() {
    if (configure() != cudaSuccess) return 0;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_verify_w<1>, kThreads, kSmemBytes) != cudaSuccess)
        return 0;
    return blocks;
}

// ring serving: `blocks` persistent blocks (at most one per SM)
cudaError_t launch_verify_w_serve(const VerifyArgs& a, const uint32_t* in_status, int blocks, int sms,
                                 cudaStream_t s) {
    if (!a.serve_avail || !a.serve_stop || !a.serve_claimed || a.serve_cap == 0 || blocks <= 0)
        return cudaErrorInvalidValue;
    cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    if (blocks > sms) blocks = sms;
    k_verify_w<1><<<blocks, kThreads, kSmemBytes, s>>>(a, in_status);
    return cudaGetLastError();
}

namespace {

// `a` from its item `first` on
VerifyArgs items_from(VerifyArgs a, int first) {
    const size_t i = (size_t)first;
    a.sigs = a.sig_compressed ? (const void*)((const uint8_t*)a.sigs + 48 * i) : (const void*)((const uint64_t*)a.sigs + 12 * i);
    a.nhms += 12 * i;
    if (a.pk_index) {
        a.pk_index += i;
    } else {                    // item i has table i
        a.pk_tables += kCoeffU64 * i;
        if (a.pk_norm) {
            a.pk_norm += kCoeffU64 * i;
            a.pk_corr += 12 * i;
        }
        if (a.pk_identity) a.pk_identity += i;
        a.n_keys -= first;
    }
    a.results += i;
    if (a.ml_out) a.ml_out += 72 * i;
    if (a.gt_out) a.gt_out += 72 * i;
    if (a.sig_xy) a.sig_xy += 12 * i;
    a.n -= first;
    return a;
}

}  // namespace

// As many lanes to an item as still give every item a place in one wave of the SMs that
// the launch plans with (chip_share.h): four up to 8 items a SM, two up to 16.  One
// launch alone of a block on every SM takes 3.42 ms with a lane to an item, 2.74 ms with
// two and 2.49 ms with four (the sums shrink from 2, 3, 5 and 9 products in the
// cyclotomic square, the line, the square and the product to 1, 2, 3 and 5, or 1, 1, 2
// and 3; the reductions stay).  A batch of several waves whose last one would be that
// empty runs it as a launch of its own: 4,737 items 5.91 ms, against 6.84 for two whole waves.
cudaError_t launch_verify_w(const VerifyArgs& a, const uint32_t* in_status, int sms, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    cudaError_t e = configure();
    if (e != cudaSuccess) return e;
    const int split = a.item_lanes ? a.item_lanes : verify_item_lanes(a.n, sms, sms);
    const int full = split == 1 ? a.n : a.n - a.n % (kV * sms);   // items with a lane each
    if (full > 0) {
        VerifyArgs f = a;
        f.n = full;
        const int need = (full + kV - 1) / kV;
        k_verify_w<1><<<f.work_counter && need > sms ? sms : need, kThreads, kSmemBytes, s>>>(f, in_status);
        if ((e = cudaGetLastError()) != cudaSuccess || full == a.n) return e;
    }
    VerifyArgs t = items_from(a, full);
    t.work_counter = nullptr;
    const uint32_t* st = in_status ? in_status + full : nullptr;
    const int items = kV / split, blocks = (t.n + items - 1) / items;
    if (split == 4)
        k_verify_w<4><<<blocks, kThreads, kSmemBytes, s>>>(t, st);
    else
        k_verify_w<2><<<blocks, kThreads, kSmemBytes, s>>>(t, st);
    return cudaGetLastError();
}

}  // namespace bls
