// m2_lane.cuh -- radix-4 steps and the centre square with one element of the
// transform per thread and field (m2_lane.cu, m2_cluster.cu).
#pragma once
#include "m2_split.cuh"

namespace M2K_NS {

namespace {

// sign-selecting add layers: r = partner + (neg ? -own : own)
struct Sel61 { u64 mask, add; };   // neg: ~own + (4 P61 + 1)
__device__ __forceinline__ Sel61 sel61(bool neg) { return neg ? Sel61{~0ull, K4_61 + 1} : Sel61{0ull, 0ull}; }

__device__ __forceinline__ X61 xshx(const X61& v, u32 m) {
    return X61{__shfl_xor_sync(0xffffffffu, v.a, m), __shfl_xor_sync(0xffffffffu, v.b, m)};
}
__device__ __forceinline__ X31 xshx(const X31& v, u32 m) {
    return X31{__shfl_xor_sync(0xffffffffu, v.c, m), __shfl_xor_sync(0xffffffffu, v.d, m)};
}
// one layer, not folded: operands below 4 P61, result below 8 P61
__device__ __forceinline__ X61 layer(const X61& own, u32 lane_mask, bool neg) {
    const X61 o = xshx(own, lane_mask);
    const Sel61 s = sel61(neg);
    return X61{(own.a ^ s.mask) + s.add + o.a, (own.b ^ s.mask) + s.add + o.b};
}
__device__ __forceinline__ X31 layer(const X31& own, u32 lane_mask, bool neg) {
    const X31 o = xshx(own, lane_mask);
    const u32 m = neg ? P31 : 0u;   // P31 - v is v ^ P31
    return X31{add31(own.c ^ m, o.c), add31(own.d ^ m, o.d)};
}
// the first layer of a step keeps differences below 3 P61 + 8 (offset 2 P61)
__device__ __forceinline__ X61 layer_first(const X61& own, u32 lane_mask, bool neg) {
    const X61 o = xshx(own, lane_mask);
    const u64 mask = neg ? ~0ull : 0ull, add = neg ? K2_61 + 1 : 0ull;
    return X61{(own.a ^ mask) + add + o.a, (own.b ^ mask) + add + o.b};
}
__device__ __forceinline__ X31 layer_first(const X31& own, u32 lane_mask, bool neg) { return layer(own, lane_mask, neg); }
__device__ __forceinline__ X61 folded(const X61& v) { return X61{fold61(v.a), fold61(v.b)}; }
__device__ __forceinline__ X31 folded(const X31& v) { return v; }
// times i (pos) or -i where `on`; GF(P61) operands below 3 P61 + 8
__device__ __forceinline__ X61 turn(const X61& v, bool on, bool pos) {
    const u64 n = K4_61 - (pos ? v.b : v.a);
    return on ? (pos ? X61{n, v.a} : X61{v.b, n}) : v;
}
__device__ __forceinline__ X31 turn(const X31& v, bool on, bool pos) {
    const u32 n = P31 - (pos ? v.d : v.c);
    return on ? (pos ? X31{n, v.c} : X31{v.d, n}) : v;
}

// Radix-4 steps on lane bits lb + 1, lb (m = their value): dif4 and dit4 of
// m2_field.cuh with one element per lane.
template <class X> __device__ __forceinline__ X step_fwd(X x, u32 lb, u32 m) {
    x = layer_first(x, 2u << lb, (m & 2u) != 0);        // v0, v1, v2, v3
    x = turn(x, m == 3u, true);                         // i v3
    return folded(layer(x, 1u << lb, (m & 1u) != 0));
}
template <class X> __device__ __forceinline__ X step_inv(X x, u32 lb, u32 m) {
    x = layer_first(x, 1u << lb, (m & 1u) != 0);        // x0 + x1, x0 - x1, x2 + x3, x2 - x3
    x = turn(x, m == 3u, false);                        // -i (x2 - x3)
    return folded(layer(x, 2u << lb, (m & 2u) != 0));
}

// the -1 of a field; a position's mirror (positions 0 and 1 are their own)
__device__ __forceinline__ X61 xminus(const X61&) { return X61{P61 - 1, 0}; }
__device__ __forceinline__ X31 xminus(const X31&) { return X31{P31 - 1, 0}; }
__device__ __forceinline__ u32 mirror(u32 k) { return k < 2 ? k : (3u << (31 - __clz(k))) - k - 1u; }
// the centre root of position k's pair: at its even position; 1 and -1 at 0 and 1
template <class X> __device__ __forceinline__ X centre_root(const DTw* tc, u32 k) {
    X z;
    ldtw(z, tc, ((k & 1u) ? mirror(k) : k) >> 1);
    return k == 1u ? xminus(z) : z;
}
// centre_pair (m2_field.cuh): position k's output, from its value x and its mirror's o
template <class X> __device__ __forceinline__ X centre_one(const X& x, const X& o, const X& zeta, u32 k) {
    const bool odd = (k & 1u) != 0 && k != 1u;
    const X zk = odd ? o : x, zm = odd ? x : o;
    const X u0 = xaddconj(zk, zm), u1 = xsubconj(zk, zm);
    const X v0 = xsub(xsqr(u0), xmul(xsqr(u1), zeta));
    const X v1 = xmul(u0, xadd(u1, u1));
    return odd ? xconjsub(v0, v1) : xadd(v0, v1);
}

}  // namespace

}  // namespace M2K_NS
