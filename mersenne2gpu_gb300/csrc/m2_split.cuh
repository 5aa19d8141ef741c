// m2_split.cuh -- the dual field's arithmetic one field at a time, for kernels
// that run the two halves on separate warps or in turn (m2_flow.cu, m2_tide.cu,
// m2_lane.cu, m2_cluster.cu, m2_duo.cu).
#pragma once
#include "m2_field.cuh"
#include "m2_kernels.cuh"

using namespace M2D_NS;

namespace M2K_NS {

namespace {

struct __align__(16) X61 { u64 a, b; };
struct __align__(8) X31 { u32 c, d; };

__device__ __forceinline__ X61 xmul(const X61& x, const X61& w) { X61 r; cmul61(x.a, x.b, w.a, w.b, r.a, r.b); return r; }
__device__ __forceinline__ X31 xmul(const X31& x, const X31& w) { X31 r; cmul31(x.c, x.d, w.c, w.d, r.c, r.d); return r; }
__device__ __forceinline__ X61 xmulc(const X61& x, const X61& w) { X61 r; cmulconj61(x.a, x.b, w.a, w.b, r.a, r.b); return r; }
__device__ __forceinline__ X31 xmulc(const X31& x, const X31& w) { X31 r; cmulconj31(x.c, x.d, w.c, w.d, r.c, r.d); return r; }
__device__ __forceinline__ X61 xsqr(const X61& x) { X61 r; csqr61(x.a, x.b, r.a, r.b); return r; }
__device__ __forceinline__ X31 xsqr(const X31& x) { X31 r; csqr31(x.c, x.d, r.c, r.d); return r; }
__device__ __forceinline__ X61 xadd(const X61& x, const X61& y) { return X61{add61(x.a, y.a), add61(x.b, y.b)}; }
__device__ __forceinline__ X31 xadd(const X31& x, const X31& y) { return X31{add31(x.c, y.c), add31(x.d, y.d)}; }
__device__ __forceinline__ X61 xsub(const X61& x, const X61& y) { return X61{sub61(x.a, y.a), sub61(x.b, y.b)}; }
__device__ __forceinline__ X31 xsub(const X31& x, const X31& y) { return X31{sub31(x.c, y.c), sub31(x.d, y.d)}; }
__device__ __forceinline__ X61 xaddconj(const X61& x, const X61& y) { return X61{add61(x.a, y.a), sub61(x.b, y.b)}; }
__device__ __forceinline__ X31 xaddconj(const X31& x, const X31& y) { return X31{add31(x.c, y.c), sub31(x.d, y.d)}; }
__device__ __forceinline__ X61 xsubconj(const X61& x, const X61& y) { return X61{sub61(x.a, y.a), add61(x.b, y.b)}; }
__device__ __forceinline__ X31 xsubconj(const X31& x, const X31& y) { return X31{sub31(x.c, y.c), add31(x.d, y.d)}; }
__device__ __forceinline__ X61 xconjsub(const X61& x, const X61& y) { return X61{sub61(x.a, y.a), sub61(y.b, x.b)}; }
__device__ __forceinline__ X31 xconjsub(const X31& x, const X31& y) { return X31{sub31(x.c, y.c), sub31(y.d, x.d)}; }
__device__ __forceinline__ X61 xtimes_i(const X61& r) { return X61{P61 - r.b, r.a}; }
__device__ __forceinline__ X31 xtimes_i(const X31& r) { return X31{P31 - r.d, r.c}; }
__device__ __forceinline__ X61 xone(const X61&) { return X61{1, 0}; }
__device__ __forceinline__ X31 xone(const X31&) { return X31{1, 0}; }

// the add layers of dif4 / dit4 (m2_field.cuh) in one field
__device__ __forceinline__ void dif_adds(X61 (&x)[4], const X61& u1, const X61& u2, const X61& u3) {
    const L61 v0 = ladd(x[0].a, x[0].b, u2.a, u2.b), v1 = ladd(u1.a, u1.b, u3.a, u3.b);
    const L61 v2 = lsub(x[0].a, x[0].b, u2.a, u2.b), v3 = lsub(u1.a, u1.b, u3.a, u3.b);
    x[0] = X61{fadd(v0.a, v1.a), fadd(v0.b, v1.b)};
    x[1] = X61{fsub(v0.a, v1.a), fsub(v0.b, v1.b)};
    x[2] = X61{fsub(v2.a, v3.b), fadd(v2.b, v3.a)};   // v2 + i v3
    x[3] = X61{fadd(v2.a, v3.b), fsub(v2.b, v3.a)};   // v2 - i v3
}
__device__ __forceinline__ void dif_adds(X31 (&x)[4], const X31& u1, const X31& u2, const X31& u3) {
    const X31 v0 = xadd(x[0], u2), v1 = xadd(u1, u3), v2 = xsub(x[0], u2), v3 = xsub(u1, u3);
    x[0] = xadd(v0, v1);
    x[1] = xsub(v0, v1);
    x[2] = X31{sub31(v2.c, v3.d), add31(v2.d, v3.c)};
    x[3] = X31{add31(v2.c, v3.d), sub31(v2.d, v3.c)};
}
__device__ __forceinline__ void dit_adds(X61 (&x)[4]) {
    const L61 v0 = ladd(x[0].a, x[0].b, x[1].a, x[1].b), v1 = lsub(x[0].a, x[0].b, x[1].a, x[1].b);
    const L61 v2 = ladd(x[2].a, x[2].b, x[3].a, x[3].b), v3 = lsub(x[3].a, x[3].b, x[2].a, x[2].b);
    x[0] = X61{fadd(v0.a, v2.a), fadd(v0.b, v2.b)};
    x[2] = X61{fsub(v0.a, v2.a), fsub(v0.b, v2.b)};
    x[1] = X61{fsub(v1.a, v3.b), fadd(v1.b, v3.a)};   // v1 + i v3
    x[3] = X61{fadd(v1.a, v3.b), fsub(v1.b, v3.a)};   // v1 - i v3
}
__device__ __forceinline__ void dit_adds(X31 (&x)[4]) {
    const X31 v0 = xadd(x[0], x[1]), v1 = xsub(x[0], x[1]), v2 = xadd(x[2], x[3]), v3 = xsub(x[3], x[2]);
    x[0] = xadd(v0, v2);
    x[2] = xsub(v0, v2);
    x[1] = X31{sub31(v1.c, v3.d), add31(v1.d, v3.c)};
    x[3] = X31{add31(v1.c, v3.d), sub31(v1.d, v3.c)};
}
template <class X> struct Tri { X r1, r2, r3; };
template <class X> __device__ __forceinline__ void xdif4(X (&x)[4], const Tri<X>& t) {
    dif_adds(x, xmul(x[1], t.r1), xmul(x[2], t.r2), xmul(x[3], t.r3));
}
template <class X> __device__ __forceinline__ void xdif4_1(X (&x)[4]) { const X a = x[1], b = x[2], c = x[3]; dif_adds(x, a, b, c); }
template <class X> __device__ __forceinline__ void xdit4(X (&x)[4], const Tri<X>& t) {
    dit_adds(x);
    x[1] = xmulc(x[1], t.r1); x[2] = xmulc(x[2], t.r2); x[3] = xmulc(x[3], t.r3);
}
// centre_pair (m2_field.cuh) in one field
template <class X> __device__ __forceinline__ void xcentre(X& zk, X& zm, const X& zeta) {
    const X u0 = xaddconj(zk, zm), u1 = xsubconj(zk, zm);
    const X v0 = xsub(xsqr(u0), xmul(xsqr(u1), zeta));
    const X v1 = xmul(u0, xadd(u1, u1));
    zk = xadd(v0, v1);
    zm = xconjsub(v0, v1);
}

// twiddle of the table in one field
__device__ __forceinline__ void ldtw(X61& w, const DTw* t, u32 i) {
    const u64* q = reinterpret_cast<const u64*>(t + i);
    w.a = __ldg(q); w.b = __ldg(q + 1);
}
__device__ __forceinline__ void ldtw(X31& w, const DTw* t, u32 i) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(t + i) + 2);
    w.c = v.x; w.d = v.y;
}
template <class X> __device__ __forceinline__ Tri<X> ldtri(const DTw* tw4, u32 blk) {   // blk = S + J
    Tri<X> t;
    ldtw(t.r1, tw4, 3 * blk); ldtw(t.r2, tw4, 3 * blk + 1); ldtw(t.r3, tw4, 3 * blk + 2);
    return t;
}

// the weighted element of digits d0, d1; s: their shifts in bytes 0 and 1
__device__ __forceinline__ X61 weigh61(i64 d0, i64 d1, u32 s) { return X61{rotl61(digit_to61(d0), s & 0xffu), rotl61(digit_to61(d1), (s >> 8) & 0xffu)}; }
__device__ __forceinline__ X31 weigh31(i64 d0, i64 d1, u32 s) { return X31{rotl31(digit_to31(d0), s & 0xffu), rotl31(digit_to31(d1), (s >> 8) & 0xffu)}; }

// ---- radix-8 levels ----
// Three levels of the per-block-twiddle transform at once: with r^8 = c the
// residues mod X^m - r w^e, w = (1 + i) / sqrt 2, e = 0, 4, 2, 6, 1, 5, 3, 7.
// sqrt 2 is 2^31 in GF(P61) and 2^16 in GF(P31): a product by w is an
// addition, a subtraction and two shifts, and 7 products by twiddles do the
// work of 9 in radix-4 levels.
//
// x below 7 2^61 times 2^30 modulo P61, below 2^61 + 2^33
__device__ __forceinline__ u64 scale61(u64 x) { return ((x & 0x7fffffffull) << 30) + (x >> 31); }
__device__ __forceinline__ u32 scale31(u32 x) { return rotl31(x, 15); }
// w (x - y): the difference offset by 2 P61 (below 3 2^61 + 8), the sum and the
// difference of its coordinates (offset by 4 P61) below 7 2^61 + 16
__device__ __forceinline__ X61 eighth_of_diff(const X61& x, const X61& y) {
    const L61 d = lsub(x.a, x.b, y.a, y.b);
    return X61{scale61(d.a + (K4_61 - d.b)), scale61(d.a + d.b)};
}
__device__ __forceinline__ X31 eighth_of_diff(const X31& x, const X31& y) {
    const X31 d = xsub(x, y);
    return X31{scale31(sub31(d.c, d.d)), scale31(add31(d.c, d.d))};
}
// conj(w) x, x below 2^61 + 8
__device__ __forceinline__ X61 eighth_conj(const X61& x) { return X61{scale61(x.a + x.b), scale61(x.b + (K2_61 - x.a))}; }
__device__ __forceinline__ X31 eighth_conj(const X31& x) { return X31{scale31(add31(x.c, x.d)), scale31(sub31(x.d, x.c))}; }

// i x, x below 2 P61
__device__ __forceinline__ X61 times_i(const X61& x) { return X61{K2_61 - x.b, x.a}; }
__device__ __forceinline__ X31 times_i(const X31& x) { return xtimes_i(x); }

template <class X> __device__ __forceinline__ void dif8_adds(X (&x)[8]) {
    X a[4], b[4];
    a[0] = xadd(x[0], x[4]); b[0] = xsub(x[0], x[4]);
    a[1] = xadd(x[1], x[5]); b[1] = eighth_of_diff(x[1], x[5]);
    a[2] = xadd(x[2], x[6]); b[2] = times_i(xsub(x[2], x[6]));
    a[3] = xadd(x[3], x[7]); b[3] = times_i(eighth_of_diff(x[3], x[7]));
    dif_adds(a, a[1], a[2], a[3]);
    dif_adds(b, b[1], b[2], b[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) { x[k] = a[k]; x[4 + k] = b[k]; }
}
template <class X> __device__ __forceinline__ void dit8_adds(X (&x)[8]) {
    X a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { a[k] = x[k]; b[k] = x[4 + k]; }
    dit_adds(a);
    dit_adds(b);
    b[1] = eighth_conj(b[1]);
    b[2] = times_i(b[2]);                  // its negative: -i b[2] is taken off
    b[3] = times_i(eighth_conj(b[3]));
    x[0] = xadd(a[0], b[0]); x[4] = xsub(a[0], b[0]);
    x[1] = xadd(a[1], b[1]); x[5] = xsub(a[1], b[1]);
    x[2] = xsub(a[2], b[2]); x[6] = xadd(a[2], b[2]);
    x[3] = xsub(a[3], b[3]); x[7] = xadd(a[3], b[3]);
}
// x[k] times entry k - 1 of t (its conjugate)
template <class X> __device__ __forceinline__ void twist8(X (&x)[8], const DTw* t) {
#pragma unroll
    for (int k = 1; k < 8; ++k) {
        X w;
        ldtw(w, t, k - 1);
        x[k] = xmul(x[k], w);
    }
}
template <class X> __device__ __forceinline__ void untwist8(X (&x)[8], const DTw* t) {
#pragma unroll
    for (int k = 1; k < 8; ++k) {
        X w;
        ldtw(w, t, k - 1);
        x[k] = xmulc(x[k], w);
    }
}

// named barrier of N threads
template <u32 N> __device__ __forceinline__ void bar_field(u32 id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory"); }

__device__ __forceinline__ u64 now_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// A bounded wait: after the limit (about a second of polls) the status word
// gets ST_WAIT_TIMEOUT and this thread waits no more in this launch; every
// other waiter sees the status word and gives up too.
struct Wait {
    int* status;
    bool dead;
    __device__ __forceinline__ bool again(u32& it) {   // after an unsuccessful poll
        if (dead) return false;
        if ((++it & 255u) == 0) {
            if (*(volatile int*)status & ST_WAIT_TIMEOUT) { dead = true; return false; }
            if (it > (1u << 21)) { atomicOr(status, ST_WAIT_TIMEOUT); dead = true; return false; }
        }
        if (it > 64) __nanosleep(40);
        return true;
    }
};
// Every CTA of a cooperative launch waits here until all of them have started;
// false: the launch is called off, for all of them.  The state stays as it was
// then, and the k squarings are added to those that the host still has to run
// (StateWords::owed).  A launch that asks (`ask`) is called off by its first CTA
// when the context's host word says that other work waits: queued launches give
// way within the one that runs.  CTAs whose grid does not start whole would call
// it off after 20 ms; on a GB300 all CTAs of a cooperative grid start at one
// instant (measured beside kernels that came free one by one).
//
// arrivals: the low 48 bits count the CTAs of all launches, bits 62 and 63 mark a
// launch of even and odd index as called off.  A mark is set while the count is
// short of the launch's last CTA (by the first CTA before it counts itself, by
// others with compare-and-swap), so a CTA that sees the full count without the
// mark sees what all the others see; the first CTA to arrive of the next launch
// takes it away, when every CTA of this one has read it.
__device__ __forceinline__ bool all_started(unsigned long long* arrivals, u32 ctas, int* status, u32 k, u32 ask) {
    __shared__ int runs;
    if (threadIdx.x == 0) {
        StateWords* words = reinterpret_cast<StateWords*>(status);
        constexpr u64 COUNT = (1ull << 48) - 1;
        const volatile unsigned* yield = ask && blockIdx.x == 0 ? words->yield : nullptr;
        const bool give_way = yield && *yield;
        const u64 t0 = now_ns();
        u64 v = *(volatile u64*)arrivals;
        if (!give_way) v = atomicAdd(arrivals, 1ull);
        // (other CTAs of this launch may arrive meanwhile, but not its last)
        const u64 launch = (v & COUNT) / ctas, full = (launch + 1) * ctas, off = 1ull << (62 + (launch & 1));
        if (give_way) {
            if (!(atomicOr(arrivals, off) & off)) atomicAdd(&words->owed, (unsigned long long)k);
            v = atomicAdd(arrivals, 1ull);
        }
        if ((v & COUNT) == launch * ctas) atomicAnd(arrivals, ~(1ull << (63 - (launch & 1))));   // the mark of the launch before
        do {
            v = *(volatile u64*)arrivals;
            if ((v & off) || (v & COUNT) >= full) break;
            if (now_ns() - t0 < 20000000ull) {
                __nanosleep(200);
            } else if (atomicCAS(arrivals, v, v | off) == v) {
                atomicAdd(&words->owed, (unsigned long long)k);
                v |= off;
            }
        } while (!(v & off));
        runs = !(v & off);
    }
    __syncthreads();
    return runs != 0;
}

}  // namespace

}  // namespace M2K_NS
