// m2_lane.cu -- k squarings of one small test (n = 32 ... 1024) in one CTA,
// one element of the transform per thread and field.
//
// A lone small transform is all latency: the one-CTA kernel of m2_kernels.cu
// gives each of its few warps four elements a step and leaves the SM's other
// schedulers idle.  Here element k lives in a register of one thread per field
// (h threads for GF(P61^2), h for GF(P31^2), on warps of their own), a radix-4
// step is one product per thread and two add layers over lane exchanges, and
// everything that does not change from squaring to squaring (twiddles, shifts,
// widths, partners) stays in registers.
//
// Distribution 0 (the first two steps) holds the top five index bits in the
// lane, distribution 1 (the other steps and the centre) the low five; the two
// are exchanged through shared memory, as are the mirror pairs of the centre,
// whose two threads each compute the output that they keep.  In the row stage
// the GF(P61) thread of an element takes its GF(P31) residue, does both
// digits, passes the carry to its successor twice (it leaves the second digit
// as -1, 0 or 1: carry span 2) and hands the new digits back.
//
// What bounds it: the serial chain of one thread (eight steps of one product
// and two add layers at h = 128, the centre, the row stage), about 3400 cycles
// at h = 128; at h = 512 the SM's integer pipes (32 warps of 64 registers).
// Measured, us per squaring, one-CTA kernel -> here: n = 2^8 7.64 -> 1.66,
// 2^9 7.84 -> 3.17, 2^10 8.61 -> 7.35; n = 2^5 0.94.
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

template <int A> struct Lane {
    static constexpr u32 H = 1u << A, NF = H < 32 ? 32 : H, NT = kDual ? 2 * NF : NF;
    static constexpr int NL = A / 2;                    // radix-4 steps
    static constexpr bool ODD = (A & 1) != 0;           // and one radix-2 step
    static constexpr int SH = A > 5 ? A - 5 : 0;        // lane bit j is element bit j + SH in distribution 0
    static constexpr int N0 = A > 5 ? 2 : NL;           // radix-4 steps in distribution 0
    // element of a thread in distribution 0 and 1 (below 32 elements, the
    // upper lanes repeat the lower ones' work)
    static __device__ __forceinline__ u32 e0(u32 t) { return A > 5 ? ((t & 31u) << SH) | (t >> 5) : t & (H - 1); }
    static __device__ __forceinline__ u32 e1(u32 t) { return t & (H - 1); }
    // slot of element e: both distributions' accesses on distinct bank groups
    static __device__ __forceinline__ u32 slot(u32 e) { return A > 5 ? e ^ ((e >> SH) & 7u) : e; }
};

template <u32 N> __device__ __forceinline__ void bar_field(u32 id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory"); }

// the transform of one thread in one field
template <int A, class X> struct Xform {
    using L = Lane<A>;
    X tw[L::NL];        // twiddle of each radix-4 step (step 0 has root 1)
    X tr, zeta;         // radix-2 twiddle, centre root
    u32 t, bar;
    X *bufa, *bufb;     // exchanges between distributions, mirror pairs

    __device__ __forceinline__ Xform(u32 t_, u32 bar_, X* buf, const DTw* tw4, const DTw* tc) : t(t_), bar(bar_) {
        bufa = buf; bufb = buf + L::H;
#pragma unroll
        for (int l = 0; l < L::NL; ++l) {
            const u32 e = l < L::N0 ? L::e0(t) : L::e1(t);
            const u32 blk = (1u << (2 * l)) + (e >> (A - 2 * l)), m = (e >> (A - 2 - 2 * l)) & 3u;
            if (m) ldtw(tw[l], tw4, 3 * blk + m - 1);
            else tw[l] = xone(tw[l]);
        }
        const u32 k = L::e1(t);
        if (k & 1u) ldtw(tr, tc, k >> 1);
        else tr = xone(tr);
        // the pair's root is at its even position; positions 0 and 1 (roots 1
        // and -1) are their own mirrors
        const u32 mk = mirror(k);
        ldtw(zeta, tc, ((k & 1u) ? mk : k) >> 1);
        if (k == 1u) zeta = xminus(zeta);
    }
    static __device__ __forceinline__ X61 xminus(const X61&) { return X61{P61 - 1, 0}; }
    static __device__ __forceinline__ X31 xminus(const X31&) { return X31{P31 - 1, 0}; }
    static __device__ __forceinline__ u32 mirror(u32 k) { return k < 2 ? k : (3u << (31 - __clz(k))) - k - 1u; }
    __device__ __forceinline__ void sync() const { bar_field<L::NF>(bar); }

    // forward transform, centre square, inverse transform: distribution 0 in and out
    __device__ __forceinline__ X square(X x) const {
        const u32 f0 = L::slot(L::e0(t)), k = L::e1(t), f1 = L::slot(k);
#pragma unroll
        for (int l = 0; l < L::N0; ++l) {
            const int b = A - 2 - 2 * l - L::SH;
            if (l > 0) x = xmul(x, tw[l]);
            x = step_fwd(x, b, (t >> b) & 3u);
        }
        if (A > 5) {
            bufa[f0] = x;
            sync();
            x = bufa[f1];
        }
#pragma unroll
        for (int l = L::N0; l < L::NL; ++l) {
            const int b = A - 2 - 2 * l;
            x = xmul(x, tw[l]);
            x = step_fwd(x, b, (t >> b) & 3u);
        }
        if (L::ODD) {
            x = xmul(x, tr);
            x = folded(layer_first(x, 1u, (t & 1u) != 0));
        }
        // centre: this thread's output of the pair
        bufb[f1] = x;
        sync();
        {
            const X o = bufb[L::slot(mirror(k))];
            const bool odd = (k & 1u) != 0 && k != 1u;
            const X zk = odd ? o : x, zm = odd ? x : o;
            const X u0 = xaddconj(zk, zm), u1 = xsubconj(zk, zm);
            const X v0 = xsub(xsqr(u0), xmul(xsqr(u1), zeta));
            const X v1 = xmul(u0, xadd(u1, u1));
            x = odd ? xconjsub(v0, v1) : xadd(v0, v1);
        }
        if (L::ODD) {
            x = folded(layer_first(x, 1u, (t & 1u) != 0));
            x = xmulc(x, tr);
        }
#pragma unroll
        for (int l = L::NL - 1; l >= L::N0; --l) {
            const int b = A - 2 - 2 * l;
            x = step_inv(x, b, (t >> b) & 3u);
            x = xmulc(x, tw[l]);
        }
        if (A > 5) {
            bufa[f1] = x;
            sync();
            x = bufa[f0];
        }
#pragma unroll
        for (int l = L::N0 - 1; l >= 0; --l) {
            const int b = A - 2 - 2 * l - L::SH;
            x = step_inv(x, b, (t >> b) & 3u);
            if (l > 0) x = xmulc(x, tw[l]);
        }
        return x;
    }
};

template <int A>
__global__ void __launch_bounds__(Lane<A>::NT, 1) k_lane(const SmallTest* tests, u32 iters_override) {
    using L = Lane<A>;
    __shared__ X61 b61[2 * L::H];
    __shared__ X31 b31[2 * L::H];
    __shared__ X31 r31[L::H];           // GF(P31) residues of the row stage
    __shared__ longlong2 dig[L::H];     // new digits for the GF(P31) threads
    __shared__ i64 cx[2][L::H];
    const SmallTest T = tests[blockIdx.x];
    const u32 iters = iters_override ? iters_override : T.iters;
    const bool second = kDual && threadIdx.x >= L::NF;
    const u32 t = second ? threadIdx.x - L::NF : threadIdx.x, k = L::e0(t);
    const int ln = T.ln;
    const u32 p = T.p;
    if (second) {
        const u32 s0 = T.w31[2 * k], s1 = T.w31[2 * k + 1];
        const u32 s = s0 | (s1 << 8);
        auto un = [&](u32 v) { const u32 q = (v + (u32)ln + 1u) % 31u; return q ? 31u - q : 0u; };
        const u32 q0 = un(s0), q1 = un(s1);
        const Xform<A, X31> F(t, 2, b31, T.tw4, T.tc);
        X31 x = weigh31(T.digits[2 * k], T.digits[2 * k + 1], s);
        for (u32 it = 0; it < iters; ++it) {
            x = F.square(x);
            r31[k] = X31{rotl31(x.c, q0), rotl31(x.d, q1)};
            __syncthreads();
            __syncthreads();
            const longlong2 d = dig[k];
            x = weigh31(d.x, d.y, s);
        }
        return;
    }
    const u32 s0 = T.w61[2 * k], s1 = T.w61[2 * k + 1];
    const u32 s = s0 | (s1 << 8);
    auto un = [&](u32 v) { const u32 q = (v + (u32)ln + 1u) % 61u; return q ? 61u - q : 0u; };
    const u32 q0 = un(s0), q1 = un(s1);
    const u32 wd0 = width_of(p, ln, 2 * k), wd1 = width_of(p, ln, 2 * k + 1);
    const u32 prev = (k - 1u) & (L::H - 1), mul = (T.mode == PRP3) ? 3u : 1u;
    const i64 sub = (T.mode == LL && k == 0) ? 2 : 0;
    const Xform<A, X61> F(t, 1, b61, T.tw4, T.tc);
    i64 d0 = T.digits[2 * k], d1 = T.digits[2 * k + 1];
    u32 bad = 0;
    for (u32 it = 0; it < iters; ++it) {
        X61 x = weigh61(d0, d1, s);
        x = F.square(x);
        const u64 x0 = rotl61(fold61(x.a), q0), x1 = rotl61(fold61(x.b), q1);
        if (kDual) __syncthreads();
        const X31 y = kDual ? r31[k] : X31{0u, 0u};
        i64 c = 0;
        d0 = crt_digit(x0, y.c, wd0, mul, sub, c, bad, !kDual);
        d1 = crt_digit(x1, y.d, wd1, mul, 0, c, bad, !kDual);
        // carry span 2: the carry into digit 0 leaves digit 1 small
        cx[0][k] = c;
        bar_field<L::NF>(1);
        c = cx[0][prev];
        d0 = split_balanced64(d0 + c, wd0, c);
        d1 = split_balanced64(d1 + c, wd1, c);
        cx[1][k] = c;
        bar_field<L::NF>(1);
        d0 += cx[1][prev];
        if (kDual) {
            dig[k] = make_longlong2(d0, d1);
            __syncthreads();
        }
    }
    if (bad) atomicExch(T.status, ST_CARRY_RANGE);
    if (t < L::H) { T.digits[2 * k] = d0; T.digits[2 * k + 1] = d1; }
}

}  // namespace

// Up to 512 elements: 1024 threads.  n = 2^11 would need two elements a thread,
// where one CTA is bound by its SM's pipes either way.
bool lane_supported(unsigned h, int span, int carry_threads) { return h >= 16 && h <= 512 && span == 2 && carry_threads > 0; }

cudaError_t launch_lane(const SmallTest* d_tests, int ntests, unsigned h, unsigned iters_override, cudaStream_t s, bool gf61) {
#if M2_DUAL
    if (gf61) return m2k_g61::launch_lane(d_tests, ntests, h, iters_override, s, true);
#endif
    switch (h) {
#define M2_LANE(A) case 1u << A: k_lane<A><<<ntests, Lane<A>::NT, 0, s>>>(d_tests, iters_override); break;
        M2_LANE(4) M2_LANE(5) M2_LANE(6) M2_LANE(7) M2_LANE(8) M2_LANE(9)
#undef M2_LANE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace M2K_NS
