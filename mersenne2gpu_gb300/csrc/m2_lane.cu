// m2_lane.cu -- k squarings of one small test (n = 32 ... 256) in one CTA,
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
// at h = 128.  Measured, us per squaring, one-CTA kernel -> here: n = 2^8 7.64
// -> 1.57; n = 2^5 0.90.
#include "m2_lane.cuh"

namespace M2K_NS {

namespace {

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
        zeta = centre_root<X>(tc, k);
    }
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
            x = centre_one(x, o, zeta, k);
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

// From h = 256 on the transform is spread over a cluster (m2_cluster.cu): here
// h = 256 took 2.98 us a squaring, h = 512 7.0 (1024 threads of 64 registers).
bool lane_supported(unsigned h, int span, int carry_threads) { return h >= 16 && h <= 128 && span == 2 && carry_threads > 0; }

cudaError_t launch_lane(const SmallTest* d_tests, int ntests, unsigned h, unsigned iters_override, cudaStream_t s, bool gf61) {
#if M2_DUAL
    if (gf61) return m2k_g61::launch_lane(d_tests, ntests, h, iters_override, s, true);
#endif
    switch (h) {
#define M2_LANE(A) case 1u << A: k_lane<A><<<ntests, Lane<A>::NT, 0, s>>>(d_tests, iters_override); break;
        M2_LANE(4) M2_LANE(5) M2_LANE(6) M2_LANE(7)
#undef M2_LANE
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace M2K_NS
