// m2_cluster.cu -- k squarings of one test of n = 2^9 ... 2^13 in one
// thread-block cluster, one element of the transform per thread and field.
//
// The design of m2_lane.cu (see there) spread over 4 to 16 SMs, which turns
// the pipe-bound time of one SM into latency again: CTAs of 64 to 256
// elements, whose exchanges across CTAs are single asynchronous stores into
// the reader's shared memory, counted by an mbarrier per reading warp: about
// 300 cycles an exchange, where a cluster barrier takes 650-750 and polling the
// slots 350-450.  A slot is written again only by values that depend on what
// its reader made of it, so nothing is overwritten before it is read.
//
// Element k of a thread (lane, warp w, CTA c), log2 of the CTA's elements = N,
// W = N - 5 warp bits:
//   distribution 0 (the first two steps)  lane at the top, c, w:  k = lane | c | w
//   distribution 1 (steps 3 and 4)        c at the top, lane, w:  k = c | lane | w
//   distribution 2 (the rest, the centre) c at the top, w, lane:  k = c | w | lane
// 0 -> 1 and 1 -> 0 and the mirror pairs cross CTAs, 1 <-> 2 stay inside.  The
// row stage runs in distribution 0; the carry goes to the owner of element
// k + 1 the same way, twice (carry span 2).
//
// What bounds it: the chain of a thread (11 half-steps, the centre and the row
// stage at h = 2048, about 5000 cycles) and five exchanges across CTAs.
// Measured, us per squaring, before -> here: n = 2^9 2.98 -> 2.06, 2^10 7.0 ->
// 2.35, 2^11 12.2 -> 2.7, 2^12 6.5 -> 3.2, 2^13 6.5 -> 4.9 (one CTA up to
// 2^11, the one-launch kernel of m2_flow.cu above).
#include "m2_lane.cuh"

namespace M2K_NS {

namespace {

__device__ __forceinline__ u32 smem_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ u32 map_to(u32 addr, u32 rank) {
    u32 r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// A word for another thread: into its slot, counted by its warp's mbarrier.
__device__ __forceinline__ void send(u32 slot, u32 bar, const X61& v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(slot), "l"(v.a), "l"(v.b), "r"(bar) : "memory");
}
__device__ __forceinline__ void send(u32 slot, u32 bar, const X31& v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(slot), "r"(v.c), "r"(v.d), "r"(bar) : "memory");
}
__device__ __forceinline__ void send(u32 slot, u32 bar, i64 c) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(slot), "l"(c), "r"(bar) : "memory");
}
// a slot that another CTA wrote
__device__ __forceinline__ X61 ld_slot(const X61* p) {
    X61 v;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ X31 ld_slot(const X31* p) {
    X31 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.c), "=r"(v.d) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ i64 ld_slot(const i64* p) {
    i64 v;
    asm volatile("ld.shared.s64 %0, [%1];" : "=l"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void arm(u32 bar, u32 bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// The warp's words of this squaring have arrived.  Bounded: after two seconds
// the status word gets ST_WAIT_TIMEOUT; a warp that has given up, or sees that
// another has, neither waits, arms nor sends any more in this launch.
__device__ __forceinline__ bool arrived(u32 bar, u32 parity) {
    u32 done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ void await(u32 bar, u32 parity, Wait& w) {
    if (w.dead || arrived(bar, parity)) return;
    const u64 t0 = now_ns();
    u32 it = 0;
    while (!arrived(bar, parity)) {
        if ((++it & 15u) != 0) continue;
        if (*(volatile int*)w.status & ST_WAIT_TIMEOUT) w.dead = true;
        else if (now_ns() - t0 > 2000000000ull) { atomicOr(w.status, ST_WAIT_TIMEOUT); w.dead = true; }
        if (w.dead) break;
    }
}

template <int A_, int N_> struct Shape {
    static constexpr int A = A_, N = N_, W = N - 5, CB = A - N;
    static constexpr u32 H = 1u << A, NE = 1u << N, CTAS = 1u << CB, NT = kDual ? 2 * NE : NE;
    static constexpr int NL = A / 2;                    // radix-4 steps
    static constexpr bool ODD = (A & 1) != 0;           // and one radix-2 step
    static constexpr bool MID = A > 9;                  // distribution 1 is used
    // its two steps' bits A - 5 ... A - 8 are lane bits there
    static_assert(!MID || (A - 5 <= N - 1 && A - 8 >= W), "steps 3 and 4 run over lanes");
    static __device__ __forceinline__ u32 k0(u32 cta, u32 t) { return ((t & 31u) << (A - 5)) | (cta << W) | (t >> 5); }
    static __device__ __forceinline__ u32 k1(u32 cta, u32 t) { return (cta << N) | ((t & 31u) << W) | (t >> 5); }
    static __device__ __forceinline__ u32 k2(u32 cta, u32 t) { return (cta << N) | t; }
    // CTA and thread of element k
    static __device__ __forceinline__ u32 cta0(u32 k) { return (k >> W) & (CTAS - 1); }
    static __device__ __forceinline__ u32 t0(u32 k) { return ((k & ((1u << W) - 1)) << 5) | (k >> (A - 5)); }
    static __device__ __forceinline__ u32 cta12(u32 k) { return k >> N; }
    static __device__ __forceinline__ u32 t1(u32 k) { return ((k & ((1u << W) - 1)) << 5) | ((k >> W) & 31u); }
    static __device__ __forceinline__ u32 t2(u32 k) { return k & (NE - 1); }
    // slot of a CTA's element in the exchanges inside it: distributions 1 and 2
    // on distinct bank groups
    static __device__ __forceinline__ u32 slot(u32 e) { return e ^ ((e >> W) & 7u); }
};

// a field's shared memory: slots read by thread index, the mbarriers of each
// warp's slots, and the exchanges between distributions 1 and 2
template <class S, class X> struct Bufs {
    X to1[S::NE], to0[S::NE], mir[S::NE], in12[S::NE], in21[S::NE];
    u64 bar1[S::NE / 32], bar0[S::NE / 32], barm[S::NE / 32];
};

template <class S, class X> struct Xform {
    X tw[S::NL], tr, zeta;
    u32 t, bar, k2;
    u32 dst1, dst0, dstm, rb1, rb0, rbm;    // where this thread's elements go: slots and mbarriers
    Bufs<S, X>* b;

    __device__ __forceinline__ Xform(u32 cta, u32 t_, u32 bar_, Bufs<S, X>* b_, const DTw* tw4, const DTw* tc) : t(t_), bar(bar_), b(b_) {
        const u32 k0 = S::k0(cta, t), k1 = S::MID ? S::k1(cta, t) : S::k2(cta, t);
        k2 = S::k2(cta, t);
#pragma unroll
        for (int l = 0; l < S::NL; ++l) {
            const u32 e = l < 2 ? k0 : l < 4 ? k1 : k2;
            const u32 blk = (1u << (2 * l)) + (e >> (S::A - 2 * l)), m = (e >> (S::A - 2 - 2 * l)) & 3u;
            if (m) ldtw(tw[l], tw4, 3 * blk + m - 1);
            else tw[l] = xone(tw[l]);
        }
        if (k2 & 1u) ldtw(tr, tc, k2 >> 1);
        else tr = xone(tr);
        zeta = centre_root<X>(tc, k2);
        const u32 t1 = S::MID ? S::t1(k0) : S::t2(k0), t0 = S::t0(k1), mk = mirror(k2), tm = S::t2(mk);
        dst1 = map_to(smem_addr(&b->to1[t1]), S::cta12(k0));
        rb1 = map_to(smem_addr(&b->bar1[t1 >> 5]), S::cta12(k0));
        dst0 = map_to(smem_addr(&b->to0[t0]), S::cta0(k1));
        rb0 = map_to(smem_addr(&b->bar0[t0 >> 5]), S::cta0(k1));
        dstm = map_to(smem_addr(&b->mir[tm]), S::cta12(mk));
        rbm = map_to(smem_addr(&b->barm[tm >> 5]), S::cta12(mk));
    }
    __device__ __forceinline__ void sync() const { bar_field<S::NE>(bar); }
    // lane bit of step l's low element bit
    static constexpr __host__ __device__ int lb(int l) { return S::A - 2 - 2 * l - (l < 2 ? S::A - 5 : (S::MID && l < 4) ? S::W : 0); }

    // forward transform, centre square, inverse transform: distribution 0 in and out
    __device__ __forceinline__ X square(X x, u32 par, Wait& w) const {
        const u32 wp = t >> 5;
        if ((t & 31u) == 0 && !w.dead) {
            arm(smem_addr(&b->bar1[wp]), 32 * sizeof(X));
            arm(smem_addr(&b->barm[wp]), 32 * sizeof(X));
            arm(smem_addr(&b->bar0[wp]), 32 * sizeof(X));
        }
        const u32 kl = ((t & 31u) << S::W) | (t >> 5);      // distribution 1: the CTA's element
        x = step_fwd(x, lb(0), (t >> lb(0)) & 3u);
        x = step_fwd(xmul(x, tw[1]), lb(1), (t >> lb(1)) & 3u);
        if (!w.dead) send(dst1, rb1, x);
        await(smem_addr(&b->bar1[wp]), par, w);
        x = ld_slot(&b->to1[t]);
#pragma unroll
        for (int l = 2; l < S::NL; ++l) {
            if (S::MID && l == 4) {
                b->in12[S::slot(kl)] = x;
                sync();
                x = b->in12[S::slot(t)];
            }
            x = step_fwd(xmul(x, tw[l]), lb(l), (t >> lb(l)) & 3u);
        }
        if (S::ODD) x = folded(layer_first(xmul(x, tr), 1u, (t & 1u) != 0));
        if (!w.dead) send(dstm, rbm, x);
        await(smem_addr(&b->barm[wp]), par, w);
        const X o = ld_slot(&b->mir[t]);
        x = centre_one(x, o, zeta, k2);
        if (S::ODD) x = xmulc(folded(layer_first(x, 1u, (t & 1u) != 0)), tr);
#pragma unroll
        for (int l = S::NL - 1; l >= 2; --l) {
            if (S::MID && l == 3) {
                b->in21[S::slot(t)] = x;
                sync();
                x = b->in21[S::slot(kl)];
            }
            x = xmulc(step_inv(x, lb(l), (t >> lb(l)) & 3u), tw[l]);
        }
        if (!w.dead) send(dst0, rb0, x);
        await(smem_addr(&b->bar0[wp]), par, w);
        x = ld_slot(&b->to0[t]);
        x = xmulc(step_inv(x, lb(1), (t >> lb(1)) & 3u), tw[1]);
        return step_inv(x, lb(0), (t >> lb(0)) & 3u);
    }
};

template <class S>
__global__ void __launch_bounds__(S::NT, 1) k_cluster(const SmallTest* test, u32 iters, u32 stall) {
    __shared__ Bufs<S, X61> b61;
    __shared__ Bufs<S, X31> b31;
    __shared__ X31 r31[S::NE];          // GF(P31) residues of the row stage
    __shared__ longlong2 dig[S::NE];    // new digits for the GF(P31) threads
    __shared__ i64 cx[2][S::NE];        // carries from element k - 1
    __shared__ u64 barc[2][S::NE / 32];
    const SmallTest T = *test;
    const u32 cta = blockIdx.x;
    const bool second = kDual && threadIdx.x >= S::NE;
    const u32 t = second ? threadIdx.x - S::NE : threadIdx.x, k = S::k0(cta, t);
    const u32 pair = 3 + (t >> 5);      // barrier of this element's two warps
    const int ln = T.ln;
    const u32 p = T.p;
    Wait w{T.status, false};
    if ((t & 31u) == 0) {
        auto init = [](u64* m) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(m)) : "memory"); };
        const u32 wp = t >> 5;
        if (second) {
            init(&b31.bar1[wp]); init(&b31.bar0[wp]); init(&b31.barm[wp]);
        } else {
            init(&b61.bar1[wp]); init(&b61.bar0[wp]); init(&b61.barm[wp]);
            init(&barc[0][wp]); init(&barc[1][wp]);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster_sync();
    if (second) {
        const u32 s0 = T.w31[2 * k], s1 = T.w31[2 * k + 1];
        const u32 s = s0 | (s1 << 8);
        auto un = [&](u32 v) { const u32 q = (v + (u32)ln + 1u) % 31u; return q ? 31u - q : 0u; };
        const u32 q0 = un(s0), q1 = un(s1);
        const Xform<S, X31> F(cta, t, 2, &b31, T.tw4, T.tc);
        X31 x = weigh31(T.digits[2 * k], T.digits[2 * k + 1], s);
        for (u32 it = 0; it < iters; ++it) {
            x = F.square(x, it & 1u, w);
            r31[t] = X31{rotl31(x.c, q0), rotl31(x.d, q1)};
            bar_field<64>(pair);
            bar_field<64>(pair);
            const longlong2 d = dig[t];
            x = weigh31(d.x, d.y, s);
        }
    } else {
        const u32 s0 = T.w61[2 * k], s1 = T.w61[2 * k + 1];
        const u32 s = s0 | (s1 << 8);
        auto un = [&](u32 v) { const u32 q = (v + (u32)ln + 1u) % 61u; return q ? 61u - q : 0u; };
        const u32 q0 = un(s0), q1 = un(s1);
        const u32 wd0 = width_of(p, ln, 2 * k), wd1 = width_of(p, ln, 2 * k + 1);
        const u32 next = (k + 1u) & (S::H - 1), mul = (T.mode == PRP3) ? 3u : 1u;
        const i64 sub = (T.mode == LL && k == 0) ? 2 : 0;
        const u32 tn = S::t0(next), cn = S::cta0(next);
        const u32 cdst0 = map_to(smem_addr(&cx[0][tn]), cn), cdst1 = map_to(smem_addr(&cx[1][tn]), cn);
        const u32 cbar0 = map_to(smem_addr(&barc[0][tn >> 5]), cn), cbar1 = map_to(smem_addr(&barc[1][tn >> 5]), cn);
        const u32 mine0 = smem_addr(&barc[0][t >> 5]), mine1 = smem_addr(&barc[1][t >> 5]);
        const u32 cbytes = stall && cta == 0 ? 33 * 8 : 32 * 8;   // stall: one carry more than there are
        const Xform<S, X61> F(cta, t, 1, &b61, T.tw4, T.tc);
        i64 d0 = T.digits[2 * k], d1 = T.digits[2 * k + 1];
        u32 bad = 0;
        for (u32 it = 0; it < iters; ++it) {
            const u32 par = it & 1u;
            if ((t & 31u) == 0 && !w.dead) { arm(mine0, cbytes); arm(mine1, 32 * 8); }
            X61 x = weigh61(d0, d1, s);
            x = F.square(x, par, w);
            const u64 x0 = rotl61(fold61(x.a), q0), x1 = rotl61(fold61(x.b), q1);
            if (kDual) bar_field<64>(pair);
            const X31 y = kDual ? r31[t] : X31{0u, 0u};
            i64 c = 0;
            d0 = crt_digit(x0, y.c, wd0, mul, sub, c, bad, !kDual);
            d1 = crt_digit(x1, y.d, wd1, mul, 0, c, bad, !kDual);
            // carry span 2: the carry into digit 0 leaves digit 1 small
            if (!w.dead) send(cdst0, cbar0, c);
            await(mine0, par, w);
            c = ld_slot(&cx[0][t]);
            d0 = split_balanced64(d0 + c, wd0, c);
            d1 = split_balanced64(d1 + c, wd1, c);
            if (!w.dead) send(cdst1, cbar1, c);
            await(mine1, par, w);
            d0 += ld_slot(&cx[1][t]);
            if (kDual) {
                dig[t] = make_longlong2(d0, d1);
                bar_field<64>(pair);
            }
        }
        if (bad) atomicOr(T.status, ST_CARRY_RANGE);
        T.digits[2 * k] = d0; T.digits[2 * k + 1] = d1;
    }
    cluster_sync();   // no CTA leaves while another may still write to it
    // words for a warp that has given up are not waited for: the last of them were
    // sent before the barrier, and its CTA stays for far longer than one takes
    if (w.dead)
        for (const u64 t0 = now_ns(); now_ns() - t0 < 20000ull;) {}
}

template <class S> cudaError_t config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, cudaStream_t s) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(S::CTAS);
    cfg.blockDim = dim3(S::NT);
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S::CTAS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return S::CTAS > 8 ? cudaFuncSetAttribute(k_cluster<S>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : cudaSuccess;
}
template <class S> cudaError_t fits() {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    cudaError_t e = config<S>(cfg, at, nullptr);
    int n = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, k_cluster<S>, &cfg);
    return e == cudaSuccess && n < 1 ? cudaErrorNotSupported : e;
}
template <class S> cudaError_t launch(const SmallTest* d_test, u32 iters, u32 stall, cudaStream_t s) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    const cudaError_t e = config<S>(cfg, at, s);
    return e ? e : cudaLaunchKernelEx(&cfg, k_cluster<S>, d_test, iters, stall);
}

// log2 h, log2 elements per CTA.  Fewer elements per CTA shorten the steps'
// share until the CTA has one warp a scheduler (h = 256: 64 elements 2.06 us a
// squaring, 128 2.4; h = 512: 64 2.35, 128 2.6; h = 2048: 128 3.2, 256 4.4);
// h = 1024 with 64 elements (16 CTAs) gained 1% over 128 (8 CTAs); h = 128 is
// better off in one CTA (1.57).
#define M2_CLUSTER_SHAPES(X) X(8, 6) X(9, 6) X(10, 7) X(11, 7) X(12, 8)

}  // namespace

bool cluster_supported(int lh, int span, bool gf61) {
#if M2_DUAL
    if (gf61) return m2k_g61::cluster_supported(lh, span, true);
#endif
    if (span != 2) return false;
    cudaError_t e = cudaErrorNotSupported;
#define M2_CLUSTER_F(A, N) if (lh == A) e = fits<Shape<A, N>>();
    M2_CLUSTER_SHAPES(M2_CLUSTER_F)
#undef M2_CLUSTER_F
    cudaGetLastError();
    return e == cudaSuccess;
}

cudaError_t launch_cluster(const SmallTest* d_test, int lh, unsigned iters, bool stall, bool gf61, cudaStream_t s) {
#if M2_DUAL
    if (gf61) return m2k_g61::launch_cluster(d_test, lh, iters, stall, true, s);
#endif
#define M2_CLUSTER_L(A, N) if (lh == A) return launch<Shape<A, N>>(d_test, iters, stall ? 1u : 0u, s);
    M2_CLUSTER_SHAPES(M2_CLUSTER_L)
#undef M2_CLUSTER_L
    return cudaErrorInvalidValue;
}

}  // namespace M2K_NS
