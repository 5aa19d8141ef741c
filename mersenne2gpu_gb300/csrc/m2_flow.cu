// m2_flow.cu -- k squarings of one mid-size test (n = 2^12 ... 2^20) in one
// cooperative launch.
//
// h = R x B elements as in the three-pass path, with the same roots, tables
// and element order.  CTA x owns column group x (C adjacent columns) and the
// x-th pair of mirror rows for the whole launch and alternates between them:
//   forward columns (once), then per squaring: row pair (last forward levels,
//   centre square, first inverse levels), column group (last inverse levels,
//   unweight, CRT, carry, weight, first forward levels).
//
// There is no grid barrier: the data carry the synchronisation.  A GF(P61)
// word uses 62 of its 64 bits and a GF(P31) word 31 of 32, so the top bit of
// every stored word is a tag: 0 when the column phase wrote it, 1 when the row
// phase did.  Every element is read by exactly one CTA per phase, and that CTA
// is the next to write it, so its tag alternates strictly: a reader loads its
// operands (relaxed, device scope) until all tags are the other phase's, and
// that is the whole hand-over.  Segment carries travel the same way: the word
// (carry << 1 | parity), the parity alternating per squaring, written by the
// thread that owns a segment and polled by the owner of the next one.
// Between launches every element's tag is 1.
//
// The two fields run on separate warps through every butterfly and meet only
// in the row stage (CRT, carry, weights): twice the warps to hide the latency
// of units that are small for an SM.  From n = 2^20 on, where a level has a
// butterfly for each of 1024 threads, every warp runs both fields in turn (59.0
// -> 57.7 us a squaring: the GF(P31) warps no longer finish early).
//
// What bounds it: up to n = 2^16 latency -- the serial chain of butterfly levels
// on a few warps per SM, and three L2 round trips (two hand-overs and the
// carry) -- and from n = 2^17 on the integer pipes of the SMs that have a unit.
// Measured, us per squaring, three-pass launches -> here: n = 2^12 16.2 -> 6.5,
// 2^13 18.5 -> 6.5, 2^14 19.5 -> 7.5, 2^15 21.7 -> 8.2, 2^16 27.5 -> 9.3,
// 2^17 31.9 -> 9.7, 2^18 37.3 -> 15.2, 2^19 45.6 -> 27.6, 2^20 80.9 -> 57.8
// (n = 2^12 and 2^13 run in a cluster since, m2_cluster.cu; the shapes here
// serve them where the carry span is 3).
// The three passes paid three launches per squaring, each with cold L1 tables,
// and ran rows on as few as 32 SMs.
#include "m2_flow.cuh"

namespace M2K_NS {

namespace {

template <int LR_, int LB_, int C_> struct Shape {
    static constexpr int LR = LR_, LB = LB_, C = C_;
    static constexpr u32 R = 1u << LR, B = 1u << LB, G = B / C, H = R * B;
    static constexpr u32 UC = R * C, UR = 2 * B;             // elements of a column group and of a row pair
    static constexpr u32 NBC = UC / 4, NBR = UR / 4;         // radix-4 butterflies of a level
    static constexpr u32 NB0 = NBC > NBR ? NBC : NBR;
    // units of 1024 butterflies a level and more run both fields on every warp
    static constexpr bool BOTH = NB0 >= 1024;
    static constexpr u32 NF = BOTH ? 1024 : NB0 < 32 ? 32 : NB0;   // threads per field
    static constexpr u32 NT = kDual && !BOTH ? 2 * NF : NF;
    static constexpr bool EARLY = NT <= 512;                 // registers to spare: twiddles before the barrier
    static constexpr u32 ROW_TAG = 1;
    static constexpr u32 SEGS = UC / 2;                      // carry segments (2 elements, 4 digits) of a column group
    static constexpr u32 SI = (SEGS + NT - 1) / NT;          // segments per thread
    static constexpr u32 SR = C / 2;                         // segments per row
    static constexpr u32 CTAS = G > R / 2 ? G : R / 2;
    static constexpr u32 SLOTS = UC > UR ? UC : UR;
    static constexpr u32 SMEM = 24 * SLOTS;
    // barriers of only the warps that share a block: n = 2^18 15.6 -> 15.1 us,
    // 2^19 30.0 -> 29.0, 2^20 60.9 -> 59.8; with 64 rows (at most four warps a
    // field, n up to 2^15) one barrier for all was faster (n = 2^12 6.6 against 9.4)
    static constexpr bool NARROW = R >= 256;
};

template <class S>
__global__ void __launch_bounds__(S::NT, 1) k_flow(FlowArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    X61* za = reinterpret_cast<X61*>(smem);
    X31* zb = reinterpret_cast<X31*>(smem + 16ull * S::SLOTS);
    const u32 tid = threadIdx.x, x = blockIdx.x;
    const bool second = tid >= S::NF;     // the GF(P31^2) half's warps
    const u32 fb = second ? tid - S::NF : tid;
    Unit<S, X61> ua{za, reinterpret_cast<X61*>(A.za), A.tw4, A.tc, fb, 1};
    Unit<S, X31> ub{zb, reinterpret_cast<X31*>(A.zb), A.tw4, A.tc, fb, 8};
    const bool has_cols = S::G == S::CTAS || x < S::G, has_rows = S::R / 2 == S::CTAS || x < S::R / 2;
    Wait w{A.status, false};
    if (!all_started(A.arrivals, S::CTAS, A.status, A.k, A.ask)) return;
    const u32 base = has_cols ? A.parity[x] : 0u;  // squarings handed over so far (bit 0); bit 1 never matches a word's tag

    const u32 seg = A.seg;
    // this thread's carry segments: segment s holds elements 2s, 2s+1 of the
    // column group's slots (row 2s / C)
    u32 w61[S::SI], w31[S::SI];
    uint4 aux[S::SI];
    u32 e0[S::SI];
    i64 d[S::SI][4];
#pragma unroll
    for (u32 q = 0; q < S::SI; ++q) {
        const u32 s = tid + q * S::NT, e = 2 * s;
        if (!has_cols || s >= S::SEGS) continue;
        e0[q] = (e / S::C) * S::B + x * S::C + e % S::C;
        w61[q] = *reinterpret_cast<const u32*>(A.w61 + 2 * e0[q]);
        w31[q] = *reinterpret_cast<const u32*>(A.w31 + 2 * e0[q]);
        aux[q] = *reinterpret_cast<const uint4*>(A.aux + e0[q]);
        // the state: digits, and the pending segment carries of the three-pass
        // kernels (read by their one user, then cleared)
        const longlong2* src = reinterpret_cast<const longlong2*>(A.digits + 2ull * e0[q]);
        const longlong2 v0 = src[0], v1 = src[1];
        d[q][0] = v0.x; d[q][1] = v0.y; d[q][2] = v1.x; d[q][3] = v1.y;
        if ((2 * e0[q]) % seg == 0) {
            const u32 idx = 2 * e0[q] / seg, prev = idx ? idx - 1 : 2 * S::H / seg - 1;
            i64 c = A.carries[prev];
            A.carries[prev] = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const u32 wd = (u & 1) ? ((u < 2 ? aux[q].y : aux[q].w) >> 8) & 0xffu : (u < 2 ? aux[q].y : aux[q].w) & 0xffu;
                if (u < A.span) d[q][u] = split_balanced64(d[q][u] + c, wd, c);
                else if (u == A.span) d[q][u] += c;
            }
        }
    }
    const u32 mul = (A.mode == PRP3) ? 3u : 1u;

    for (u32 it = 0;; ++it) {
        // full registers: the levels' addresses and twiddles are made anew in
        // every squaring (kept over the loop they were spilled)
        if (S::NT > 512) asm volatile("" : "+r"(ua.fb), "+r"(ub.fb));
        if (has_cols) {
            // weigh this thread's digits into the slots, then the forward levels
#pragma unroll
            for (u32 q = 0; q < S::SI; ++q) {
                const u32 s = tid + q * S::NT;
                if (s >= S::SEGS) continue;
                const u32 p = sw(2 * s);
                za[p] = weigh61(d[q][0], d[q][1], w61[q]);
                za[p ^ sw(1)] = weigh61(d[q][2], d[q][3], w61[q] >> 16);
                if (kDual) {
                    zb[p] = weigh31(d[q][0], d[q][1], w31[q]);
                    zb[p ^ sw(1)] = weigh31(d[q][2], d[q][3], w31[q] >> 16);
                }
            }
            __syncthreads();
            if (S::BOTH && kDual) run_cols_fwd<S>(x, ua, ub);
            else if (!second) run_cols_fwd<S>(x, ua);
            else run_cols_fwd<S>(x, ub);
        }
        if (!has_cols || !has_rows) __syncthreads();   // this CTA's stores of one tag before its polls for the other
        if (has_rows) {
            if (S::BOTH && kDual) run_rows<S>(x, w, ua, ub);
            else if (!second) run_rows<S>(x, w, ua);
            else run_rows<S>(x, w, ub);
        }
        if (!has_cols) {
            if (it + 1 == A.k) break;
            continue;
        }
        if (S::BOTH && kDual) run_cols_inv<S>(x, w, ua, ub);
        else if (!second) run_cols_inv<S>(x, w, ua);
        else run_cols_inv<S>(x, w, ub);
        __syncthreads();
        // unweight, CRT, carry chain of each segment; the carry goes to the
        // next segment's owner
        const u32 par = (base ^ 1u ^ it) & 1u;
        i64 cin[S::SI];
        u32 bad = 0;
#pragma unroll
        for (u32 q = 0; q < S::SI; ++q) {
            const u32 s = tid + q * S::NT;
            if (s >= S::SEGS) continue;
            const u32 p = sw(2 * s), r = s / S::SR;
            i64 c = 0;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const X61 v = za[p ^ sw(k)];
                const X31 u = kDual ? zb[p ^ sw(k)] : X31{0u, 0u};
                const u32 rot = k ? aux[q].z : aux[q].x, wd = k ? aux[q].w : aux[q].y;
                const u64 x0 = rotl61(fold61(v.a), rot & 0xffu), x1 = rotl61(fold61(v.b), (rot >> 8) & 0xffu);
                const u32 y0 = kDual ? rotl31(u.c, (rot >> 16) & 0xffu) : 0u, y1 = kDual ? rotl31(u.d, rot >> 24) : 0u;
                const i64 sub = (A.mode == LL && k == 0 && e0[q] == 0) ? 2 : 0;
                d[q][2 * k] = crt_digit(x0, y0, wd & 0xffu, mul, sub, c, bad, !kDual);
                d[q][2 * k + 1] = crt_digit(x1, y1, (wd >> 8) & 0xffu, mul, 0, c, bad, !kDual);
            }
            if (s % S::SR == S::SR - 1) st_relaxed(A.fcar + x * S::R + r, ((u64)c << 1) | par);
            cin[q] = c;
        }
        if (bad) atomicOr(A.status, ST_CARRY_RANGE);
#pragma unroll
        for (u32 q = 0; q < S::SI; ++q) {
            const u32 s = tid + q * S::NT;
            if (s >= S::SEGS) continue;
            const u32 r = s / S::SR;
            i64 c = cin[q];
            if (S::SR > 1) c = __shfl_up_sync(0xffffffffu, c, 1);
            if (s % S::SR == 0) {
                // the segment before this row's first one
                const u64* from = x ? A.fcar + (x - 1) * S::R + r : A.fcar + (S::G - 1) * S::R + ((r - 1) & (S::R - 1));
                u32 n = 0;
                u64 v;
                do {
                    v = ld_relaxed(from);
                    if ((((u32)v & 1u) | (base & 2u)) == par) break;
                } while (w.again(n));
                c = (i64)v >> 1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const u32 wd = (u & 1) ? ((u < 2 ? aux[q].y : aux[q].w) >> 8) & 0xffu : (u < 2 ? aux[q].y : aux[q].w) & 0xffu;
                if (u < A.span) d[q][u] = split_balanced64(d[q][u] + c, wd, c);
                else if (u == A.span) d[q][u] += c;
            }
        }
        if (it + 1 == A.k) break;
    }
    if (!has_cols) return;
    // the state, with no pending carries
#pragma unroll
    for (u32 q = 0; q < S::SI; ++q) {
        const u32 s = tid + q * S::NT;
        if (s >= S::SEGS) continue;
        longlong2* dst = reinterpret_cast<longlong2*>(A.digits + 2ull * e0[q]);
        dst[0] = make_longlong2(d[q][0], d[q][1]);
        dst[1] = make_longlong2(d[q][2], d[q][3]);
    }
    __syncthreads();   // every thread has read parity[x]
    if (tid == 0) A.parity[x] = base ^ (A.k & 1u);
}

template <class S> cudaError_t flow_setup() {
    cudaError_t e = cudaFuncSetAttribute(k_flow<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (e) return e;
    int dev = 0, sms = 0, per = 0, coop = 0;
    if ((e = cudaGetDevice(&dev)) || (e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev)) ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_flow<S>, (int)S::NT, S::SMEM)))
        return e;
    return (coop && (u32)(per * sms) >= S::CTAS) ? cudaSuccess : cudaErrorNotSupported;
}
template <class S> cudaError_t flow_launch(const FlowArgs& A, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(S::CTAS);
    cfg.blockDim = dim3(S::NT);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_flow<S>, A);
}

// The shapes by log2 h: log2 rows, log2 row length, columns per group.  R and C
// put the two phases' units on about as many CTAs as SMs where the size allows
// (128 of each from h = 2^16), with segments of at least 4 digits; from h = 2^18
// the SM count fixes the units (2048 and 4096 elements, 84% of the SMs) and a
// CTA fills its SM with 1024 threads of 64 registers (h = 2^18: 512 threads
// 34.0 us a squaring, 1024 30.4; h = 2^19: 512 68.4, 1024 62.3).  Larger sizes
// are cut to the number of SMs instead (m2_tide.cu).
#define M2_FLOW_SHAPES(X) \
    X(11, 6, 5, 2) X(12, 6, 6, 2) X(13, 6, 7, 2) X(14, 6, 8, 4) X(15, 8, 7, 2) X(16, 8, 8, 2) X(17, 8, 9, 4) X(18, 8, 10, 8) X(19, 8, 11, 16)

}  // namespace

size_t flow_carry_words(int lh) {
#define M2_FLOW_W(LH, LR, LB, C) if (lh == LH) return ((size_t)1 << (LR + LB)) / C;
    M2_FLOW_SHAPES(M2_FLOW_W)
#undef M2_FLOW_W
    return 0;
}
size_t flow_groups(int lh) {
#define M2_FLOW_G(LH, LR, LB, C) if (lh == LH) return ((size_t)1 << LB) / C;
    M2_FLOW_SHAPES(M2_FLOW_G)
#undef M2_FLOW_G
    return 0;
}
cudaError_t flow_setup(int lh, bool gf61) {
#if M2_DUAL
    if (gf61) return m2k_g61::flow_setup(lh, true);
#endif
#define M2_FLOW_S(LH, LR, LB, C) if (lh == LH) return flow_setup<Shape<LR, LB, C>>();
    M2_FLOW_SHAPES(M2_FLOW_S)
#undef M2_FLOW_S
    return cudaErrorNotSupported;
}
cudaError_t launch_flow(int lh, bool gf61, const FlowArgs& A, cudaStream_t s) {
#if M2_DUAL
    if (gf61) return m2k_g61::launch_flow(lh, true, A, s);
#endif
#define M2_FLOW_L(LH, LR, LB, C) if (lh == LH) return flow_launch<Shape<LR, LB, C>>(A, s);
    M2_FLOW_SHAPES(M2_FLOW_L)
#undef M2_FLOW_L
    return cudaErrorNotSupported;
}

}  // namespace M2K_NS
