// m2_pass.cu -- passes of the three-pass kernels with the two fields one after
// the other: row pairs of 2 x 64 to 2 x 512 elements, groups of 4 columns of 64 rows.
//
// The levels are those of m2_flow.cuh, between plain (untagged) arrays: one
// radix-4 butterfly per thread and level, 64 registers, so that CTAs of 32 to
// 256 threads fill an SM with 32 warps, where the generic kernels ran 256
// threads for 32 to 256 butterflies of a row pair and 512 for 64 of a column
// group, and held both fields at once.
//
// What bounds it: the integer pipes when many tests share the GPU (the server),
// a chain of levels and three launches when a test is alone.  Measured, us a
// squaring, the kernels before (generic up to n = 2^18, quad-shuffle with a
// fused column pass above) -> here, a test alone and 8 in the server (4 at 2^20):
//   n      2^13       2^14       2^15       2^16       2^17       2^18       2^19       2^20
//   alone  18 -> 13.6 19 -> 14.3 21 -> 15.2 27 -> 18.4 31 -> 20.6 36 -> 22.8 44 -> 36.6 79 -> 66.6
//   shared            (16 of 2^15: 3.7 -> 2.1, of 2^16: 7.0 -> 3.3)  9.9 -> 6.6 19.3 -> 11.4 25.9 -> 23.6 58.4 -> 52.4
// Row passes alone gave about a quarter of it; the rest are the column passes.
#include "m2_flow.cuh"

namespace M2K_NS {

namespace {

template <int LR_, int LB_> struct Shape {
    static constexpr int LR = LR_, LB = LB_;
    static constexpr u32 R = 1u << LR, B = 1u << LB, H = R * B, C = 4;
    static constexpr u32 NBR = 2 * B / 4, NBC = NBR, NF = NBR, NT = NF;
    static constexpr bool NARROW = true, EARLY = false;
    static constexpr u32 ROW_TAG = 0, SMEM = 24 * 2 * B;
};

template <class S> __global__ void __launch_bounds__(S::NT, 1024 / S::NT) k_pair(LargeBufs bf) {
    extern __shared__ __align__(16) unsigned char smem[];
    Wait w{bf.status, false};
    const Unit<S, X61> ua{reinterpret_cast<X61*>(smem), reinterpret_cast<X61*>(bf.za), bf.tw4, bf.tc, threadIdx.x, 1};
    if (!kDual) {
        run_rows<S>(blockIdx.x, w, ua);
        return;
    }
    const Unit<S, X31> ub{reinterpret_cast<X31*>(smem + 16 * 2 * S::B), reinterpret_cast<X31*>(bf.zb), bf.tw4, bf.tc, threadIdx.x, 1};
    run_rows<S>(blockIdx.x, w, ua, ub);
}

// rotations that unweight digits of shifts s <= 60, s <= 30: by 2^-(s + ln + 1), ln <= 22
__device__ __forceinline__ u32 unrot61(u32 s, u32 ln) { const u32 t = s + ln + 1u; return min(61u - t, 122u - t); }
__device__ __forceinline__ u32 unrot31(u32 s, u32 ln) { const u32 t = s + ln + 1u; return min(31u - t, 62u - t); }

// columns 4 g ... 4 g + 3: the segment before's carry into a row's 8 digits,
// weights, forward levels
template <class S> __global__ void __launch_bounds__(S::NTC, 1024 / S::NTC) k_col4_fwd(LargePlan P, LargeBufs bf) {
    extern __shared__ __align__(16) unsigned char smem[];
    X61* za = reinterpret_cast<X61*>(smem);
    X31* zb = reinterpret_cast<X31*>(smem + 16 * S::R * S::C);
    const u32 t = threadIdx.x, g = blockIdx.x, s = t * P.G + g;
    i64 c = bf.carries[s ? s - 1 : S::R * P.G - 1];
    const u32 e0 = t * S::B + g * S::C;
#pragma unroll
    for (u32 k = 0; k < S::C; ++k) {
        longlong2 d = reinterpret_cast<const longlong2*>(bf.digits)[e0 + k];
        const u32 j = 2 * (e0 + k);
        if (2 * (int)k < P.span) d.x = split_balanced64(d.x + c, width_of(P.p, P.ln, j), c);
        else if (2 * (int)k == P.span) d.x += c;
        if (2 * (int)k + 1 < P.span) d.y = split_balanced64(d.y + c, width_of(P.p, P.ln, j + 1), c);
        else if (2 * (int)k + 1 == P.span) d.y += c;
        const u32 z = sw(S::C * t + k);
        za[z] = weigh61(d.x, d.y, reinterpret_cast<const unsigned short*>(bf.w61)[e0 + k]);
        if (kDual) zb[z] = weigh31(d.x, d.y, reinterpret_cast<const unsigned short*>(bf.w31)[e0 + k]);
    }
    __syncthreads();
    const Unit<S, X61> ua{za, reinterpret_cast<X61*>(bf.za), bf.tw4, bf.tc, t, 1};
    const Unit<S, X31> ub{zb, reinterpret_cast<X31*>(bf.zb), bf.tw4, bf.tc, t, 1};
    if (kDual) run_cols_fwd<S>(g, ua, ub);
    else run_cols_fwd<S>(g, ua);
}
// inverse levels, unweight, CRT, carry over a row's 8 digits
template <class S> __global__ void __launch_bounds__(S::NTC, 1024 / S::NTC) k_col4_inv(LargePlan P, LargeBufs bf) {
    extern __shared__ __align__(16) unsigned char smem[];
    X61* za = reinterpret_cast<X61*>(smem);
    X31* zb = reinterpret_cast<X31*>(smem + 16 * S::R * S::C);
    const u32 t = threadIdx.x, g = blockIdx.x;
    Wait w{bf.status, false};
    const Unit<S, X61> ua{za, reinterpret_cast<X61*>(bf.za), bf.tw4, bf.tc, t, 1};
    const Unit<S, X31> ub{zb, reinterpret_cast<X31*>(bf.zb), bf.tw4, bf.tc, t, 1};
    if (kDual) run_cols_inv<S>(g, w, ua, ub);
    else run_cols_inv<S>(g, w, ua);
    __syncthreads();
    const u32 mul = (P.mode == PRP3) ? 3u : 1u, e0 = t * S::B + g * S::C, ln = (u32)P.ln;
    i64 c = 0;
    u32 bad = 0;
#pragma unroll 1
    for (u32 k = 0; k < S::C; ++k) {
        const u32 e = e0 + k, j = 2 * e, z = sw(S::C * t + k);
        const u32 s61 = reinterpret_cast<const unsigned short*>(bf.w61)[e];
        const u32 s31 = kDual ? reinterpret_cast<const unsigned short*>(bf.w31)[e] : 0u;
        const X61 v = za[z];
        const X31 u = kDual ? zb[z] : X31{0u, 0u};
        const u64 x0 = rotl61(fold61(v.a), unrot61(s61 & 0xffu, ln)), x1 = rotl61(fold61(v.b), unrot61(s61 >> 8, ln));
        const u32 y0 = kDual ? rotl31(u.c, unrot31(s31 & 0xffu, ln)) : 0u, y1 = kDual ? rotl31(u.d, unrot31(s31 >> 8, ln)) : 0u;
        longlong2 d;
        d.x = crt_digit(x0, y0, width_of(P.p, P.ln, j), mul, (P.mode == LL && e == 0) ? 2 : 0, c, bad, !kDual);
        d.y = crt_digit(x1, y1, width_of(P.p, P.ln, j + 1), mul, 0, c, bad, !kDual);
        reinterpret_cast<longlong2*>(bf.digits)[e] = d;
    }
    if (bad) atomicExch(bf.status, ST_CARRY_RANGE);
    bf.carries[(u64)t * P.G + g] = c;
}
template <int LR_, int LB_> struct ColShape {
    static constexpr int LR = LR_, LB = LB_;
    static constexpr u32 R = 1u << LR, B = 1u << LB, H = R * B, C = 4;
    static constexpr u32 NBC = R * C / 4, NBR = NBC, NF = NBC, NT = NF, NTC = R;   // a butterfly, and a row, per thread
    static constexpr bool NARROW = true, EARLY = false;
    static constexpr u32 ROW_TAG = 0, SMEM = 24 * R * C;
};

#define M2_COL4_SHAPES(X) X(6, 6) X(6, 7) X(6, 8) X(6, 9) X(8, 8) X(8, 9) X(8, 10) X(8, 11)
#define M2_PAIR_SHAPES(X) X(6, 6) X(6, 7) X(6, 8) X(6, 9) X(8, 8) X(8, 9) X(8, 10) X(8, 11)

}  // namespace

cudaError_t pass_setup(const LargePlan& P) {
#if M2_DUAL
    if (P.gf61) return m2k_g61::pass_setup(P);
#endif
    cudaFuncAttributes at;
    cudaError_t e = cudaSuccess;
    if (pair_supported(P)) {
#define M2_PAIR_A(LR, LB) if (P.R == 1u << LR && P.B == 1u << LB) e = cudaFuncGetAttributes(&at, k_pair<Shape<LR, LB>>);
        M2_PAIR_SHAPES(M2_PAIR_A)
#undef M2_PAIR_A
    }
    if (col4_supported(P)) {
#define M2_COL4_A(LR, LB)                                                                        \
    if (P.R == 1u << LR && P.B == 1u << LB) {                                                    \
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, k_col4_fwd<ColShape<LR, LB>>);      \
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, k_col4_inv<ColShape<LR, LB>>);      \
    }
        M2_COL4_SHAPES(M2_COL4_A)
#undef M2_COL4_A
    }
    return e;
}

// rows of 1024 and 2048 elements where the plan asks for them
bool pair_supported(const LargePlan& P) {
    if (P.B >= 1024u && !P.in_turn) return false;
#define M2_PAIR_S(LR, LB) if (P.R == 1u << LR && P.B == 1u << LB) return true;
    M2_PAIR_SHAPES(M2_PAIR_S)
#undef M2_PAIR_S
    return false;
}
cudaError_t launch_pair(const LargePlan& P, const LargeBufs& b, cudaStream_t s) {
#define M2_PAIR_L(LR, LB)                                             \
    if (P.R == 1u << LR && P.B == 1u << LB) {                         \
        using S = Shape<LR, LB>;                                      \
        cudaFuncSetAttribute(k_pair<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM); \
        k_pair<S><<<S::R / 2, S::NT, S::SMEM, s>>>(b);                \
        return cudaGetLastError();                                    \
    }
    M2_PAIR_SHAPES(M2_PAIR_L)
#undef M2_PAIR_L
    return cudaErrorInvalidValue;
}

// (a segment of 8 digits takes a carry span of up to 7)
bool col4_supported(const LargePlan& P) {
    if (P.C != 4u || P.span >= 8) return false;
#define M2_COL4_S(LR, LB) if (P.R == 1u << LR && P.B == 1u << LB) return true;
    M2_COL4_SHAPES(M2_COL4_S)
#undef M2_COL4_S
    return false;
}
cudaError_t launch_col4(const LargePlan& P, const LargeBufs& b, bool inverse, cudaStream_t s) {
#define M2_COL4_L(LR, LB)                                                          \
    if (P.R == 1u << LR && P.B == 1u << LB) {                                      \
        using S = ColShape<LR, LB>;                                                \
        if (inverse) k_col4_inv<S><<<P.G, S::NTC, S::SMEM, s>>>(P, b);             \
        else k_col4_fwd<S><<<P.G, S::NTC, S::SMEM, s>>>(P, b);                     \
        return cudaGetLastError();                                                 \
    }
    M2_COL4_SHAPES(M2_COL4_L)
#undef M2_COL4_L
    return cudaErrorInvalidValue;
}

}  // namespace M2K_NS
