// m2_tide.cu -- k squarings of one large test (n = 2^21, 2^22) in one
// cooperative launch of one CTA per SM.
//
// The scheme of m2_flow.cu (see there: tagged words hand the data over) with
// the units cut to the number of SMs instead of to powers of two.  The 1024 rows' columns are dealt out in
// groups of 6 or 7 adjacent ones, one group per CTA (two at n = 2^22), so the
// column phase keeps all 152 SMs busy, where groups of 4 leave a third of them
// one group short of the others; the 512 row pairs go round the CTAs in turn.
//
// Seven columns of 1024 elements fill 168 KiB of shared memory, row-major with
// a stride of 7 slots.  In the row stage each of the 1024 threads has one row
// of 12 or 14 digits: CRT and carry chain into the slots, the carry to the next
// group's thread of that row, the carry of the group before into the first
// digits, weights.  With two groups per CTA the second one's inverse half runs
// first and parks its digits in the state's buffer, so that no group waits for
// a carry that its neighbour has not yet begun to make.
//
// The first two levels of the columns, and at n = 2^21 of the rows, are
// radix-8 with a butterfly per thread: 6 twiddle products per element and
// squaring for 7.5 (the columns' first level has none in either form), a
// quarter fewer passes over shared memory and barriers.
//
// What bounds it: the integer pipes (ALU and multiply-add each about 60% busy,
// issue 0.6 a cycle and scheduler), with the row pairs' 3.37 per SM rounded up
// to 4.  Measured, us per squaring, three-pass kernels -> here:
// n = 2^21 128.6 -> 103.4, 2^22 289 -> 233, GF(P61^2) alone at 2^22 204 -> 166
// (134.3, 299.5 and 208 before the arithmetic steps of m2_field.cuh).  On the
// way (n = 2^21): the two fields on separate warps 128.6 (the GF(P31) warps
// finish early and leave half the warps to the rest), both on every warp 117;
// row-stage tables in row order 110; radix-8 columns 107; four row pairs at a
// time instead of two 105.7; radix-8 rows 103.4.  At n = 2^22 radix-8 columns
// took 235 to 233; radix-8 rows there spill and take 241.
#include "m2_flow.cuh"

namespace M2K_NS {

namespace {

template <int LB_, int UNITS_, u32 PAIRS_, bool ROWS8_> struct Shape {
    static constexpr int LR = 10, LB = LB_, C = 7, UNITS = UNITS_;
    static constexpr u32 R = 1u << LR, B = 1u << LB, H = R * B;
    static constexpr u32 NBC = R / 4 * C, NBR = 2 * B / 4;   // radix-4 butterflies of a level
    static constexpr u32 PAIRS = PAIRS_;                     // row pairs at a time
    static constexpr bool ROWS8 = ROWS8_;                    // radix-8 levels in the rows, too
    static constexpr u32 NT = 1024, NF = NT / PAIRS;         // threads of the CTA, of a row pair
    static constexpr u32 SLOTS = 2 * B * PAIRS, SMEM = 24 * SLOTS;   // the row pairs, or a column group
    static constexpr u32 SLOT_R = R * C;
    static constexpr bool EARLY = false;
    static constexpr u32 ROW_TAG = 1;
    static constexpr bool NARROW = PAIRS == 2;               // 15 barriers: 7 per row pair, or one
    static constexpr u32 BARS = NARROW ? 7 : 1;
    static_assert(SLOT_R <= SLOTS, "a column group fits");
    static_assert(!ROWS8 || NF == 2 * B / 8, "a radix-8 butterfly per thread");
    static_assert(NT == R, "a thread per row in the row stage");
};

// the column levels: columns c0 ... c0 + nc - 1 (nc <= 7), slot 7 r + c; every
// thread runs both fields' butterflies threadIdx.x, threadIdx.x + 1024, ...
template <class S, class X> struct Cols {
    X* z;
    X* g;
    const DTw* tw4;
    const DTw* tw8;
    u32 c0, nc;

    // radix-8 level l: blocks of R / 8^l rows
    template <class F> __device__ __forceinline__ void each8(F&& f) const {
        const u32 rho = threadIdx.x / S::C, cc = threadIdx.x - rho * S::C;
        if (rho < S::R / 8 && cc < nc) f(rho, cc);
    }
    __device__ __forceinline__ void fwd_level8(int l) const {
        const u32 M = S::R >> (3 * l), Q = M / 8;
        each8([&](u32 rho, u32 cc) {
            X* s = z + (rho / Q * M + rho % Q) * S::C + cc;
            X x[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) x[m] = s[m * Q * S::C];
            if (l > 0) twist8(x, tw8 + 7 * ((1u << (3 * l)) + rho / Q));
            dif8_adds(x);
#pragma unroll
            for (int m = 0; m < 8; ++m) s[m * Q * S::C] = x[m];
        });
    }
    __device__ __forceinline__ void inv_level8(int l) const {
        const u32 M = S::R >> (3 * l), Q = M / 8;
        each8([&](u32 rho, u32 cc) {
            X* s = z + (rho / Q * M + rho % Q) * S::C + cc;
            X x[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) x[m] = s[m * Q * S::C];
            dit8_adds(x);
            if (l > 0) untwist8(x, tw8 + 7 * ((1u << (3 * l)) + rho / Q));
#pragma unroll
            for (int m = 0; m < 8; ++m) s[m * Q * S::C] = x[m];
        });
    }
    template <class F> __device__ __forceinline__ void each(F&& f) const {
#pragma unroll 1
        for (u32 b = threadIdx.x; b < S::NBC; b += S::NT) {
            const u32 rho = b / S::C, cc = b - rho * S::C;
            if (cc < nc) f(rho, cc);
        }
    }
    __device__ __forceinline__ void fwd_level(int l) const {
        const u32 M = S::R >> (2 * l), Q = M / 4;
        each([&](u32 rho, u32 cc) {
            X* s = z + (rho / Q * M + rho % Q) * S::C + cc;
            X x[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) x[m] = s[m * Q * S::C];
            if (l == 0) xdif4_1(x);
            else xdif4(x, ldtri<X>(tw4, (1u << (2 * l)) + rho / Q));
            if (l < S::LR / 2 - 1) {
#pragma unroll
                for (int m = 0; m < 4; ++m) s[m * Q * S::C] = x[m];
            } else {
                X* p = g + (u64)(4 * rho) * S::B + c0 + cc;
#pragma unroll
                for (int m = 0; m < 4; ++m) st_tagged<0>(p + m * S::B, x[m]);
            }
        });
    }
    __device__ __forceinline__ void inv_level(int l, Wait& w) const {
        const u32 M = S::R >> (2 * l), Q = M / 4;
        each([&](u32 rho, u32 cc) {
            X* s = z + (rho / Q * M + rho % Q) * S::C + cc;
            X x[4];
            if (l == S::LR / 2 - 1) {
                take<1>(x, g + (u64)(4 * rho) * S::B + c0 + cc, S::B, w);
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m) x[m] = s[m * Q * S::C];
            }
            if (l == 0) dit_adds(x);
            else xdit4(x, ldtri<X>(tw4, (1u << (2 * l)) + rho / Q));
#pragma unroll
            for (int m = 0; m < 4; ++m) s[m * Q * S::C] = x[m];
        });
    }
};
template <class S, class... F> __device__ __forceinline__ void cols_fwd(const F&... f) {
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        __syncthreads();
        ((f.fwd_level8(l), asm_fence()), ...);
    }
#pragma unroll
    for (int l = 3; l < S::LR / 2; ++l) {
        __syncthreads();
        ((f.fwd_level(l), asm_fence()), ...);
    }
}
template <class S, class... F> __device__ __forceinline__ void cols_inv(Wait& w, const F&... f) {
#pragma unroll
    for (int l = S::LR / 2 - 1; l >= 3; --l) {
        __syncthreads();
        ((f.inv_level(l, w), asm_fence()), ...);
    }
#pragma unroll
    for (int l = 1; l >= 0; --l) {
        __syncthreads();
        ((f.inv_level8(l), asm_fence()), ...);
    }
}

// a row pair: two radix-8 levels, then the radix-4 levels and the tail of m2_flow.cuh
template <class S, class X> __device__ __forceinline__ void rows_fwd_level8(const Unit<S, X>& u, const DTw* tw8, int l, u32 t0, u32 t1, Wait& w) {
    const u32 M = S::B >> (3 * l), Q = M / 8, rho = u.fb % (S::B / 8), sl = u.fb / (S::B / 8), t = sl ? t1 : t0;
    const u32 s0 = sw(sl * S::B + rho / Q * M + rho % Q);
    X x[8];
    if (l == 0) {
        take<0>(x, u.g + (u64)t * S::B + rho, Q, w);
    } else {
#pragma unroll
        for (int m = 0; m < 8; ++m) x[m] = u.z[s0 ^ sw(m * Q)];
    }
    twist8(x, tw8 + 7 * ((S::R + t) * (1u << (3 * l)) + rho / Q));
    dif8_adds(x);
#pragma unroll
    for (int m = 0; m < 8; ++m) u.z[s0 ^ sw(m * Q)] = x[m];
}
template <class S, class X> __device__ __forceinline__ void rows_inv_level8(const Unit<S, X>& u, const DTw* tw8, int l, u32 t0, u32 t1) {
    const u32 M = S::B >> (3 * l), Q = M / 8, rho = u.fb % (S::B / 8), sl = u.fb / (S::B / 8), t = sl ? t1 : t0;
    const u32 s0 = sw(sl * S::B + rho / Q * M + rho % Q);
    X x[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) x[m] = u.z[s0 ^ sw(m * Q)];
    dit8_adds(x);
    untwist8(x, tw8 + 7 * ((S::R + t) * (1u << (3 * l)) + rho / Q));
    if (l > 0) {
#pragma unroll
        for (int m = 0; m < 8; ++m) u.z[s0 ^ sw(m * Q)] = x[m];
    } else {
        X* p = u.g + (u64)t * S::B + rho;
#pragma unroll
        for (int m = 0; m < 8; ++m) st_tagged<1>(p + m * Q, x[m]);
    }
}
template <class S, class U0, class... U> __device__ __forceinline__ void rows8(u32 pi, const DTw* tw8, Wait& w, const U0& u0, const U&... u) {
    u32 t0, t1;
    row_pair(pi, t0, t1);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        u0.sync();
        rows_fwd_level8(u0, tw8, l, t0, t1, w);
        asm_fence();
        ((rows_fwd_level8(u, tw8, l, t0, t1, w), asm_fence()), ...);
    }
    run_rows_from<S, 3>(pi, t0, t1, w, u0, u...);
#pragma unroll
    for (int l = 1; l >= 0; --l) {
        u0.sync();
        rows_inv_level8(u0, tw8, l, t0, t1);
        asm_fence();
        ((rows_inv_level8(u, tw8, l, t0, t1), asm_fence()), ...);
    }
}

template <class S> __host__ __device__ __forceinline__ u32 first_column(u32 g, u32 groups) { return (u32)((u64)g * S::B / groups); }

// The row stage's tables by group, column and row: a warp's 32 rows read 32
// neighbouring records (in element order they lie B apart, one cache line
// each: 20 of 117 us a squaring at n = 2^21).
template <class S> __global__ void __launch_bounds__(256) k_tide_tables(FlowArgs A, uint2* taux, u32* tshift, u32 groups) {
    const u32 i = blockIdx.x * 256u + threadIdx.x, r = i % S::R, gc = i / S::R, g = gc / S::C, c = gc % S::C;
    if (g >= groups) return;
    const u32 col = first_column<S>(g, groups) + c;
    if (col >= first_column<S>(g + 1, groups)) return;
    const u64 e = (u64)r * S::B + col;
    taux[i] = A.aux[e];
    tshift[i] = A.w61[2 * e] | (A.w61[2 * e + 1] << 8) | (A.w31[2 * e] << 16) | ((u32)A.w31[2 * e + 1] << 24);
}

template <class S>
__global__ void __launch_bounds__(S::NT, 1) k_tide(TideArgs TA) {
    const FlowArgs& A = TA.f;
    extern __shared__ __align__(16) unsigned char smem[];
    X61* za = reinterpret_cast<X61*>(smem);
    X31* zb = reinterpret_cast<X31*>(smem + 16ull * S::SLOTS);
    const u32 tid = threadIdx.x, cta = blockIdx.x, groups = gridDim.x * S::UNITS;
    const u32 part = tid / S::NF;        // each part of the threads takes row pairs of its own
    X61* ga = reinterpret_cast<X61*>(A.za);
    X31* gb = reinterpret_cast<X31*>(A.zb);
    Unit<S, X61> ua{za + part * 2 * S::B, ga, A.tw4, A.tc, tid % S::NF, 1 + S::BARS * part};
    Unit<S, X31> ub{zb + part * 2 * S::B, gb, A.tw4, A.tc, tid % S::NF, 1 + S::BARS * part};
    Wait w{A.status, false};
    if (!all_started(A.arrivals, gridDim.x, A.status, A.k, A.ask)) return;
    const u32 base = A.parity[cta];      // squarings handed over so far (bit 0); bit 1 never matches a word's tag
    const u32 r = tid;                   // this thread's row in the row stage
    const u32 mul = (A.mode == PRP3) ? 3u : 1u;
    longlong2* zd = reinterpret_cast<longlong2*>(za);   // a slot holds its element's two digits between the halves

    auto first = [&](u32 g) { return first_column<S>(g, groups); };
    auto load = [&](u32 g) {             // digits of the state -> slots
        const u32 c0 = first(g), nc = first(g + 1) - c0;
        const longlong2* src = reinterpret_cast<const longlong2*>(A.digits) + ((u64)r * S::B + c0);
        for (u32 c = 0; c < nc; ++c) zd[r * S::C + c] = src[c];
    };
    auto store = [&](u32 g) {
        const u32 c0 = first(g), nc = first(g + 1) - c0;
        longlong2* dst = reinterpret_cast<longlong2*>(A.digits) + ((u64)r * S::B + c0);
        for (u32 c = 0; c < nc; ++c) dst[c] = zd[r * S::C + c];
    };
    // a group's digits between its inverse and its forward half
    longlong2* park = S::UNITS > 1 ? TA.park + (u64)cta * (S::UNITS - 1) * S::SLOT_R : nullptr;
    auto put = [&](u32 v) {
        for (u32 c = 0; c < S::C; ++c) park[((v - 1) * S::C + c) * S::R + r] = zd[r * S::C + c];
    };
    auto get = [&](u32 v) {
        for (u32 c = 0; c < S::C; ++c) zd[r * S::C + c] = park[((v - 1) * S::C + c) * S::R + r];
    };
    // carry of the segment before this row's into its first digits
    auto carry_in = [&](u32 g, u32 par) {
        const unsigned long long* from = g ? A.fcar + (g - 1) * S::R + r : A.fcar + (groups - 1) * S::R + ((r - 1) & (S::R - 1));
        u32 n = 0;
        u64 v;
        do {
            v = ld_relaxed(from);
            if ((((u32)v & 1u) | (base & 2u)) == par) break;
        } while (w.again(n));
        i64 c = (i64)v >> 1;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            longlong2 d = zd[r * S::C + k];
            const u32 wd = __ldg(&TA.taux[(g * S::C + k) * S::R + r].y);
            if (2 * k < A.span) d.x = split_balanced64(d.x + c, wd & 0xffu, c);
            else if (2 * k == A.span) d.x += c;
            if (2 * k + 1 < A.span) d.y = split_balanced64(d.y + c, (wd >> 8) & 0xffu, c);
            else if (2 * k + 1 == A.span) d.y += c;
            zd[r * S::C + k] = d;
        }
    };
    auto forward = [&](u32 g) {          // digits in the slots -> weights, forward levels
        const u32 c0 = first(g), nc = first(g + 1) - c0;
        const u32* at = TA.tshift + g * S::C * S::R + r;
        u32 ahead = __ldg(at);
#pragma unroll 1
        for (u32 c = 0; c < nc; ++c) {
            const u32 s = ahead;
            if (c + 1 < nc) ahead = __ldg(at + (c + 1) * S::R);
            const longlong2 d = zd[r * S::C + c];
            za[r * S::C + c] = weigh61(d.x, d.y, s);
            if (kDual) zb[r * S::C + c] = weigh31(d.x, d.y, s >> 16);
        }
        const Cols<S, X61> fa{za, ga, A.tw4, TA.tw8, c0, nc};
        if (kDual) cols_fwd<S>(fa, Cols<S, X31>{zb, gb, A.tw4, TA.tw8, c0, nc});
        else cols_fwd<S>(fa);
    };
    auto inverse = [&](u32 g, u32 par) { // inverse levels, unweight, CRT, carry chain: digits in the slots
        const u32 c0 = first(g), nc = first(g + 1) - c0;
        const Cols<S, X61> fa{za, ga, A.tw4, TA.tw8, c0, nc};
        if (kDual) cols_inv<S>(w, fa, Cols<S, X31>{zb, gb, A.tw4, TA.tw8, c0, nc});
        else cols_inv<S>(w, fa);
        __syncthreads();
        i64 c = 0;
        u32 bad = 0;
        const uint2* at = TA.taux + g * S::C * S::R + r;
        uint2 ahead = __ldg(at);         // records come from L2: one element ahead
#pragma unroll 1
        for (u32 k = 0; k < nc; ++k) {
            const uint2 t = ahead;
            if (k + 1 < nc) ahead = __ldg(at + (k + 1) * S::R);
            const X61 v = za[r * S::C + k];
            const X31 u = kDual ? zb[r * S::C + k] : X31{0u, 0u};
            const u64 x0 = rotl61(fold61(v.a), t.x & 0xffu), x1 = rotl61(fold61(v.b), (t.x >> 8) & 0xffu);
            const u32 y0 = kDual ? rotl31(u.c, (t.x >> 16) & 0xffu) : 0u, y1 = kDual ? rotl31(u.d, t.x >> 24) : 0u;
            longlong2 d;
            d.x = crt_digit(x0, y0, t.y & 0xffu, mul, (A.mode == LL && r + c0 + k == 0) ? 2 : 0, c, bad, !kDual);
            d.y = crt_digit(x1, y1, (t.y >> 8) & 0xffu, mul, 0, c, bad, !kDual);
            zd[r * S::C + k] = d;
        }
        st_relaxed(A.fcar + g * S::R + r, ((u64)c << 1) | par);
        if (bad) atomicOr(A.status, ST_CARRY_RANGE);
    };

    const u32 g0 = cta * S::UNITS;
#pragma unroll 1
    for (u32 v = 0; v < S::UNITS; ++v) {
        if (v) __syncthreads();          // the slots' last reads are done
        load(g0 + v);
        forward(g0 + v);
    }
    for (u32 it = 0;; ++it) {
        asm volatile("" : "+r"(ua.fb), "+r"(ub.fb));   // addresses and twiddles made anew in every squaring
        __syncthreads();   // the slots' last reads are done
#pragma unroll 1
        for (u32 pi = cta + part * gridDim.x; pi < S::R / 2; pi += S::PAIRS * gridDim.x) {
            if constexpr (S::ROWS8) {
                if (kDual) rows8<S>(pi, TA.tw8, w, ua, ub);
                else rows8<S>(pi, TA.tw8, w, ua);
            } else {
                if (kDual) run_rows<S>(pi, w, ua, ub);
                else run_rows<S>(pi, w, ua);
            }
        }
        const u32 par = (base ^ 1u ^ it) & 1u;
        const bool last = it + 1 == A.k;
        // every group's carries out before any carry in
#pragma unroll 1
        for (int v = S::UNITS - 1; v > 0; --v) {
            inverse(g0 + v, par);
            put(v);
            __syncthreads();
        }
        inverse(g0, par);
#pragma unroll 1
        for (u32 v = 0; v < S::UNITS; ++v) {
            if (v) {
                __syncthreads();
                get(v);
            }
            carry_in(g0 + v, par);
            if (last) store(g0 + v);
            else forward(g0 + v);
        }
        if (last) break;
    }
    __syncthreads();   // every thread has read parity[cta]
    if (tid == 0) A.parity[cta] = base ^ (A.k & 1u);
}

int sm_count() {
    int dev = 0, sms = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
        return 0;
    return sms;
}
template <class S> bool fits() {
    // groups of at most 7 columns, and of at least 2 (4 digits, for the carry span)
    const u32 groups = (u32)sm_count() * S::UNITS;
    int per = 0;
    return groups * 7 >= S::B && groups * 2 <= S::B &&
           cudaFuncSetAttribute(k_tide<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM) == cudaSuccess &&
           cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_tide<S>, (int)S::NT, S::SMEM) == cudaSuccess && per >= 1;
}
template <class S> cudaError_t launch(const TideArgs& A, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)sm_count());
    cfg.blockDim = dim3(S::NT);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_tide<S>, A);
}

template <class S> cudaError_t tables(const TideArgs& A, cudaStream_t s) {
    const u32 groups = (u32)sm_count() * S::UNITS;
    k_tide_tables<S><<<groups * S::C * S::R / 256, 256, 0, s>>>(A.f, const_cast<uint2*>(A.taux), const_cast<u32*>(A.tshift), groups);
    return cudaGetLastError();
}

}  // namespace

// one group of columns per CTA at h = 2^20, two at h = 2^21; row pairs at a
// time (196 KiB of slots) and whether their first levels are radix-8: above
#define M2_TIDE_SHAPES(X) X(20, 10, 1, 4, true) X(21, 11, 2, 2, false)

size_t tide_groups(int lh) {
#define M2_TIDE_G(LH, LB, U, P, R8) if (lh == LH) return (size_t)sm_count() * U;
    M2_TIDE_SHAPES(M2_TIDE_G)
#undef M2_TIDE_G
    return 0;
}
// records of the row stage's tables, and of the digits parked meanwhile
size_t tide_records(int lh) { return tide_groups(lh) * 7 * 1024; }
size_t tide_parked(int lh) {
#define M2_TIDE_P(LH, LB, U, P, R8) if (lh == LH) return (size_t)sm_count() * (U - 1) * 7 * 1024;
    M2_TIDE_SHAPES(M2_TIDE_P)
#undef M2_TIDE_P
    return 0;
}
cudaError_t tide_tables(int lh, const TideArgs& A, cudaStream_t s) {
#define M2_TIDE_T(LH, LB, U, P, R8) if (lh == LH) return tables<Shape<LB, U, P, R8>>(A, s);
    M2_TIDE_SHAPES(M2_TIDE_T)
#undef M2_TIDE_T
    return cudaErrorInvalidValue;
}
bool tide_supported(int lh, int span, bool gf61) {
#if M2_DUAL
    if (gf61) return m2k_g61::tide_supported(lh, span, true);
#endif
    bool ok = false;
#define M2_TIDE_F(LH, LB, U, P, R8) if (lh == LH) ok = fits<Shape<LB, U, P, R8>>();
    M2_TIDE_SHAPES(M2_TIDE_F)
#undef M2_TIDE_F
    cudaGetLastError();
    return ok && span <= 3;
}
cudaError_t launch_tide(int lh, bool gf61, const TideArgs& A, cudaStream_t s) {
#if M2_DUAL
    if (gf61) return m2k_g61::launch_tide(lh, true, A, s);
#endif
#define M2_TIDE_L(LH, LB, U, P, R8) if (lh == LH) return launch<Shape<LB, U, P, R8>>(A, s);
    M2_TIDE_SHAPES(M2_TIDE_L)
#undef M2_TIDE_L
    return cudaErrorInvalidValue;
}

}  // namespace M2K_NS
