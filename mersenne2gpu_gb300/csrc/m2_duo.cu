// m2_duo.cu -- one test per CTA for the shared launches of batches and the
// server (n = 256 ... 16384), the two fields one after the other.
//
// The one-CTA kernel of m2_kernels.cu holds an element's four words and a
// butterfly's twiddles of both fields at once: 106-128 registers, 16 warps an
// SM (8 at n = 16384).  Here a thread runs a butterfly in GF(P61^2), then the
// same one in GF(P31^2): 64 registers, 32 warps an SM.  The transform's middle
// (last forward level, centre square, first inverse level) is one pass over
// mirror blocks, and a radix-4 level waits only for the warps that wrote its
// blocks.  From n = 4096 on the first two levels are radix-8, a butterfly per
// thread (n = 4096 118 -> 111 ns below); at smaller sizes that would halve the
// threads (n = 2048: 53.7 -> 56.4, 1024 27.7 -> 30.1).
//
// What bounds it: the SM's integer pipes (n = 4096: 72% of the cycles, the
// multiplier another 30%, 23 warps an SM).  Measured, ns per test-squaring of a
// full GPU, the one-CTA kernel's best combination -> here:
//   n    256  512   1024  2048  4096  8192  16384
//        7.5  15.3  30.9  63.4  138   287   689
//     -> 6.2  13.0  27.7  53.7  111   229   494
// and us per squaring of a lone test: 5.9 -> 6.6, 6.4 -> 6.8 (n = 256, 512),
// 12.3 -> 10.2, 24.6 -> 21.2, 51.7 -> 36.6, 104 -> 75 (n = 2048 ... 16384).
#include <algorithm>

#include "m2_flow.cuh"

namespace M2K_NS {

namespace {

template <int A_> struct Shape {
    static constexpr int A = A_;
    static constexpr u32 H = 1u << A, NB = H / 4;
    static constexpr bool R8 = A >= 11, NARROW = true, ODD = (A & 1) != 0;   // R8: the first two levels are radix-8
    static constexpr u32 NT = R8 ? H / 8 : NB, NF = NT;
    static constexpr u32 EP = H / NT;                    // consecutive elements of a thread in the row stage
    static constexpr int FIRST = R8 ? 3 : 0;             // radix-4 levels FIRST ... NL - 1 outside the middle
    static constexpr int NL = A / 2 - (ODD ? 0 : 1);
    static constexpr u32 SMEM = 24 * H, FIT = 232448 / (SMEM + 8 * NT + 1040), PER = 1024 / NT < FIT ? 1024 / NT : FIT;   // CTAs of an SM
};

// the radix-8 level's twiddles w_64^(a br_8(j)), at 7 j + a - 1 from here: in the
// part of the radix-4 table that belongs to no level (32 ... 63 blocks)
constexpr u32 TW8_AT = 3 * 32;

// XOR swizzle of the slots (as sw, m2_flow.cuh): also for threads 8 elements apart
__host__ __device__ constexpr u32 swd(u32 e) {
    return e ^ ((e >> 3) & 1u) ^ (((e >> 4) & 1u) * 6u) ^ (((e >> 5) & 1u) * 12u) ^ (((e >> 6) & 1u) << 3);
}

// rotations that unweight digits of shifts s <= 60, s <= 30: by 2^-(s + log2 n + 1)
template <class S> __device__ __forceinline__ u32 unrot61(u32 s) { return min(61u - (S::A + 2) - s, 122u - (S::A + 2) - s); }
template <class S> __device__ __forceinline__ u32 unrot31(u32 s) { return min(31u - (S::A + 2) - s, 62u - (S::A + 2) - s); }

// the levels of a whole transform in one field
template <class S, class X> struct Whole {
    X* z;
    const DTw* tw4;
    const DTw* tc;

    template <class F> __device__ __forceinline__ void each(F&& f) const {
#pragma unroll 1
        for (u32 b = threadIdx.x; b < S::NB; b += S::NT) f(b);
    }
    // radix-8 level l = 0, 1: blocks of H / 8^l
    template <bool FWD> __device__ __forceinline__ void level8(int l) const {
        const u32 M = S::H >> (3 * l), Q = M / 8;
#pragma unroll 1
        for (u32 b = threadIdx.x; b < S::H / 8; b += S::NT) {
            const u32 s0 = swd(b / Q * M + b % Q);
            X x[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) x[m] = z[s0 ^ swd(m * Q)];
            if (!FWD) dit8_adds(x);
            if (l > 0) {
                const DTw* t = tw4 + TW8_AT + 7 * (b / Q);
                if (FWD) twist8(x, t);
                else untwist8(x, t);
            }
            if (FWD) dif8_adds(x);
#pragma unroll
            for (int m = 0; m < 8; ++m) z[s0 ^ swd(m * Q)] = x[m];
        }
    }
    __device__ __forceinline__ void fwd_level(int l) const {
        const u32 M = S::H >> (2 * l), Q = M / 4;
        each([&](u32 b) {
            const u32 s0 = swd(b / Q * M + b % Q);
            X x[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ swd(m * Q)];
            if (l == 0) xdif4_1(x);
            else xdif4(x, ldtri<X>(tw4, (1u << (2 * l)) + b / Q));
#pragma unroll
            for (int m = 0; m < 4; ++m) z[s0 ^ swd(m * Q)] = x[m];
        });
    }
    __device__ __forceinline__ void inv_level(int l) const {
        const u32 M = S::H >> (2 * l), Q = M / 4;
        each([&](u32 b) {
            const u32 s0 = swd(b / Q * M + b % Q);
            X x[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ swd(m * Q)];
            if (l == 0) dit_adds(x);
            else xdit4(x, ldtri<X>(tw4, (1u << (2 * l)) + b / Q));
#pragma unroll
            for (int m = 0; m < 4; ++m) z[s0 ^ swd(m * Q)] = x[m];
        });
    }
    // blocks j and jm hold each other's mirrors (block j >= 2 mirrors
    // 3 2^e - 1 - j, 2^e <= j < 2^(e+1)); item 0 is blocks 0 and 1, their own
    static __device__ __forceinline__ void blocks(u32 item, u32& j, u32& jm) {
        if (item == 0) { j = 0; jm = 1; return; }
        j = item + (1u << (31 - __clz(item)));
        jm = (3u << (31 - __clz(j))) - 1u - j;
    }
    __device__ __forceinline__ void middle() const {
        each([&](u32 b) {
            if (S::ODD) middle2(b);
            else middle4(b);
        });
    }
    // odd log2 h: radix-2 level, centre, inverse, on two blocks of 2 positions
    __device__ __forceinline__ void middle2(u32 b) const {
        u32 j, jm;
        blocks(b, j, jm);
        X cx, cy;
        ldtw(cx, tc, j);
        ldtw(cy, tc, jm);
        const u32 sx = swd(2 * j), sy = swd(2 * jm);
        X x0 = z[sx], x1 = z[sx ^ swd(1)], y0 = z[sy], y1 = z[sy ^ swd(1)];
        const X ux = xmul(x1, cx), uy = xmul(y1, cy);
        x1 = xsub(x0, ux); x0 = xadd(x0, ux);
        y1 = xsub(y0, uy); y0 = xadd(y0, uy);
        // even position of each block with the odd one of the other; item 0:
        // position 0 with itself, 1 with itself, 2 with 3
        const bool own = b == 0;
        X p1 = own ? x0 : y1, q1 = own ? y1 : x1;
        xcentre(x0, p1, own ? xone(cx) : cx);
        xcentre(y0, q1, cy);
        if (own) { y1 = q1; x1 = xsqr(xadd(x1, x1)); }
        else { y1 = p1; x1 = q1; }
        const X dx = xsub(x0, x1), dy = xsub(y0, y1);
        z[sx] = xadd(x0, x1); z[sx ^ swd(1)] = xmulc(dx, cx);
        z[sy] = xadd(y0, y1); z[sy ^ swd(1)] = xmulc(dy, cy);
    }
    // even log2 h: last radix-4 level, centre, inverse; neighbouring lanes hold
    // mirror blocks and swap odd positions
    __device__ __forceinline__ void middle4(u32 b) const {
        static_assert(S::ODD || S::NB % 32 == 0, "whole warps take part");
        const u32 item = b >> 1, s = b & 1u;
        u32 j, jm;
        blocks(item, j, jm);
        if (s) j = jm;
        const Tri<X> t = ldtri<X>(tw4, S::H / 4 + j);
        const u32 s0 = swd(4 * j);
        X x[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ swd(m)];
        xdif4(x, t);
        const bool own = item == 0;              // blocks 0 and 1: their own mirrors
        const int src = (int)(threadIdx.x & 31u) ^ (own ? 0 : 1);
        X y1 = xshfl(x[1], src), y3 = xshfl(x[3], src);
        const X o1 = x[1];
        const bool zero = own && s == 0;         // positions 0 (with itself), 1 (with itself), 2 with 3
        if (zero) { y1 = x[3]; y3 = x[0]; }
        xcentre(x[0], y3, t.r1);
        xcentre(x[2], y1, xtimes_i(t.r1));
        x[1] = xshfl(y1, src);
        x[3] = xshfl(y3, src);
        if (zero) { x[3] = y1; x[1] = xsqr(xadd(o1, o1)); }
        xdit4(x, t);
#pragma unroll
        for (int m = 0; m < 4; ++m) z[s0 ^ swd(m)] = x[m];
    }
};

template <class S> __device__ __forceinline__ void run_duo(const SmallTest& T, u32 iters, X61* za, X31* zb, i64* cx) {
    const u32 t = threadIdx.x;
    longlong2* zd = reinterpret_cast<longlong2*>(za);   // a slot holds its element's two digits between squarings
    const u32 mul = (T.mode == PRP3) ? 3u : 1u;
    const u32 s0 = swd(S::EP * t);
    const Whole<S, X61> ua{za, T.tw4, T.tc};
    const Whole<S, X31> ub{zb, T.tw4, T.tc};
    const longlong2* src = reinterpret_cast<const longlong2*>(T.digits);
#pragma unroll
    for (u32 k = 0; k < S::EP; ++k) zd[s0 ^ swd(k)] = src[S::EP * t + k];
    u32 bad = 0;
    // digit j of ceil(p (j+1) / n) - ceil(p j / n) bits: floor(p / n) and one more
    // where -p j mod n is below p mod n
    const u32 n1 = 2 * S::H - 1, wq = T.p >> (S::A + 1), wr = T.p & n1;
    auto digit_width = [&](u32 j) { return wq + (((0u - T.p * j) & n1) < wr ? 1u : 0u); };
    for (u32 it = 0; it < iters; ++it) {
        // weights
#pragma unroll 1
        for (u32 k = 0; k < S::EP; k += 2) {
            const u32 s61 = __ldg(reinterpret_cast<const u32*>(T.w61) + (S::EP * t + k) / 2);
            const u32 s31 = __ldg(reinterpret_cast<const u32*>(T.w31) + (S::EP * t + k) / 2);
            const u32 p = s0 ^ swd(k), q = s0 ^ swd(k + 1);
            const longlong2 d = zd[p], f = zd[q];
            za[p] = weigh61(d.x, d.y, s61);
            za[q] = weigh61(f.x, f.y, s61 >> 16);
            zb[p] = weigh31(d.x, d.y, s31);
            zb[q] = weigh31(f.x, f.y, s31 >> 16);
        }
        if (S::R8) {
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                __syncthreads();
                ua.template level8<true>(l);
                asm_fence();
                ub.template level8<true>(l);
                asm_fence();
            }
        }
#pragma unroll
        for (int l = S::FIRST; l < S::NL; ++l) {
            if (l == S::FIRST) __syncthreads();
            else sync_group<S>(S::H >> (2 * l), t, 1);
            ua.fwd_level(l);
            asm_fence();
            ub.fwd_level(l);
            asm_fence();
        }
        __syncthreads();
        ua.middle();
        asm_fence();
        ub.middle();
        __syncthreads();
#pragma unroll
        for (int l = S::NL - 1; l >= S::FIRST; --l) {
            if (l < S::NL - 1) sync_group<S>((S::H >> (2 * l)) / 4, t, 1);
            ua.inv_level(l);
            asm_fence();
            ub.inv_level(l);
            asm_fence();
        }
        if (S::R8) {
#pragma unroll
            for (int l = 1; l >= 0; --l) {
                if (l == 0 || S::NL > S::FIRST) __syncthreads();
                ua.template level8<false>(l);
                asm_fence();
                ub.template level8<false>(l);
                asm_fence();
            }
        }
        __syncthreads();
        // unweight, CRT, carry chain of the thread's digits; the carry to the next thread
        i64 c = 0;
#pragma unroll 1
        for (u32 k = 0; k < S::EP; ++k) {
            const u32 e = S::EP * t + k, p = s0 ^ swd(k);
            const u32 s61 = __ldg(reinterpret_cast<const unsigned short*>(T.w61) + e);
            const u32 s31 = __ldg(reinterpret_cast<const unsigned short*>(T.w31) + e);
            const X61 v = za[p];
            const X31 u = zb[p];
            longlong2 d;
            d.x = crt_digit(rotl61(fold61(v.a), unrot61<S>(s61 & 0xffu)), rotl31(u.c, unrot31<S>(s31 & 0xffu)),
                            digit_width(2 * e), mul, (T.mode == LL && e == 0) ? 2 : 0, c, bad, false);
            d.y = crt_digit(rotl61(fold61(v.b), unrot61<S>(s61 >> 8)), rotl31(u.d, unrot31<S>(s31 >> 8)),
                            digit_width(2 * e + 1), mul, 0, c, bad, false);
            zd[p] = d;
        }
        cx[t] = c;
        __syncthreads();
        c = cx[(t - 1) & (S::NT - 1)];
#pragma unroll
        for (u32 k = 0; k < 4; ++k) {
            if (2 * (int)k > T.span) break;
            const u32 e = S::EP * t + k, p = s0 ^ swd(k);
            longlong2 d = zd[p];
            if (2 * (int)k < T.span) d.x = split_balanced64(d.x + c, digit_width(2 * e), c);
            else d.x += c;
            if (2 * (int)k + 1 < T.span) d.y = split_balanced64(d.y + c, digit_width(2 * e + 1), c);
            else if (2 * (int)k + 1 == T.span) d.y += c;
            zd[p] = d;
        }
    }
    if (bad) atomicExch(T.status, ST_CARRY_RANGE);
    longlong2* dst = reinterpret_cast<longlong2*>(T.digits);
#pragma unroll
    for (u32 k = 0; k < S::EP; ++k) dst[S::EP * t + k] = zd[s0 ^ swd(k)];
}

// One CTA per test (queue == nullptr), or a persistent grid whose CTAs take
// test indices from *queue until all `ntests` are done (as k_small).
template <class S>
__global__ void __launch_bounds__(S::NT, S::PER) k_duo(const SmallTest* tests, int ntests, u32 iters_override, int* queue) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ i64 cx[S::NT];
    __shared__ int s_next;
    X61* za = reinterpret_cast<X61*>(smem);
    X31* zb = reinterpret_cast<X31*>(smem + 16ull * S::H);
    if (queue == nullptr) {
        const SmallTest T = tests[blockIdx.x];
        run_duo<S>(T, iters_override ? iters_override : T.iters, za, zb, cx);
        return;
    }
    for (;;) {
        if (threadIdx.x == 0) s_next = atomicAdd(queue, 1);
        __syncthreads();
        const int idx = s_next;
        __syncthreads();
        if (idx >= ntests) break;
        const SmallTest T = tests[idx];
        run_duo<S>(T, iters_override ? iters_override : T.iters, za, zb, cx);
        __syncthreads();
    }
}

// Every size asks for all of the SM's shared memory.  Left to the driver, the
// sizes of one batch get different splits, an SM keeps its split while a CTA is
// on it, and the later size's CTAs crowd onto the SMs that have theirs (502
// tests of n = 512 with 106 of n = 256: 6.95 ms for 2.2 here).
template <class S> cudaError_t prepare() {
    const cudaError_t e = cudaFuncSetAttribute(k_duo<S>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(k_duo<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn_smem_limit((const void*)k_duo<S>));
}
template <class S> int resident() {
    int nb = 0;
    if (prepare<S>() != cudaSuccess || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_duo<S>, (int)S::NT, S::SMEM) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return nb;
}
template <class S> cudaError_t launch(const SmallTest* d_tests, int ntests, u32 iters_override, int* d_queue, int grid, cudaStream_t s, size_t min_smem) {
    const cudaError_t e = prepare<S>();
    if (e != cudaSuccess) return e;
    const size_t sm = std::max<size_t>(S::SMEM, std::min<size_t>(min_smem, (size_t)std::max<int>(dyn_smem_limit((const void*)k_duo<S>), 0)));
    k_duo<S><<<grid, S::NT, sm, s>>>(d_tests, ntests, iters_override, d_queue);
    return cudaGetLastError();
}

#define M2_DUO_SIZES(X) X(7) X(8) X(9) X(10) X(11) X(12) X(13)

}  // namespace

// h = 128 ... 8192: below, a warp has no block for each lane; above, the state
// outgrows an SM's shared memory.  A thread's segment has 8 digits or more:
// carry spans of up to 7 (the tests of these sizes have 2 or 3).
bool duo_supported(unsigned h, int span, int carry_threads) { return h >= 128 && h <= 8192 && span <= 7 && carry_threads > 0; }
int duo_threads(unsigned h) {
#define M2_DUO_N(A) if (h == 1u << A) return (int)Shape<A>::NT;
    M2_DUO_SIZES(M2_DUO_N)
#undef M2_DUO_N
    return 0;
}
int duo_ctas_per_sm(unsigned h) {
#define M2_DUO_R(A) if (h == 1u << A) return resident<Shape<A>>();
    M2_DUO_SIZES(M2_DUO_R)
#undef M2_DUO_R
    return 0;
}
cudaError_t launch_duo(const SmallTest* d_tests, int ntests, unsigned h, unsigned iters_override, cudaStream_t s, int* d_queue, int grid,
                       size_t min_smem) {
#define M2_DUO_L(A) if (h == 1u << A) return launch<Shape<A>>(d_tests, ntests, iters_override, d_queue, d_queue ? grid : ntests, s, min_smem);
    M2_DUO_SIZES(M2_DUO_L)
#undef M2_DUO_L
    return cudaErrorInvalidValue;
}

}  // namespace M2K_NS
