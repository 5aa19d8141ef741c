// m2_flow.cuh -- tagged hand-over through global memory and the levels of
// column groups and row pairs on warps of one field (m2_flow.cu, m2_tide.cu).
#pragma once
#include "m2_split.cuh"

namespace M2K_NS {

namespace {

__device__ __forceinline__ X61 xshfl(const X61& v, int src) {
    return X61{__shfl_sync(0xffffffffu, v.a, src), __shfl_sync(0xffffffffu, v.b, src)};
}
__device__ __forceinline__ X31 xshfl(const X31& v, int src) {
    return X31{__shfl_sync(0xffffffffu, v.c, src), __shfl_sync(0xffffffffu, v.d, src)};
}

// ---------------- tagged words in global memory ----------------
__device__ __forceinline__ X61 ld_relaxed(const X61* p) {
    X61 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p));
    return v;
}
__device__ __forceinline__ X31 ld_relaxed(const X31* p) {
    X31 v;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.c), "=r"(v.d) : "l"(p));
    return v;
}
__device__ __forceinline__ u64 ld_relaxed(const u64* p) {
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_relaxed(u64* p, u64 v) { asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v)); }
template <u32 TAG> __device__ __forceinline__ void st_tagged(X61* p, const X61& v) {
    constexpr u64 t = (u64)TAG << 63;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v.a | t), "l"(v.b | t));
}
template <u32 TAG> __device__ __forceinline__ void st_tagged(X31* p, const X31& v) {
    constexpr u32 t = TAG << 31;
    asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(v.c | t), "r"(v.d | t));
}
// sign bit set when a word of v does not carry the tag
template <u32 TAG> __device__ __forceinline__ u32 off_tag(const X61& v) {
    return TAG ? ~((u32)(v.a >> 32) & (u32)(v.b >> 32)) : ((u32)(v.a >> 32) | (u32)(v.b >> 32));
}
template <u32 TAG> __device__ __forceinline__ u32 off_tag(const X31& v) { return TAG ? ~(v.c & v.d) : (v.c | v.d); }
__device__ __forceinline__ X61 untag(const X61& v) { return X61{v.a & ~(1ull << 63), v.b & ~(1ull << 63)}; }
__device__ __forceinline__ X31 untag(const X31& v) { return X31{v.c & P31, v.d & P31}; }

// (the warp's active lanes poll together: diverged loops cost the lone warps of
// the small shapes their branch latency at every poll)
template <u32 TAG, int N, class X> __device__ __forceinline__ void take(X (&x)[N], const X* p, u32 stride, Wait& w) {
    u32 it = 0;
    const u32 lanes = __activemask();
    do {
        u32 off = 0;
#pragma unroll
        for (int m = 0; m < N; ++m) x[m] = ld_relaxed(p + (u64)m * stride);
#pragma unroll
        for (int m = 0; m < N; ++m) off |= off_tag<TAG>(x[m]);
        if (__all_sync(lanes, (int)off >= 0)) break;
    } while (__any_sync(lanes, w.again(it)));
#pragma unroll
    for (int m = 0; m < N; ++m) x[m] = untag(x[m]);
}

// XOR swizzle of a unit's shared-memory slots (16-byte GF(P61^2) slots, 8-byte
// GF(P31^2) slots): the low four index bits take in bits 3-6, so that eight
// (sixteen) consecutive lanes of every access hit distinct 16-byte (8-byte)
// bank groups: butterflies of every stride, rows of 4 or 2 columns.  Linear
// over GF(2): sw(a + b) = sw(a) ^ sw(b) for a and b on disjoint bits.
__host__ __device__ constexpr u32 sw(u32 e) {
    return e ^ ((e >> 3) & 1u) ^ (((e >> 4) & 1u) * 6u) ^ (((e >> 5) & 1u) << 3);
}

// Barrier of the aligned group of at least `d` threads of the field (threads
// fb, NF in all) that this thread is in: a warp, a quarter, half or all of the
// field's threads.  bar: the first of the field's seven barriers.
template <class S> __device__ __forceinline__ void sync_group(u32 d, u32 fb, u32 bar) {
    constexpr u32 NF = S::NF;
    if (S::NARROW && d <= 32) __syncwarp();
    else if (S::NARROW && d <= NF / 4) bar_field<NF / 4>(bar + 3 + fb / (NF / 4));
    else if (S::NARROW && d <= NF / 2) bar_field<NF / 2>(bar + 1 + fb / (NF / 2));
    else bar_field<NF>(bar);
}

// the levels of one CTA's units in one field: each thread runs the butterflies
// fb, fb + NF, ... of a level
template <class S, class X> struct Unit {
    X* z;              // shared slots
    X* g;              // global elements
    const DTw* tw4;
    const DTw* tc;
    u32 fb;            // thread of the field
    u32 bar;           // first barrier of the field's warps

    static constexpr u32 IC = (S::NBC + S::NF - 1) / S::NF, IR = (S::NBR + S::NF - 1) / S::NF;
    __device__ __forceinline__ void sync() const { sync_group<S>(S::NF, fb, bar); }

    // One level.  group: the threads that wrote what this level reads (the
    // butterflies of one block of the level above, which are consecutive): the
    // size of the barrier before it, 0 for none.  tw, ld, st: twiddles, operands and results of a butterfly by
    // its index; op: the level's arithmetic.  With registers to spare the
    // twiddles are fetched before the barrier; with 1024 threads of 64
    // registers the other warps hide them (h = 2^19: 62.3 -> 60.1 us).
    template <u32 ITERS, u32 NB, class TW, class LD, class OP, class ST>
    __device__ __forceinline__ void level(u32 group, TW&& tw, LD&& ld, OP&& op, ST&& st) const {
        constexpr bool EARLY = S::EARLY;
        Tri<X> t;
        const bool on = NB % S::NF == 0 || fb < NB;
        if (EARLY && on) tw(fb, t);
        if (group) sync_group<S>(group, fb, bar);
        if (!on) return;
        if (ITERS == 1 && EARLY) {
            X x[4];
            ld(fb, x);
            op(x, t);
            st(fb, x);
        } else {
#pragma unroll 1
            for (u32 b = fb; b < NB; b += S::NF) {
                X x[4];
                if (!EARLY || b != fb) tw(b, t);
                ld(b, x);
                op(x, t);
                st(b, x);
            }
        }
    }

    // ---- column group cg ----
    // forward level l: shared slots in, the last one's results to global memory
    __device__ __forceinline__ void cols_fwd_level(int l, u32 cg, bool barrier) const {
        constexpr int NL = S::LR / 2;
        {
            const u32 M = S::R >> (2 * l), Q = M / 4;
            level<IC, S::NBC>(l > 0 && barrier ? M * S::C : 0, [&](u32 b, Tri<X>& t) { if (l > 0) t = ldtri<X>(tw4, (1u << (2 * l)) + b / S::C / Q); },
                  [&](u32 b, X (&x)[4]) {
                      const u32 rho = b / S::C, s0 = sw((rho / Q * M + rho % Q) * S::C + b % S::C);
#pragma unroll
                      for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ sw(m * Q * S::C)];
                  },
                  [&](X (&x)[4], const Tri<X>& t) { if (l == 0) xdif4_1(x); else xdif4(x, t); },
                  [&](u32 b, const X (&x)[4]) {
                      const u32 rho = b / S::C, cc = b % S::C;
                      if (l < NL - 1) {
                          const u32 s0 = sw((rho / Q * M + rho % Q) * S::C + cc);
#pragma unroll
                          for (int m = 0; m < 4; ++m) z[s0 ^ sw(m * Q * S::C)] = x[m];
                      } else {
                          X* p = g + (u64)(4 * rho) * S::B + cg * S::C + cc;
#pragma unroll
                          for (int m = 0; m < 4; ++m) st_tagged<0>(p + m * S::B, x[m]);
                      }
                  });
        }
    }
    // inverse level l: shared slots out, the first one's operands from global memory
    __device__ __forceinline__ void cols_inv_level(int l, u32 cg, Wait& w, bool barrier) const {
        constexpr int NL = S::LR / 2;
        {
            const u32 M = S::R >> (2 * l), Q = M / 4;
            level<IC, S::NBC>(!barrier ? 0 : l == NL - 1 ? S::NF : Q * S::C, [&](u32 b, Tri<X>& t) { if (l > 0) t = ldtri<X>(tw4, (1u << (2 * l)) + b / S::C / Q); },
                  [&](u32 b, X (&x)[4]) {
                      const u32 rho = b / S::C, cc = b % S::C;
                      if (l == NL - 1) {
                          take<S::ROW_TAG>(x, g + (u64)(4 * rho) * S::B + cg * S::C + cc, S::B, w);
                      } else {
                          const u32 s0 = sw((rho / Q * M + rho % Q) * S::C + cc);
#pragma unroll
                          for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ sw(m * Q * S::C)];
                      }
                  },
                  [&](X (&x)[4], const Tri<X>& t) { if (l == 0) dit_adds(x); else xdit4(x, t); },
                  [&](u32 b, const X (&x)[4]) {
                      const u32 rho = b / S::C, s0 = sw((rho / Q * M + rho % Q) * S::C + b % S::C);
#pragma unroll
                      for (int m = 0; m < 4; ++m) z[s0 ^ sw(m * Q * S::C)] = x[m];
                  });
        }
    }

    // ---- row pair (t0, t1), slot s B + i for element i of row t_s ----
    static constexpr bool ODD = (S::LB & 1) != 0;
    static constexpr int NF4 = S::LB / 2 - (ODD ? 0 : 1);    // radix-4 levels outside the tail
    // (the first level: its operands from global memory, or written by another kind of level)
    __device__ __forceinline__ void rows_fwd_level(int l, u32 t0, u32 t1, Wait& w, bool barrier, bool first) const {
        {
            const u32 M = S::B >> (2 * l), Q = M / 4;
            level<IR, S::NBR>(!barrier ? 0 : first ? S::NF : M, [&](u32 b, Tri<X>& t) {
                      const u32 rho = b % (S::B / 4), trow = b / (S::B / 4) ? t1 : t0;
                      t = ldtri<X>(tw4, (S::R + trow) * (1u << (2 * l)) + rho / Q);
                  },
                  [&](u32 b, X (&x)[4]) {
                      const u32 rho = b % (S::B / 4), sl = b / (S::B / 4);
                      if (l == 0) {
                          take<0>(x, g + (u64)(sl ? t1 : t0) * S::B + rho, Q, w);
                      } else {
                          const u32 s0 = sw(sl * S::B + rho / Q * M + rho % Q);
#pragma unroll
                          for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ sw(m * Q)];
                      }
                  },
                  [&](X (&x)[4], const Tri<X>& t) { xdif4(x, t); },
                  [&](u32 b, const X (&x)[4]) {
                      const u32 rho = b % (S::B / 4), sl = b / (S::B / 4), s0 = sw(sl * S::B + rho / Q * M + rho % Q);
#pragma unroll
                      for (int m = 0; m < 4; ++m) z[s0 ^ sw(m * Q)] = x[m];
                  });
        }
    }
    __device__ __forceinline__ void rows_tail(u32 pi, u32 t0, u32 t1, bool barrier) const {
        if (barrier) sync();
#pragma unroll 1
        for (u32 b = fb; b < S::NBR; b += S::NF) {
            if (ODD) tail2(pi, t0, t1, b);
            else tail4(pi, t0, t1, b);
        }
    }
    __device__ __forceinline__ void rows_inv_level(int l, u32 t0, u32 t1, bool barrier) const {
        {
            const u32 M = S::B >> (2 * l), Q = M / 4;
            level<IR, S::NBR>(!barrier ? 0 : l == NF4 - 1 ? S::NF : Q, [&](u32 b, Tri<X>& t) {
                      const u32 rho = b % (S::B / 4), trow = b / (S::B / 4) ? t1 : t0;
                      t = ldtri<X>(tw4, (S::R + trow) * (1u << (2 * l)) + rho / Q);
                  },
                  [&](u32 b, X (&x)[4]) {
                      const u32 rho = b % (S::B / 4), sl = b / (S::B / 4), s0 = sw(sl * S::B + rho / Q * M + rho % Q);
#pragma unroll
                      for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ sw(m * Q)];
                  },
                  [&](X (&x)[4], const Tri<X>& t) { xdit4(x, t); },
                  [&](u32 b, const X (&x)[4]) {
                      const u32 rho = b % (S::B / 4), sl = b / (S::B / 4);
                      if (l > 0) {
                          const u32 s0 = sw(sl * S::B + rho / Q * M + rho % Q);
#pragma unroll
                          for (int m = 0; m < 4; ++m) z[s0 ^ sw(m * Q)] = x[m];
                      } else {
                          X* p = g + (u64)(sl ? t1 : t0) * S::B + rho;
#pragma unroll
                          for (int m = 0; m < 4; ++m) st_tagged<S::ROW_TAG>(p + m * Q, x[m]);
                      }
                  });
        }
    }
    // blocks j (row t0) and j' (row t1) of `per` consecutive positions that
    // hold each other's mirrors, by item index: offsets into the pair's 2B
    // slots.  Rows 0 and 1 mirror within themselves: as one run of 2B
    // positions, block j >= 2 mirrors 3 2^e - 1 - j (2^e <= j < 2^(e+1));
    // item 0 there is blocks 0 and 1, each its own mirror.
    static __device__ __forceinline__ void blocks(u32 pi, u32 item, u32 per, u32& j, u32& jm) {
        if (pi) { j = item; jm = S::B / per + (S::B / per - 1 - item); }
        else if (item == 0) { j = 0; jm = 1; }
        else {
            j = item + (1u << (31 - __clz(item)));
            jm = (3u << (31 - __clz(j))) - 1u - j;
        }
    }
    // global block index of the pair's block j
    static __device__ __forceinline__ u32 gblock(u32 t0, u32 t1, u32 per, u32 j) {
        const u32 nb = S::B / per;
        return (j >= nb ? t1 : t0) * nb + (j & (nb - 1));
    }
    // log2 B odd: the radix-2 level, the centre square and the inverse level
    // on two mirror blocks of 2 positions per thread
    __device__ __forceinline__ void tail2(u32 pi, u32 t0, u32 t1, u32 b) const {
        u32 j, jm;
        blocks(pi, b, 2, j, jm);
        X cx, cy;
        ldtw(cx, tc, gblock(t0, t1, 2, j));
        ldtw(cy, tc, gblock(t0, t1, 2, jm));
        const u32 sx = sw(2 * j), sy = sw(2 * jm);
        X x0 = z[sx], x1 = z[sx ^ sw(1)], y0 = z[sy], y1 = z[sy ^ sw(1)];
        const X ux = xmul(x1, cx), uy = xmul(y1, cy);
        x1 = xsub(x0, ux); x0 = xadd(x0, ux);
        y1 = xsub(y0, uy); y0 = xadd(y0, uy);
        // even position of each block with the odd one of the other
        const bool self = pi == 0 && b == 0;   // position 0 with itself, 1 with itself, 2 with 3
        X p1 = y1, q1 = x1;
        X zx = cx;
        if (pi == 0 && self) { p1 = x0; q1 = y1; zx = xone(cx); }
        xcentre(x0, p1, zx);
        xcentre(y0, q1, cy);
        if (pi == 0 && self) { y1 = q1; x1 = xsqr(xadd(x1, x1)); }
        else { y1 = p1; x1 = q1; }
        const X dx = xsub(x0, x1), dy = xsub(y0, y1);
        x0 = xadd(x0, x1); y0 = xadd(y0, y1);
        z[sx] = x0; z[sx ^ sw(1)] = xmulc(dx, cx);
        z[sy] = y0; z[sy ^ sw(1)] = xmulc(dy, cy);
    }
    // log2 B even: the last radix-4 level, the centre square and its inverse
    // level; neighbouring lanes hold mirror blocks and swap odd positions
    __device__ __forceinline__ void tail4(u32 pi, u32 t0, u32 t1, u32 b) const {
        static_assert((S::LB & 1) || S::NBR % 32 == 0, "whole warps take part");
        const u32 item = b >> 1, s = b & 1u;
        u32 j, jm;
        blocks(pi, item, 4, j, jm);
        if (s) j = jm;
        const Tri<X> t = ldtri<X>(tw4, S::H / 4 + gblock(t0, t1, 4, j));
        const u32 s0 = sw(4 * j);
        X x[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = z[s0 ^ sw(m)];
        xdif4(x, t);
        const bool own = pi == 0 && item == 0;   // blocks 0 and 1: their own mirrors
        const int src = own ? (int)(threadIdx.x & 31u) : (int)((threadIdx.x & 31u) ^ 1u);
        X y1 = xshfl(x[1], src), y3 = xshfl(x[3], src);
        const X o1 = x[1];
        const bool zero = own && s == 0;         // positions 0 (with itself), 1 (with itself), 2 with 3
        if (pi == 0 && zero) { y1 = x[3]; y3 = x[0]; }
        xcentre(x[0], y3, t.r1);
        xcentre(x[2], y1, xtimes_i(t.r1));
        x[1] = xshfl(y1, src);
        x[3] = xshfl(y3, src);
        if (pi == 0 && zero) { x[3] = y1; x[1] = xsqr(xadd(o1, o1)); }
        xdit4(x, t);
#pragma unroll
        for (int m = 0; m < 4; ++m) z[s0 ^ sw(m)] = x[m];
    }
};

__device__ __forceinline__ int asm_fence() { asm volatile("" ::: "memory"); return 0; }
// A unit's levels in the fields of `u`: one field (each on warps of its own),
// or both in turn on the same warps between two barriers.
template <class S, class... U> __device__ __forceinline__ void run_cols_fwd(u32 cg, const U&... u) {
#pragma unroll
    for (int l = 0; l < S::LR / 2; ++l) {
        bool barrier = true;
        ((u.cols_fwd_level(l, cg, barrier), barrier = false, asm_fence()), ...);
    }
}
template <class S, class... U> __device__ __forceinline__ void run_cols_inv(u32 cg, Wait& w, const U&... u) {
#pragma unroll
    for (int l = S::LR / 2 - 1; l >= 0; --l) {
        bool barrier = true;
        ((u.cols_inv_level(l, cg, w, barrier), barrier = false, asm_fence()), ...);
    }
}
// rows of pair pi
__device__ __forceinline__ void row_pair(u32 pi, u32& t0, u32& t1) {
    t0 = 0; t1 = 1;
    if (pi) {
        const u32 e = 32u - __clz(pi), a = pi - (1u << (e - 1));
        t0 = (1u << e) + a;
        t1 = (2u << e) - 1u - a;
    }
}
// a pair's levels from radix-4 level FIRST on and back
template <class S, int FIRST, class... U> __device__ __forceinline__ void run_rows_from(u32 pi, u32 t0, u32 t1, Wait& w, const U&... u) {
    constexpr int NF4 = S::LB / 2 - ((S::LB & 1) ? 0 : 1);
#pragma unroll
    for (int l = FIRST; l < NF4; ++l) {
        bool barrier = true;
        ((u.rows_fwd_level(l, t0, t1, w, barrier, l == FIRST), barrier = false, asm_fence()), ...);
    }
    {
        bool barrier = true;
        ((u.rows_tail(pi, t0, t1, barrier), barrier = false, asm_fence()), ...);
    }
#pragma unroll
    for (int l = NF4 - 1; l >= FIRST; --l) {
        bool barrier = true;
        ((u.rows_inv_level(l, t0, t1, barrier), barrier = false, asm_fence()), ...);
    }
}
template <class S, class... U> __device__ __forceinline__ void run_rows(u32 pi, Wait& w, const U&... u) {
    u32 t0, t1;
    row_pair(pi, t0, t1);
    run_rows_from<S, 0>(pi, t0, t1, w, u...);
}

}  // namespace

}  // namespace M2K_NS
