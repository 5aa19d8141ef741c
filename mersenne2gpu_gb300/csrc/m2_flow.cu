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
// of units that are small for an SM.
//
// What bounds it: up to n = 2^16 latency -- the serial chain of butterfly levels
// on a few warps per SM, and three L2 round trips (two hand-overs and the
// carry) -- and from n = 2^17 on the integer pipes of the SMs that have a unit.
// Measured, us per squaring, three-pass launches -> here: n = 2^12 16.2 -> 6.5,
// 2^13 18.5 -> 6.6, 2^14 19.5 -> 7.6, 2^15 21.7 -> 8.2, 2^16 27.5 -> 9.6,
// 2^17 31.9 -> 10.0, 2^18 37.3 -> 15.7, 2^19 44.9 -> 30.4, 2^20 79.6 -> 62.3.
// The three passes paid three launches per squaring, each with cold L1 tables,
// and ran rows on as few as 32 SMs.
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
template <u32 TAG, class X> __device__ __forceinline__ void take4(X (&x)[4], const X* p, u32 stride, Wait& w) {
    u32 it = 0;
    const u32 lanes = __activemask();
    do {
        u32 off = 0;
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = ld_relaxed(p + (u64)m * stride);
#pragma unroll
        for (int m = 0; m < 4; ++m) off |= off_tag<TAG>(x[m]);
        if (__all_sync(lanes, (int)off >= 0)) break;
    } while (__any_sync(lanes, w.again(it)));
#pragma unroll
    for (int m = 0; m < 4; ++m) x[m] = untag(x[m]);
}

// XOR swizzle of a unit's shared-memory slots (16-byte GF(P61^2) slots, 8-byte
// GF(P31^2) slots): the low four index bits take in bits 3-6, so that eight
// (sixteen) consecutive lanes of every access hit distinct 16-byte (8-byte)
// bank groups: butterflies of every stride, rows of 4 or 2 columns.  Linear
// over GF(2): sw(a + b) = sw(a) ^ sw(b) for a and b on disjoint bits.
__host__ __device__ constexpr u32 sw(u32 e) {
    return e ^ ((e >> 3) & 1u) ^ (((e >> 4) & 1u) * 6u) ^ (((e >> 5) & 1u) << 3);
}

template <int LR_, int LB_, int C_> struct Shape {
    static constexpr int LR = LR_, LB = LB_, C = C_;
    static constexpr u32 R = 1u << LR, B = 1u << LB, G = B / C, H = R * B;
    static constexpr u32 UC = R * C, UR = 2 * B;             // elements of a column group and of a row pair
    static constexpr u32 NBC = UC / 4, NBR = UR / 4;         // radix-4 butterflies of a level
    static constexpr u32 NB0 = NBC > NBR ? NBC : NBR;
    static constexpr u32 NF = NB0 < 32 ? 32 : NB0 > 512 ? 512 : NB0;   // threads per field
    static constexpr u32 NT = kDual ? 2 * NF : NF;
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
        constexpr bool EARLY = S::NT <= 512;
        Tri<X> t;
        const bool on = NB % S::NF == 0 || fb < NB;
        if (EARLY && on) tw(fb, t);
        if (group) sync_group<S>(group, fb, bar);
        if (!on) return;
        if (ITERS == 1) {
            X x[4];
            ld(fb, x);
            if (!EARLY) tw(fb, t);
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
    // the forward levels: shared slots in, global out
    __device__ __forceinline__ void cols_fwd(u32 cg) const {
        constexpr int NL = S::LR / 2;
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            const u32 M = S::R >> (2 * l), Q = M / 4;
            level<IC, S::NBC>(l > 0 ? M * S::C : 0, [&](u32 b, Tri<X>& t) { if (l > 0) t = ldtri<X>(tw4, (1u << (2 * l)) + b / S::C / Q); },
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
    // the inverse levels: global in, shared slots out
    __device__ __forceinline__ void cols_inv(u32 cg, Wait& w) const {
        constexpr int NL = S::LR / 2;
#pragma unroll
        for (int l = NL - 1; l >= 0; --l) {
            const u32 M = S::R >> (2 * l), Q = M / 4;
            level<IC, S::NBC>(l == NL - 1 ? S::NF : Q * S::C, [&](u32 b, Tri<X>& t) { if (l > 0) t = ldtri<X>(tw4, (1u << (2 * l)) + b / S::C / Q); },
                  [&](u32 b, X (&x)[4]) {
                      const u32 rho = b / S::C, cc = b % S::C;
                      if (l == NL - 1) {
                          take4<1>(x, g + (u64)(4 * rho) * S::B + cg * S::C + cc, S::B, w);
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
    __device__ __forceinline__ void rows(u32 pi, Wait& w) const {
        constexpr int NL = S::LB / 2;                        // radix-4 levels
        constexpr bool ODD = (S::LB & 1) != 0;
        constexpr int NF4 = ODD ? NL : NL - 1;               // those outside the tail
        u32 t0 = 0, t1 = 1;
        if (pi) {
            const u32 e = 32u - __clz(pi), a = pi - (1u << (e - 1));
            t0 = (1u << e) + a;
            t1 = (2u << e) - 1u - a;
        }
#pragma unroll
        for (int l = 0; l < NF4; ++l) {
            const u32 M = S::B >> (2 * l), Q = M / 4;
            level<IR, S::NBR>(l > 0 ? M : S::NF, [&](u32 b, Tri<X>& t) {
                      const u32 rho = b % (S::B / 4), trow = b / (S::B / 4) ? t1 : t0;
                      t = ldtri<X>(tw4, (S::R + trow) * (1u << (2 * l)) + rho / Q);
                  },
                  [&](u32 b, X (&x)[4]) {
                      const u32 rho = b % (S::B / 4), sl = b / (S::B / 4);
                      if (l == 0) {
                          take4<0>(x, g + (u64)(sl ? t1 : t0) * S::B + rho, Q, w);
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
        sync();
#pragma unroll 1
        for (u32 b = fb; b < S::NBR; b += S::NF) {
            if (ODD) tail2(pi, t0, t1, b);
            else tail4(pi, t0, t1, b);
        }
#pragma unroll
        for (int l = NF4 - 1; l >= 0; --l) {
            const u32 M = S::B >> (2 * l), Q = M / 4;
            level<IR, S::NBR>(l == NF4 - 1 ? S::NF : Q, [&](u32 b, Tri<X>& t) {
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
                          for (int m = 0; m < 4; ++m) st_tagged<1>(p + m * Q, x[m]);
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

template <class S>
__global__ void __launch_bounds__(S::NT, 1) k_flow(FlowArgs A) {
    extern __shared__ __align__(16) unsigned char smem[];
    X61* za = reinterpret_cast<X61*>(smem);
    X31* zb = reinterpret_cast<X31*>(smem + 16ull * S::SLOTS);
    const u32 tid = threadIdx.x, x = blockIdx.x;
    const bool second = kDual && tid >= S::NF;     // the GF(P31^2) half's warps
    const u32 fb = second ? tid - S::NF : tid;
    Unit<S, X61> ua{za, reinterpret_cast<X61*>(A.za), A.tw4, A.tc, fb, 1};
    Unit<S, X31> ub{zb, reinterpret_cast<X31*>(A.zb), A.tw4, A.tc, fb, 8};
    const bool has_cols = S::G == S::CTAS || x < S::G, has_rows = S::R / 2 == S::CTAS || x < S::R / 2;
    Wait w{A.status, false};
    const u32 base = has_cols ? A.parity[x] : 0u;  // squarings handed over so far (bit 0); bit 1 never matches a word's tag

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
        if ((2 * e0[q]) % A.seg == 0) {
            const u32 idx = 2 * e0[q] / A.seg, prev = idx ? idx - 1 : 2 * S::H / A.seg - 1;
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
            if (!second) ua.cols_fwd(x);
            else ub.cols_fwd(x);
        }
        if (!has_cols || !has_rows) __syncthreads();   // this CTA's stores of one tag before its polls for the other
        if (has_rows) {
            if (!second) ua.rows(x, w);
            else ub.rows(x, w);
        }
        if (!has_cols) {
            if (it + 1 == A.k) break;
            continue;
        }
        if (!second) ua.cols_inv(x, w);
        else ub.cols_inv(x, w);
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
// CTA fills its SM with 512 threads per field, 64 registers each (h = 2^18:
// 256 threads per field 34.0 us a squaring, 512 30.4; h = 2^19: 256 68.4, 512
// 62.3).  Larger sizes keep the three-pass kernels: at h = 2^20 a unit of 8192
// elements per SM would take as long as those, which use all 152 SMs.
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
