// m2_tables.cu -- what a test needs before its first squaring, built on the
// device: twiddle tables of a transform size, and per test the IBDWT shifts,
// the unweighting records and the start state; and the batch's results,
// canonicalised on the device.
//
// These are O(n) loops that the host ran before (2-60 ms per context at n =
// 2^18 ... 2^22, 0.5 s for the first context of n = 2^22's tables, 26 ms of a
// batch of 1024 tests); here they are a few microseconds of a kernel, bound by
// its launch.
#include "m2_field.cuh"
#include "m2_host.hpp"
#include "m2_kernels.cuh"

using namespace m2d;

namespace m2k {

namespace {

__device__ __forceinline__ E dpow(E x, u64 e) {
    E r{1, 0, 1, 0};
    while (e) {
        if (e & 1) r = emul(r, x);
        x = esqr(x);
        e >>= 1;
    }
    return r;
}
__device__ __forceinline__ u32 brev(u32 i, int bits) { return bits ? (__brev(i) >> (32 - bits)) : 0u; }
// tables hold coordinates in [0, P61] / [0, P31] (products leave up to P61 + 8)
__device__ __forceinline__ void put_tw(DTw* t, u32 i, const E& v) { t[i] = DTw{fold61(v.a), fold61(v.b), v.c, v.d}; }

// Twiddle tables for the in-place decimation-in-frequency transform of length
// h with per-block twiddles (natural order in, bit-reversed out):
//   tw4[3*(S+j) + a-1] = r^a, r = w_{4S}^{br_S(j)}, for every radix-4 step with
//                        S blocks before the step (S = 1, 4, 16, ...)
//   tw4[96 + 7*j + a-1] = w_64^(a br_8(j)), j < 8, a = 1 ... 7: the radix-8 step
//                        with 8 blocks before it (m2_duo.cu), for h >= 2048
//   tc[j]              = w_h^{br_{h/2}(j)}, j < h/2: the centre twiddle of
//                        position 2j; also the radix-2 step's twiddle when
//                        log2 h is odd.
__global__ void __launch_bounds__(256) k_twiddles(DTw* tw4, DTw* tc, u32 h, int lh, E wh) {
    for (u32 t = blockIdx.x * blockDim.x + threadIdx.x; t < h / 2; t += gridDim.x * blockDim.x) {
        put_tw(tc, t, dpow(wh, brev(t, lh - 1)));
        // radix-4 step S owns entries S..2S-1; t in [S, 2S) for exactly one power of two S
        if (t == 0) continue;
        const int sb = 31 - __clz(t);
        const u32 S = 1u << sb;
        if (sb == 3 && h >= 2048u) {
            const E r = dpow(wh, (u64)(h / 64u) * brev(t - S, 3));
            E q = r;
            for (u32 a = 0; a < 7; ++a) {
                put_tw(tw4, 96u + 7u * (t - S) + a, q);
                q = emul(q, r);
            }
        }
        if ((sb & 1) == 0 && 4u * S <= h) {
            const E r = dpow(wh, (u64)(h / (4u * S)) * brev(t - S, sb));
            const E r2 = esqr(r), r3 = emul(r2, r);
            put_tw(tw4, 3u * t, r); put_tw(tw4, 3u * t + 1, r2); put_tw(tw4, 3u * t + 2, r3);
        }
    }
}

__global__ void __launch_bounds__(256) k_twiddles8(DTw* tw8, u32 h, E wh) {
    const u32 t = blockIdx.x * 256u + threadIdx.x;   // S + j
    if (t < 8 || t >= 16384) return;
    const int sb = 31 - __clz(t);
    if (sb != 3 && sb != 10 && sb != 13) return;
    const E r = dpow(wh, (u64)(h >> (sb + 3)) * brev(t - (1u << sb), sb));
    E q = r;
    for (u32 a = 0; a < 7; ++a) {
        put_tw(tw8, 7u * t + a, q);
        q = emul(q, r);
    }
}

// w61/w31[j] = n^-1 (n - p j mod n) mod 61 / 31 (shift 0 for j = 0); aux: the
// rotations by 2^-(s + ln + 1) that unweight an element's two digits, and the
// digits' widths; digits: the small start value x0
__device__ __forceinline__ void init_element(const TestInit& T, u32 k) {
    const u32 n = 1u << T.ln;
    const u32 lr61 = (u32)((1ull << (60 - T.ln)) % 61), lr31 = (u32)((1ull << (30 - T.ln)) % 31);
    u32 s61[2], s31[2], u61[2], u31[2];
#pragma unroll
    for (u32 c = 0; c < 2; ++c) {
        const u32 j = 2 * k + c, r = (u32)((u64)T.p * j) & (n - 1);
        s61[c] = j ? m2::weight_shift(lr61, n - r, 61u) : 0u;
        s31[c] = j ? m2::weight_shift(lr31, n - r, 31u) : 0u;
        const u32 a = (s61[c] + (u32)T.ln + 1u) % 61u, b = (s31[c] + (u32)T.ln + 1u) % 31u;
        u61[c] = a ? 61u - a : 0u;
        u31[c] = b ? 31u - b : 0u;
    }
    reinterpret_cast<uchar2*>(T.w61)[k] = make_uchar2((unsigned char)s61[0], (unsigned char)s61[1]);
    reinterpret_cast<uchar2*>(T.w31)[k] = make_uchar2((unsigned char)s31[0], (unsigned char)s31[1]);
    if (T.aux) T.aux[k] = make_uint2(u61[0] | (u61[1] << 8) | (u31[0] << 16) | (u31[1] << 24),
                                     width_of(T.p, T.ln, 2 * k) | (width_of(T.p, T.ln, 2 * k + 1) << 8));
    if (T.digits) reinterpret_cast<longlong2*>(T.digits)[k] = make_longlong2(k == 0 ? T.x0 : 0, 0);
}
__global__ void __launch_bounds__(256) k_init_one(TestInit T) {
    const u32 k = blockIdx.x * 256u + threadIdx.x;
    if (k < (1u << (T.ln - 1))) init_element(T, k);
}
__global__ void __launch_bounds__(256) k_init_batch(const TestInit* tests) {
    const TestInit T = tests[blockIdx.x];
    for (u32 k = threadIdx.x; k < (1u << (T.ln - 1)); k += 256u) init_element(T, k);
}

// One CTA per finished test: the exact carry propagation of its signed digits
// by one thread over shared memory (as k_norm_tiny; at n = 4096 about 50 us,
// all tests of a bucket at once), then the low 64 bits and the verdict.
__global__ void __launch_bounds__(128) k_results(const SmallTest* tests, u64* res64, int* prime) {
    extern __shared__ i64 d[];
    const SmallTest T = tests[blockIdx.x];
    const u32 n = 1u << T.ln, p = T.p;
    for (u32 j = threadIdx.x; j < n; j += blockDim.x) d[j] = T.digits[j];
    __syncthreads();
    if (threadIdx.x == 0) {
        i64 c = 0;
        for (int pass = 0; pass < 66; ++pass) {
            for (u32 j = 0; j < n && (pass == 0 || c != 0); ++j) {
                const u32 w = width_of(p, T.ln, j);
                const i64 v = d[j] + c;
                d[j] = w ? (i64)((u64)v & ((1ull << w) - 1)) : 0;
                c = w ? v >> w : v;
            }
            if (c == 0) break;
        }
        if (c != 0) atomicExch(T.status, ST_NORMALIZE);
    }
    __syncthreads();
    // all ones is M_p: zero
    bool ones = true;
    for (u32 j = threadIdx.x; j < n; j += blockDim.x) ones = ones && (u64)d[j] == (1ull << width_of(p, T.ln, j)) - 1;
    ones = __syncthreads_and(ones);
    u64 want = T.mode == LL ? 0 : (T.mode == PRP ? 9 : 3);
    if (p < 64) want %= (1ull << p) - 1;
    bool same = true;
    for (u32 j = threadIdx.x; j < n; j += blockDim.x) {
        const u32 w = width_of(p, T.ln, j);
        const u64 pos = j ? (((u64)p * j - 1) >> T.ln) + 1 : 0;
        const u64 digit = pos < 64 ? (want >> pos) & ((1ull << w) - 1) : 0;
        same = same && (ones ? 0 : (u64)d[j]) == digit;
    }
    same = __syncthreads_and(same);
    if (threadIdx.x == 0) {
        u64 r = 0;
        for (u32 j = 0; j < n && !ones; ++j) {
            const u64 pos = j ? (((u64)p * j - 1) >> T.ln) + 1 : 0;
            if (pos >= 64) break;
            r |= (u64)d[j] << pos;
        }
        res64[blockIdx.x] = r;
        prime[blockIdx.x] = same;
    }
}

}  // namespace

size_t twiddle_entries(u64 h) {
    u64 smax = 0;
    for (u64 S = 1; 4 * S <= h; S *= 4) smax = S;
    return smax ? 3 * 2 * smax : 3;
}
cudaError_t launch_twiddles(DTw* tw4, DTw* tc, unsigned h, cudaStream_t s) {
    const m2::Dual w = m2::root_of_unity(h);
    int lh = 0;
    while ((1u << lh) < h) ++lh;
    const unsigned g = (h / 2 + 255) / 256;
    k_twiddles<<<g < 4096 ? g : 4096, 256, 0, s>>>(tw4, tc, h, lh, E{w.a, w.b, w.c, w.d});
    return cudaGetLastError();
}
size_t twiddle8_entries(unsigned long long h) { return h >= (1ull << 20) ? 7 * 16384 : 0; }
cudaError_t launch_twiddles8(DTw* tw8, unsigned h, cudaStream_t s) {
    const m2::Dual w = m2::root_of_unity(h);
    k_twiddles8<<<64, 256, 0, s>>>(tw8, h, E{w.a, w.b, w.c, w.d});
    return cudaGetLastError();
}
cudaError_t launch_test_init(const TestInit& T, cudaStream_t s) {
    k_init_one<<<(unsigned)(((1ull << T.ln) / 2 + 255) / 256), 256, 0, s>>>(T);
    return cudaGetLastError();
}
cudaError_t launch_test_init(const TestInit* d_tests, int ntests, cudaStream_t s) {
    k_init_batch<<<ntests, 256, 0, s>>>(d_tests);
    return cudaGetLastError();
}
cudaError_t launch_results(const SmallTest* d_tests, int ntests, int ln, u64* res64, int* prime, cudaStream_t s) {
    const size_t sm = sizeof(i64) << ln;
    const cudaError_t e = cudaFuncSetAttribute(k_results, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    if (e) return e;
    k_results<<<ntests, 128, sm, s>>>(d_tests, res64, prime);
    return cudaGetLastError();
}

}  // namespace m2k
