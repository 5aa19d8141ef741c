// m2_kernels.cuh -- kernel parameter blocks and launch wrappers (host-visible).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace m2k {

// Dual-field twiddle as stored on the device (24 bytes, same as m2::Dual).
struct DTw { unsigned long long a, b; unsigned int c, d; };

enum Mode : int { LL = 0, PRP = 1, PRP3 = 2 };

// Status word written by kernels (0 = ok).
enum Status : int { ST_OK = 0, ST_CARRY_RANGE = 1, ST_NORMALIZE = 2, ST_WAIT_TIMEOUT = 4 };

// A context's words for its host: the status, and the squarings that one-launch
// kernels (m2_flow.cu, m2_tide.cu) were to run but did not start on.
struct StateWords {
    int status;
    int pad;
    unsigned long long owed;
    const unsigned* yield;   // host word, not 0: launches that ask are called off (or null)
};

// One independent test for the whole-iteration-in-one-CTA kernel.
struct SmallTest {
    long long* digits;        // n balanced digits (in/out)
    const unsigned char* w61; // n shifts
    const unsigned char* w31;
    const DTw* tw4;           // radix-4 twiddles of this h
    const DTw* tc;            // centre twiddles of this h
    int* status;
    unsigned int p;
    unsigned int iters;
    int ln;
    int mode;
    int span;                 // carry span (digits normalized after a segment carry)
    int carry_threads;        // threads taking part in the segmented carry (0 = one thread, full normalization)
    int gf61_only;            // 1: the GF(P61) residue alone is the convolution word (no CRT)
    int fuse_middle;          // 1: the last forward level, the centre and the first inverse level in one pass
};

// Plan of the three-pass path for one transform length.
struct LargePlan {
    int ln, L, L1, L2;        // log2 n, log2 h, log2 rows, log2 row length
    unsigned int R, B, C, G;  // rows, row length, columns per CTA, column groups
    int span;
    unsigned int p;
    int mode;
    unsigned int in_turn;      // 1: R = 256 runs the passes of m2_pass.cu at every row length, not the fused column kernel
    unsigned int mid_tickets;  // fused column kernel: 0 = cooperative (CTA index = group), 1 = groups by arrival ticket
    unsigned int gf61;         // 1: the GF(P61^2)-only layout; each word is the signed GF(P61) residue (no CRT)
    unsigned int mid_barrier;  // cooperative fused column kernel: 1 = all groups publish before any goes on
};

struct LargeBufs {
    long long* digits;        // n
    long long* carries;       // R*G segment carries
    ulonglong2* za;           // h GF(P61^2) coordinates
    uint2* zb;                // h GF(P31^2) coordinates
    const unsigned char* w61;
    const unsigned char* w31;
    const DTw* tw4;
    const DTw* tc;
    int* status;
    unsigned int* flags;      // G epoch flags of the fused column kernel, then its 64-bit ticket counter and
    unsigned long long* ticket;   // its 64-bit phase counter (zero-initialised)
    unsigned long long* phase;
    // per element k (digits 2k, 2k+1): x = the two digits' unweighting rotations mod 61 (bytes 0, 1) and
    // mod 31 (bytes 2, 3), y = their widths (bytes 0, 1); read by the quad-shuffle column passes
    const uint2* aux;
};

// Arguments of the one-launch kernel of mid-size transforms (m2_flow.cu).
struct FlowArgs {
    long long* digits;         // n digits of the state; left with no pending carries
    long long* carries;        // pending segment carries of the three-pass kernels, applied and cleared
    ulonglong2* za;            // h tagged GF(P61^2) elements, every tag 1 between launches
    uint2* zb;                 // h tagged GF(P31^2) elements
    const unsigned char* w61;
    const unsigned char* w31;
    const uint2* aux;          // per element: LargeBufs::aux
    const DTw* tw4;
    const DTw* tc;
    unsigned long long* fcar;  // flow_carry_words tagged segment carries
    unsigned long long* arrivals;   // CTAs started, over all launches, and the marks of launches that did not run
    unsigned int* parity;      // flow_groups words: squarings done, modulo 2
    int* status;               // of the context's StateWords
    unsigned int k;            // squarings of this launch (>= 1)
    unsigned short seg;        // digits per pending carry segment
    unsigned short ask;        // 1: the launch looks at StateWords::yield first
    int span;                  // at most 3
    int mode;
};
// and of the one of large transforms (m2_tide.cu)
struct TideArgs {
    FlowArgs f;
    // aux and the weighting rotations of column c of group g, row r at
    // (7 g + c) 1024 + r, and where a CTA leaves a group's digits meanwhile
    const uint2* taux;
    const unsigned int* tshift;
    longlong2* park;
    const DTw* tw8;            // the radix-8 levels' twiddles (launch_twiddles8)
};

constexpr int LARGE_STAGES = 3;
constexpr int STAGE_MID = 3;   // the fused inverse + forward column pass (k_cols_mid_q)

// ---- tables, start states and batch results (m2_tables.cu) ----
struct TestInit {
    unsigned char* w61;
    unsigned char* w31;
    uint2* aux;                // LargeBufs::aux, or null
    long long* digits;         // the start state x0 (a value below 2^(w_0 - 1)), or null
    long long x0;
    unsigned int p;
    int ln;                    // at most 30
};
size_t twiddle_entries(unsigned long long h);   // DTw entries of tw4; tc has h / 2
// The radix-8 levels' tables (m2_tide.cu): w_{8S}^(a br_S(j)) at 7 (S + j) + a - 1
// for S = 8, 1024, 8192 blocks before the step, a = 1 ... 7
size_t twiddle8_entries(unsigned long long h);   // 0 below h = 2^20
cudaError_t launch_twiddles8(DTw* tw8, unsigned int h, cudaStream_t s);
cudaError_t launch_twiddles(DTw* tw4, DTw* tc, unsigned int h, cudaStream_t s);   // h >= 4
cudaError_t launch_test_init(const TestInit& T, cudaStream_t s);
cudaError_t launch_test_init(const TestInit* d_tests, int ntests, cudaStream_t s);
// low 64 bits and verdict of each test's state (n = 2^ln <= 16384 digits)
cudaError_t launch_results(const SmallTest* d_tests, int ntests, int ln, unsigned long long* res64, int* prime, cudaStream_t s);

// ---- one test per CTA, fields in turn, both fields' layout only (m2_duo.cu) ----
bool duo_supported(unsigned int h, int span, int carry_threads);
int duo_threads(unsigned int h);
int duo_ctas_per_sm(unsigned int h);
// one CTA per test, or (d_queue) a persistent grid; iters_override and min_smem as launch_small
cudaError_t launch_duo(const SmallTest* d_tests, int ntests, unsigned int h, unsigned int iters_override, cudaStream_t s,
                       int* d_queue = nullptr, int grid = 0, size_t min_smem = 0);

// Throughput of 32x32->64-bit integer multiplies (mul.wide.u32 / mad.wide.u32)
// on every SM: independent chains, returns products per second.
double measure_wide_mul_rate(int device);

// ---- full carry propagation (m2_carry.cu) ----
struct NormSum;
struct NormArgs {
    const long long* digits;          // n signed digit words
    const long long* carries;         // pending segment carries (n / seg of them) or null
    unsigned long long seg;           // digits per segment (a multiple of 8) when carries != null
    unsigned long long n, p;
    int ln;
    unsigned long long* out;          // n canonical digits
    int* status;                      // |= 2 when the state is outside the propagation's range
    NormSum* block_sum;               // scratch (norm_bind_scratch)
    long long* block_cin;
    unsigned int* flags;              // bit 0: the result was all ones (written as zero); bit 1: a digit >= 8 is nonzero
};
size_t norm_scratch_bytes(unsigned long long n);
void norm_bind_scratch(NormArgs& a, void* scratch);
cudaError_t launch_normalize(const NormArgs& a, cudaStream_t s);
cudaError_t normalize_setup();   // loads its kernels and launch_balance's (see pass_setup)
// canonical digits -> balanced digits with no pending carries; *bad |= 1 when
// an input digit is not canonical (bad may be null)
cudaError_t launch_balance(const unsigned long long* canon, long long* digits, unsigned long long p, int ln,
                           unsigned long long n, unsigned int* bad, cudaStream_t s);

}  // namespace m2k

// The transform kernels are built twice (m2_field.cuh): M2_DUAL = 1 into
// namespace m2k, M2_DUAL = 0 (GF(P61^2) alone) into m2k_g61.  A kernel build
// sees only its own entry points, so that calls inside it resolve to them.
#ifndef M2_DUAL
#define M2_DUAL 1
#endif
#if M2_DUAL
#define M2K_NS m2k
namespace m2k {
#include "m2_launch.inc"
}  // namespace m2k
#else
#define M2K_NS m2k_g61
#endif
namespace m2k_g61 {
using namespace m2k;
#include "m2_launch.inc"
}  // namespace m2k_g61
