// m2_api.cu -- the C ABI of include/m2gpu.h on top of the kernels.
#include "../../include/m2gpu.h"
#include "m2_host.hpp"
#include "m2_board.hpp"
#include "m2_internal.hpp"
#include "m2_kernels.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <stdexcept>
#include <tuple>
#include <vector>
#include <chrono>
#include <deque>
#include <thread>
#include <tuple>

using m2::i64;
using m2::u32;
using m2::u64;

namespace {

// ---------------- device twiddle cache (one table set per device and h) ----------------
struct TwTables {
    m2k::DTw* tw4 = nullptr;
    m2k::DTw* tw8 = nullptr;
    m2k::DTw* tc = nullptr;
    size_t bytes = 0;
};
std::mutex g_tw_mu;
std::map<std::pair<int, u64>, TwTables> g_tw;

cudaMemPool_t ctx_pool(int device);

// Tables of a new transform size come from the stream-ordered pool and are
// built on a stream of their own, so making them waits for nothing else running
// on the device (a cudaMalloc may synchronise the whole device).  Kept until
// the process ends.
int get_twiddles(int device, u64 h, TwTables& out) {
    std::lock_guard<std::mutex> lk(g_tw_mu);
    auto it = g_tw.find({device, h});
    if (it != g_tw.end()) { out = it->second; return M2_OK; }
    TwTables t;
    const size_t b4 = m2k::twiddle_entries(h) * sizeof(m2k::DTw), bc = std::max<u64>(h / 2, 1) * sizeof(m2k::DTw);
    cudaMemPool_t mp = ctx_pool(device);
    cudaStream_t s = nullptr;
    if (!mp || cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) { cudaGetLastError(); return M2_ECUDA; }
    cudaError_t e = cudaMallocFromPoolAsync((void**)&t.tw4, b4, mp, s);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync((void**)&t.tc, bc, mp, s);
    const size_t b8 = m2k::twiddle8_entries(h) * sizeof(m2k::DTw);
    if (e == cudaSuccess && b8) e = cudaMallocFromPoolAsync((void**)&t.tw8, b8, mp, s);
    if (e == cudaSuccess) e = m2k::launch_twiddles(t.tw4, t.tc, (unsigned)h, s);
    if (e == cudaSuccess && b8) e = m2k::launch_twiddles8(t.tw8, (unsigned)h, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? M2_ENOMEM : M2_ECUDA;
    }
    t.bytes = b4 + bc + b8;
    g_tw[{device, h}] = t;
    out = t;
    return M2_OK;
}

// ---------------- context memory: one stream-ordered pool per device ----------------
// Contexts allocate and free on their own stream (cudaMallocFromPoolAsync /
// cudaFreeAsync), so creating or destroying one never waits for work that other
// contexts have in flight: the serving engine retires tests while others run.
// The pool keeps freed blocks for reuse (release threshold: unlimited).
std::mutex g_pool_mu;
std::map<int, cudaMemPool_t> g_pool;

cudaMemPool_t ctx_pool(int device) {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pool.find(device);
    if (it != g_pool.end()) return it->second;
    cudaMemPoolProps pp{};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.location.type = cudaMemLocationTypeDevice;
    pp.location.id = device;
    cudaMemPool_t mp = nullptr;
    if (cudaMemPoolCreate(&mp, &pp) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    uint64_t keep = ~uint64_t(0);
    cudaMemPoolSetAttribute(mp, cudaMemPoolAttrReleaseThreshold, &keep);
    g_pool[device] = mp;
    return mp;
}

thread_local char g_last_error[256] = "";

// records where a CUDA call failed (readable through m2_last_error) and maps the code
int fail_cuda(const char* where, cudaError_t e) {
    std::snprintf(g_last_error, sizeof(g_last_error), "%s: %s", where, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? M2_ENOMEM : M2_ECUDA;
}

// Digits that the host keeps the layout of: enough for 64 bits and for small
// values wherever digits have a bit at all (n > 64 has q >= 10).
constexpr u64 HEAD = 72;

u32 total_iters_for(u32 p, int mode) {
    if (mode == M2_MODE_LL) return p >= 2 ? p - 2 : 0;
    if (mode == M2_MODE_PRP3) return p - 1;
    return p;
}

// Carry threads of the one-CTA path: a power of two (threads >> shift at most),
// each owning n/Tc >= span+1 digits; 0 selects the single-thread full
// normalization (tiny exponents).
int small_carry_threads(const m2::Layout& L, int span, int threads, int shift = 0) {
    if (L.q < 4) return 0;
    u64 tc = (u64)(threads >> shift);
    if (tc < 1) tc = 1;
    while (tc > 1 && L.n / tc < (u64)span + 1) tc >>= 1;
    if (L.n / tc < (u64)span + 1) return 0;
    return (int)tc;
}

}  // namespace

struct m2_ctx {
    m2::Layout L;
    int mode = M2_MODE_PRP;
    int path = M2_PATH_SMALL;
    u32 iteration = 0;
    int device = 0;
    m2_opts opts{};            // as passed to m2_create, stream cleared
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int span = 0;
    uint64_t bytes = 0;
    // tables
    unsigned char* d_w61 = nullptr;
    unsigned char* d_w31 = nullptr;
    TwTables tw;
    m2k::StateWords* d_words = nullptr;
    unsigned* yield = nullptr; // host word that calls its queued one-launch kernels off
    int* d_status = nullptr;   // d_words->status
    long long* d_digits = nullptr;
    // small path
    m2k::SmallTest* d_test = nullptr;
    m2k::SmallTest h_test{};   // host copy of the descriptor (the serving engine batches these)
    int threads = 0;
    int carry_threads = 0;
    bool lane = false;         // squarings run in the one-element-per-thread kernel (m2_lane.cu)
    // large path
    m2k::LargePlan plan{};
    m2k::LargeBufs bufs{};
    long long* d_carries = nullptr;
    ulonglong2* d_za = nullptr;
    uint2* d_zb = nullptr;
    unsigned* d_flags = nullptr;
    uint2* d_aux = nullptr;    // per-element unweighting rotations and digit widths (m2k::LargeBufs::aux)
    bool fused = false;        // inverse and next forward column pass as one cooperative launch
    bool gf61 = false;         // GF(P61^2)-only transform (M2_FIELDS_GF61)
    bool flow = false;         // squarings run in a one-launch kernel (m2_flow.cu)
    bool tide = false;         // the one of large sizes (m2_tide.cu)
    size_t flow_bytes = 0;     // of d_flow
    bool cluster = false;      // squarings run in one thread-block cluster (m2_cluster.cu)
    bool stall = false;        // its next launch waits for a carry that never comes (m2_test_stall_fused)
    bool staged = false;       // a three-pass stage ran since: pending carries, untagged elements
    bool untagged = false;     // three-pass kernels wrote the elements last
    m2k::FlowArgs fargs{};
    char* d_flow = nullptr;    // its tagged carries, arrival counter and parity words
    uint2* d_taux = nullptr;   // the large sizes' row-stage tables and parked digits
    uint32_t* d_tshift = nullptr;
    longlong2* d_park = nullptr;
    // contexts whose kernels wait for each other: the plan of passes that do not
    m2k::LargePlan free_plan{};
    // GRAPH_ITERS[i] iterations of the three-pass path captured once and replayed, by plan and by free_plan
    cudaGraphExec_t graph[2][2] = {};
    bool graph_failed = false;
    void* d_slab = nullptr;    // the allocation that holds the buffers above
    std::shared_ptr<m2b::Run> run;   // its work in flight, as other contexts see it
    bool may_owe = false;      // a launch that may be called off was enqueued since the last settle
    // canonical digits and carry-propagation scratch (allocated on first read, in d_read)
    void* d_read = nullptr;
    unsigned long long* d_canon = nullptr;
    void* d_norm = nullptr;
};

namespace {

// One allocation for a set of buffers (256-byte aligned parts).  An allocation
// from the stream-ordered pool costs about 5 us per stream that has used the
// pool (it looks for blocks freed on each), so a context of ten buffers made
// beside 60 others took 2 ms when it asked for each.
struct Slab {
    struct Part { void** p; size_t bytes; };
    std::vector<Part> parts;
    template <class T> void add(T** p, size_t bytes) { parts.push_back(Part{(void**)p, bytes}); }
    int alloc(m2_ctx* c, void** base) {
        // (recorded by a capture, the memory would be the graph's, not the context's)
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(c->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return fail_cuda("allocation", cudaErrorStreamCaptureUnsupported);
        }
        cudaMemPool_t mp = ctx_pool(c->device);
        if (!mp) return M2_ECUDA;
        size_t total = 0;
        for (const Part& q : parts) total += (q.bytes + 255) & ~size_t(255);
        if (cudaMallocFromPoolAsync(base, total, mp, c->stream) != cudaSuccess) { cudaGetLastError(); *base = nullptr; return M2_ENOMEM; }
        char* at = static_cast<char*>(*base);
        for (const Part& q : parts) {
            *q.p = at;
            at += (q.bytes + 255) & ~size_t(255);
            c->bytes += q.bytes;
        }
        return M2_OK;
    }
};

// canonical digits and the carry propagation's scratch, on the first read
int canon_alloc(m2_ctx* c) {
    if (c->d_canon) return M2_OK;
    Slab m;
    m.add(&c->d_canon, c->L.n * sizeof(u64));
    m.add(&c->d_norm, m2k::norm_scratch_bytes(c->L.n));
    return m.alloc(c, &c->d_read);
}

// the fused column kernel's G epoch flags followed by its 64-bit ticket and
// phase counters (G is even, so the counters are 8-byte aligned)
size_t flags_bytes(const m2k::LargePlan& P) { return sizeof(unsigned) * ((size_t)P.G + 4); }


// Iterations of the three-pass path per graph replay, long and short.  With the
// fused column pass a replay of k squarings is 2k + 1 kernels (the forward
// column pass opens it, the inverse one closes it), so the long graph spends
// less on those two passes per squaring.
constexpr uint32_t GRAPH_ITERS[2] = {500, 50};

// k squarings by the three-pass kernels; free: by those of them that wait for nothing
cudaError_t launch_passes(m2_ctx* c, uint32_t k, bool free) {
    return m2k::launch_large_run(free ? c->free_plan : c->plan, c->bufs, k, c->fused && !free, c->stream);
}

// Captures GRAPH_ITERS[i] iterations on the context's stream into an executable
// graph (once); replays cost one launch instead of 2 or 3 per iteration.  Not done
// while the caller is capturing the stream itself, or if capture is refused
// (the legacy default stream): launches are then issued one by one.
bool ensure_graph(m2_ctx* c, int i, bool free) {
    cudaGraphExec_t& exec = c->graph[free][i];
    if (exec) return true;
    if (c->graph_failed) return false;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;
    }
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        c->graph_failed = true;
        return false;
    }
    cudaError_t e = cudaSuccess;
    e = launch_passes(c, GRAPH_ITERS[i], free);
    const cudaError_t ee = cudaStreamEndCapture(c->stream, &g);
    if (e == cudaSuccess && ee == cudaSuccess && g && cudaGraphInstantiate(&exec, g, 0) == cudaSuccess) {
        cudaGraphDestroy(g);
        return true;
    }
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    exec = nullptr;
    c->graph_failed = true;
    return false;
}

// Squarings per launch of the one-launch kernel: long enough that a launch's
// start is nothing (58 ms at n = 2^20), short enough that other contexts'
// launches get their turn; and by passes between two looks at what is in flight.
constexpr uint32_t FLOW_ITERS = 1000;
constexpr uint32_t TIDE_ITERS = 250;
constexpr uint32_t FREE_ITERS = 1000;

m2k::TideArgs tide_args(const m2_ctx* c) { return m2k::TideArgs{c->fargs, c->d_taux, c->d_tshift, c->d_park, c->tw.tw8}; }

// the one-launch kernel's tags as every launch expects them: all element tags
// 1, carries of parity 0
cudaError_t flow_reset(m2_ctx* c) {
    cudaError_t e = cudaMemsetAsync(c->d_za, 0xff, sizeof(ulonglong2) * c->L.h, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->d_zb, 0xff, sizeof(uint2) * c->L.h, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->d_flow, 0, c->flow_bytes, c->stream);
    c->untagged = false;
    return e;
}

// what a new state needs beside its digits: no pending carries, epoch flags
// and tags as at creation (a good status and nothing owed are clear_words')
cudaError_t reset_sync_words(m2_ctx* c) {
    cudaError_t e = cudaSuccess;
    if (c->path == M2_PATH_LARGE) e = cudaMemsetAsync(c->d_carries, 0, sizeof(i64) * (size_t)c->plan.R * c->plan.G, c->stream);
    if (e == cudaSuccess && c->d_flags) e = cudaMemsetAsync(c->d_flags, 0, flags_bytes(c->plan), c->stream);
    if (e == cudaSuccess && c->flow) e = flow_reset(c);
    if (e == cudaSuccess) c->staged = false;
    return e;
}

cudaError_t clear_words(m2_ctx* c) { return cudaMemsetAsync(c->d_words, 0, offsetof(m2k::StateWords, yield), c->stream); }

// Words of pinned host memory that call queued launches off, one per one-launch
// context: 64 bytes apart, in pages kept for the process (a launch of a context
// that is gone may still look at its word).
std::mutex g_yield_mu;
std::vector<unsigned*> g_yield;
unsigned* yield_word() {
    std::lock_guard<std::mutex> lk(g_yield_mu);
    if (g_yield.empty()) {
        unsigned* page = nullptr;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // another thread may be capturing
        cudaThreadExchangeStreamCaptureMode(&mode);
        const cudaError_t e = cudaHostAlloc((void**)&page, 4096, cudaHostAllocPortable | cudaHostAllocMapped);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) { cudaGetLastError(); return nullptr; }
        for (int i = 0; i < 64; ++i) g_yield.push_back(page + 16 * i);
    }
    unsigned* w = g_yield.back();
    g_yield.pop_back();
    *w = 0;
    return w;
}

// waits for the context's stream and reads its words
int read_words(m2_ctx* c, m2k::StateWords& w) {
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e == cudaSuccess) e = cudaMemcpy(&w, c->d_words, sizeof(w), cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? M2_OK : M2_ECUDA;
}
int status_code(int st) { return (st & m2k::ST_WAIT_TIMEOUT) ? M2_ETIMEOUT : st ? M2_ESTATE : M2_OK; }

int cuda_err(cudaError_t e) { return e == cudaSuccess ? M2_OK : (e == cudaErrorMemoryAllocation ? M2_ENOMEM : M2_ECUDA); }

int upload_state(m2_ctx* c, const m2::Layout& L, const std::vector<u64>& canon) {
    std::vector<i64> bal = m2::balanced_digits(L, canon);
    cudaError_t e = cudaMemcpyAsync(c->d_digits, bal.data(), bal.size() * sizeof(i64), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = reset_sync_words(c);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    return cuda_err(e);
}

// Full carry propagation of the context's state on its stream (m2_carry.cu):
// canonical digits land in d_canon, the summary flags in the scratch.
int device_canonical(m2_ctx* c, m2k::NormArgs& a) {
    int rc;
    if ((rc = canon_alloc(c))) return rc;
    a = m2k::NormArgs{};
    a.digits = c->d_digits;
    a.carries = (c->path == M2_PATH_LARGE) ? c->d_carries : nullptr;
    a.seg = (c->path == M2_PATH_LARGE) ? 2ull * c->plan.C : 0;
    a.n = c->L.n; a.p = c->L.p; a.ln = c->L.ln;
    a.out = c->d_canon;
    a.status = c->d_status;
    m2k::norm_bind_scratch(a, c->d_norm);
    const cudaError_t e = m2k::launch_normalize(a, c->stream);
    return e == cudaSuccess ? M2_OK : fail_cuda("carry propagation launch", e);
}

}  // namespace

namespace m2i {
// Plan of the three-pass path: rows 4^floor(log2 h / 4), row length h / rows,
// C columns per CTA (carry_pairs when it is a power of two in [4, 16], else 4,
// widened until a segment of 2C digits exceeds the carry span).
bool plan_large(const m2::Layout& L, int span, uint32_t carry_pairs, m2k::LargePlan& P) {
    const int Lh = L.ln - 1;
    if (Lh < 6) return false;
    int L1 = 2 * (Lh / 4);
    if (L1 < 2) L1 = 2;
    const int L2 = Lh - L1;
    P.ln = L.ln; P.L = Lh; P.L1 = L1; P.L2 = L2;
    P.R = 1u << L1; P.B = 1u << L2;
    P.span = span; P.p = L.p;
    // columns per CTA: 4 (the quad-shuffle column kernels' shape for R = 256
    // and 1024, and more CTAs for the small grids of the other mid-size plans)
    uint32_t C = 4;
    if (carry_pairs >= 4 && carry_pairs <= 16 && (carry_pairs & (carry_pairs - 1)) == 0) C = carry_pairs;
    while (2 * C < (uint32_t)span + 1 && C < 16) C <<= 1;
    if (2 * C < (uint32_t)span + 1 || C > P.B) return false;
    P.C = C; P.G = P.B / C;
    // a row pair and a column group must each fit one CTA's shared memory
    // (227 KiB on this GPU): rows of up to 4096 elements, n <= 2^23 digits
    // (p <= 285212671 with both fields, 150994943 with GF(P61^2) alone)
    constexpr uint64_t kSmem = 227ull * 1024;
    if (24ull * 2 * P.B > kSmem || 24ull * P.C * P.R > kSmem) return false;
    return true;
}

const m2::Layout& layout(const m2_ctx* c) { return c->L; }
m2_opts creation_opts(const m2_ctx* c) { return c->opts; }
cudaStream_t stream(const m2_ctx* c) { return c->stream; }

int canonical(m2_ctx* c, const unsigned long long** out) {
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    m2k::NormArgs a;
    const int rc = device_canonical(c, a);
    if (!rc) *out = c->d_canon;
    return rc;
}

int raw_state(m2_ctx* c, long long** digits) {
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    cudaError_t e = cudaSuccess;
    if (c->path == M2_PATH_LARGE) e = cudaMemsetAsync(c->d_carries, 0, sizeof(i64) * (size_t)c->plan.R * c->plan.G, c->stream);
    if (e != cudaSuccess) return fail_cuda("state reset", e);
    *digits = c->d_digits;
    return M2_OK;
}

int canon_buffer(m2_ctx* c, unsigned long long** buf) {
    int rc;
    if ((rc = canon_alloc(c))) return rc;
    *buf = c->d_canon;
    return M2_OK;
}

int load_canon(m2_ctx* c, uint32_t iteration) {
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    cudaError_t e = m2k::launch_balance(c->d_canon, c->d_digits, c->L.p, c->L.ln, c->L.n, nullptr, c->stream);
    if (e == cudaSuccess) e = reset_sync_words(c);
    if (e == cudaSuccess) e = clear_words(c);
    if (e != cudaSuccess) return fail_cuda("state load", e);
    c->iteration = iteration;
    return M2_OK;
}
}  // namespace m2i

namespace {

// the context's squarings run in a kernel that loops over them itself: one CTA
// or cluster, or one cooperative launch of many CTAs
bool own_kernel(const m2_ctx* c) { return c->path == M2_PATH_SMALL || c->cluster || c->flow; }
const char* own_kernel_name(const m2_ctx* c) {
    return c->cluster ? "k_cluster" : c->lane ? "k_lane" : c->tide ? "k_tide" : c->flow ? "k_flow" : "k_small";
}
uint32_t iters_per_launch(const m2_ctx* c) { return c->tide ? TIDE_ITERS : c->flow ? FLOW_ITERS : ~0u; }

// (ask: the launches look first whether they are called off)
cudaError_t launch_own(m2_ctx* c, uint32_t k, bool ask) {
    cudaError_t e = cudaSuccess;
    c->fargs.ask = ask;
    const unsigned h = (unsigned)c->L.h;
    const int lh = c->L.ln - 1;
    for (uint32_t left = k, now; left > 0 && e == cudaSuccess; left -= now) {
        now = std::min(left, iters_per_launch(c));
        c->fargs.k = now;
        if (c->cluster) {
            e = m2k::launch_cluster(c->d_test, lh, now, c->stall, c->gf61, c->stream);
            c->stall = false;
        } else if (c->lane) {
            e = m2k::launch_lane(c->d_test, 1, h, now, c->stream, c->gf61);
        } else if (c->tide) {
            e = m2k::launch_tide(lh, c->gf61, tide_args(c), c->stream);
        } else if (c->flow) {
            e = m2k::launch_flow(lh, c->gf61, c->fargs, c->stream);
        } else {
            e = m2k::launch_small(c->d_test, 1, h, c->threads, now, c->stream, c->h_test.fuse_middle != 0, c->gf61);
        }
    }
    return e;
}

// After three-pass kernels: the one-launch kernel of mid sizes applies pending
// carries itself and wants its tags back; the others start from digits with
// none.
int unstage(m2_ctx* c) {
    if (!c->staged) return M2_OK;
    cudaError_t e = cudaSuccess;
    if (c->flow && !c->tide) {
        e = flow_reset(c);
    } else {
        m2k::NormArgs a;
        const int rc = device_canonical(c, a);
        if (rc) return rc;
        e = m2k::launch_balance(c->d_canon, c->d_digits, c->L.p, c->L.ln, c->L.n, nullptr, c->stream);
        if (e == cudaSuccess) e = reset_sync_words(c);
    }
    if (e != cudaSuccess) return fail_cuda("state after three-pass kernels", e);
    c->staged = false;
    return M2_OK;
}

// k squarings by the three-pass kernels; free: by those of them that wait for nothing
int run_passes(m2_ctx* c, uint64_t k, bool free) {
    bool ready[2];
    for (int i = 0; i < 2; ++i)
        ready[i] = k >= GRAPH_ITERS[i] && (i == 0 || k % GRAPH_ITERS[0] >= GRAPH_ITERS[1] || !ready[0]) && ensure_graph(c, i, free);
    cudaError_t e = cudaSuccess;
    c->untagged = true;
    if (c->flow) c->staged = true;
    for (int i = 0; i < 2; ++i)
        if (ready[i])
            for (; k >= GRAPH_ITERS[i] && e == cudaSuccess; k -= GRAPH_ITERS[i]) e = cudaGraphLaunch(c->graph[free][i], c->stream);
    if (k > 0 && e == cudaSuccess) e = launch_passes(c, (uint32_t)k, free);
    return e == cudaSuccess ? M2_OK : fail_cuda("three-pass launch", e);
}

m2b::Kind alone(const m2_ctx* c) { return c->flow ? m2b::ONE : c->fused ? m2b::FUSED : m2b::FREE; }

// k squarings on the context's stream, by the kernels of its size (at most
// `most`) or by those that what else is in flight on the device calls for
// (m2_board.hpp).  A one-launch context is left as its own kernel leaves it:
// graphs that its caller captured may run that next.
int advance(m2_ctx* c, uint32_t k, m2b::Kind most) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        // recorded for the caller to replay: the kernels of a context alone
        cudaGetLastError();
        const bool staged = c->staged;
        int rc = unstage(c);
        c->staged = staged;   // the state's, which changes when the graph is replayed
        if (rc) return rc;
        const cudaError_t e = own_kernel(c) ? launch_own(c, k, false) : launch_passes(c, k, false);
        return e == cudaSuccess ? M2_OK : fail_cuda("m2_iterate launch", e);
    }
    m2b::Board& board = m2b::Board::of(c->device);
    m2b::Kind kind = board.begin(*c->run, most);
    bool ask = c->tide;   // the queued launches of a long call; every one of those that take the whole GPU
    int rc = M2_OK;
    for (uint32_t left = k, now; left > 0 && !rc; left -= now) {
        if (left != k) kind = board.again(*c->run, most);
        if (c->flow && kind == m2b::FREE) {
            now = std::min(left, FREE_ITERS);
            rc = run_passes(c, now, true);
        } else if (own_kernel(c)) {
            now = std::min(left, iters_per_launch(c));
            if ((rc = unstage(c))) break;
            const cudaError_t e = launch_own(c, now, ask);
            if (e != cudaSuccess) rc = fail_cuda("m2_iterate launch", e);
            c->may_owe |= ask && c->flow;
            ask = true;
        } else {
            now = left;
            rc = run_passes(c, now, kind == m2b::FREE && c->fused);
        }
    }
    if (!rc && c->flow) rc = unstage(c);
    const cudaError_t e = board.end(*c->run);
    return rc ? rc : e == cudaSuccess ? M2_OK : fail_cuda("end of run", e);
}

// Waits for the context's work, runs the squarings of launches that were called
// off, and returns the state's code; *more (may be null): there were any.
int settle(m2_ctx* c, bool* more = nullptr) {
    if (more) *more = false;
    for (uint64_t owed = 0;;) {
        m2k::StateWords w{};
        int rc = read_words(c, w);
        if (rc) return rc;
        if ((rc = status_code(w.status))) return rc;
        owed += w.owed;
        if (owed == 0) {
            c->may_owe = false;
            return M2_OK;
        }
        if (more) *more = true;
        if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
        const cudaError_t e = cudaMemsetAsync(&c->d_words->owed, 0, sizeof(w.owed), c->stream);
        if (e != cudaSuccess) return fail_cuda("state words", e);
        // in parts, each by what is in flight then; the part after a launch that
        // was called off in kernels that always start
        const uint32_t now = (uint32_t)std::min<uint64_t>(owed, w.owed ? FREE_ITERS : iters_per_launch(c));
        if ((rc = advance(c, now, w.owed ? m2b::FREE : alone(c)))) return rc;
        owed -= now;
    }
}

// Reads of the state: `enqueue` puts canonicalisation and copies on the
// context's stream, again if squarings were still owed at their end.
template <class F> int read_settled(m2_ctx* c, F&& enqueue) {
    for (bool more = true; more;) {
        int rc = enqueue();
        if (!rc) rc = settle(c, &more);
        if (rc) return rc;
    }
    return M2_OK;
}

// the first digits (enough for 64 bits) and the summary flags of the canonical state
int read_head(m2_ctx* c, std::vector<u64>& head, unsigned& flags) {
    return read_settled(c, [&] {
        m2k::NormArgs a;
        const int rc = device_canonical(c, a);
        if (rc) return rc;
        head.assign(std::min<u64>(c->L.n, HEAD), 0);
        cudaError_t e = m2i::read_back(head.data(), c->d_canon, head.size() * sizeof(u64), c->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&flags, a.flags, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream);
        return e == cudaSuccess ? M2_OK : fail_cuda("digits read", e);
    });
}

}  // namespace

namespace m2i {
int settle(m2_ctx* c) { return c->may_owe ? ::settle(c) : M2_OK; }
int iterate_unowed(m2_ctx* c, uint32_t k) {
    if (!c->tide) return m2_iterate(c, k);
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    const int rc = run_passes(c, k, true);
    if (!rc) c->iteration += k;
    return rc;
}
void share_turns(m2_ctx* a, m2_ctx* b) { m2b::Board::of(a->device).group(*a->run, *b->run, a); }
}  // namespace m2i

extern "C" {

const char* m2_last_error(void) { return g_last_error; }

const char* m2_strerror(int code) {
    switch (code) {
        case M2_OK: return "ok";
        case M2_EINVAL: return "invalid argument";
        case M2_ENOMEM: return "out of device memory";
        case M2_ECUDA: return "CUDA runtime error";
        case M2_ETIMEOUT: return "device wait timed out";
        case M2_ESTATE: return "device reported an out-of-range carry";
        case M2_EUNSUPPORTED: return "unsupported exponent or option";
        case M2_ECHECK: return "error check failed; state reset to the last verified one";
        default: return "unknown error";
    }
}

int m2_layout(uint32_t p, int* ln, uint64_t* n, uint8_t* widths) { return m2_layout_fields(p, M2_FIELDS_DUAL, ln, n, widths); }

int m2_layout_fields(uint32_t p, int fields, int* ln, uint64_t* n, uint8_t* widths) {
    if (p < 3 || (fields != M2_FIELDS_DUAL && fields != M2_FIELDS_GF61)) return M2_EINVAL;
    if (m2::transform_log2(p, fields == M2_FIELDS_GF61 ? 61 : 92) > 30) return M2_EUNSUPPORTED;
    m2::Layout L = m2::make_layout(p, fields == M2_FIELDS_GF61 ? 61 : 92);
    if (ln) *ln = L.ln;
    if (n) *n = L.n;
    if (widths) std::memcpy(widths, L.width.data(), L.n);
    return M2_OK;
}

int m2_create(m2_ctx** out, uint32_t p, int mode, const m2_opts* opts) {
    if (!out) return M2_EINVAL;
    *out = nullptr;
    if (p < 3 || mode < M2_MODE_LL || mode > M2_MODE_PRP3) return M2_EINVAL;
    m2_opts o{};
    if (opts) o = *opts;
    if (o.fields != M2_FIELDS_DUAL && o.fields != M2_FIELDS_GF61) return M2_EINVAL;
    const bool gf61 = (o.fields == M2_FIELDS_GF61);
    if (m2::transform_log2(p, gf61 ? 61 : 92) > 30) return M2_EUNSUPPORTED;
    std::unique_ptr<m2_ctx> c(new (std::nothrow) m2_ctx());
    if (!c) return M2_ENOMEM;
    c->L = m2::make_layout(p, gf61 ? 61 : 92, HEAD);
    c->gf61 = gf61;
    c->mode = mode;
    c->device = o.device;
    c->opts = o;
    c->opts.stream = nullptr;
    if (cudaSetDevice(o.device) != cudaSuccess) { cudaGetLastError(); return M2_EINVAL; }
    c->span = m2::carry_span(c->L);
    const u64 h = c->L.h;
    int path = o.path;
    // a lone test of h >= 2048 runs faster on the three-pass path's many CTAs
    // than in one CTA (the one-CTA path pays off when many tests share a launch)
    if (path == M2_PATH_AUTO) path = (h <= 1024) ? M2_PATH_SMALL : M2_PATH_LARGE;
    if (path == M2_PATH_SMALL && h > 8192) return M2_EUNSUPPORTED;
    if (path == M2_PATH_LARGE && !m2i::plan_large(c->L, c->span, o.carry_pairs, c->plan)) return M2_EUNSUPPORTED;
    c->path = path;
    if (o.stream) { c->stream = (cudaStream_t)o.stream; }
    else {
        if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) return M2_ECUDA;
        c->own_stream = true;
    }
    int rc;
    const u64 n = c->L.n;
    if ((rc = get_twiddles(c->device, h, c->tw))) { m2_destroy(c.release()); return rc; }
    m2_ctx* raw = c.get();
    Slab mem;
    mem.add(&raw->d_w61, n);
    mem.add(&raw->d_w31, n);
    mem.add(&raw->d_words, sizeof(m2k::StateWords));
    mem.add(&raw->d_digits, n * sizeof(i64));
    const int lh = raw->L.ln - 1;
    size_t cw = 0;
    mem.add(&raw->d_test, sizeof(m2k::SmallTest));
    if (path == M2_PATH_LARGE) {
        const m2k::LargePlan& P = raw->plan;
        mem.add(&raw->d_carries, sizeof(i64) * (size_t)P.R * P.G);
        mem.add(&raw->d_za, sizeof(ulonglong2) * h);
        mem.add(&raw->d_zb, sizeof(uint2) * h);
        mem.add(&raw->d_flags, flags_bytes(P));
        // one launch for all squarings of a call where a shape of that kernel
        // serves the size; M2_PATH_LARGE and a -B hint ask for the three-pass kernels
        const bool lone = o.path == M2_PATH_AUTO && o.carry_pairs == 0;
        raw->cluster = lone && m2k::cluster_supported(lh, raw->span, gf61);
        raw->tide = lone && m2k::tide_supported(lh, raw->span, gf61);
        raw->flow = raw->tide || (lone && !raw->cluster && raw->span <= 3 && m2k::flow_carry_words(lh) != 0 &&
                                  m2k::flow_setup(lh, gf61) == cudaSuccess);
        cudaGetLastError();
        // the inverse column passes' per-element table
        if (m2k::cols_q_supported(P) || raw->flow) mem.add(&raw->d_aux, sizeof(uint2) * h);
        if (raw->flow) {
            cw = raw->tide ? m2k::tide_groups(lh) * raw->plan.R : m2k::flow_carry_words(lh);
            raw->flow_bytes = 8 * (cw + 1) + 4 * (raw->tide ? m2k::tide_groups(lh) : m2k::flow_groups(lh));
            mem.add(&raw->d_flow, raw->flow_bytes);
            if (raw->tide) {
                mem.add(&raw->d_taux, sizeof(uint2) * m2k::tide_records(lh));
                mem.add(&raw->d_tshift, sizeof(uint32_t) * m2k::tide_records(lh));
                mem.add(&raw->d_park, sizeof(longlong2) * m2k::tide_parked(lh));
            }
        }
    }
    if ((rc = mem.alloc(raw, &raw->d_slab))) { m2_destroy(c.release()); return rc; }
    raw->d_status = &raw->d_words->status;
    m2k::StateWords words{};
    if (raw->flow) words.yield = raw->yield = yield_word();
    try {
        raw->run = std::make_shared<m2b::Run>();
        m2b::Board::of(raw->device).add(raw->run);
    } catch (const std::bad_alloc&) {
        m2_destroy(c.release());
        return M2_ENOMEM;
    }
    raw->run->stream = raw->stream;
    raw->run->large = path == M2_PATH_LARGE && !raw->cluster;
    raw->run->whole = raw->tide;
    raw->run->crowds = raw->L.ln <= 18;
    raw->run->yield = raw->yield;
    cudaError_t e = cudaMemcpyAsync(raw->d_words, &words, sizeof(words), cudaMemcpyHostToDevice, raw->stream);
    if (e != cudaSuccess) { m2_destroy(c.release()); return M2_ECUDA; }
    if (path == M2_PATH_SMALL) {
        raw->threads = m2k::small_threads_for((unsigned)h);
        if (o.wg >= 32 && o.wg <= 256 && (o.wg & (o.wg - 1)) == 0) raw->threads = (int)o.wg;
        raw->carry_threads = small_carry_threads(raw->L, raw->span, raw->threads);
        if (o.carry_pairs > 0 && raw->carry_threads > 0) {
            // -B: segments of about 2 carry_pairs digits, a power of two of them
            int shift = 0;
            while (shift < 8 && (u64)(raw->threads >> (shift + 1)) >= 1 &&
                   2ull * o.carry_pairs * (u64)(raw->threads >> shift) > n)
                ++shift;
            raw->carry_threads = small_carry_threads(raw->L, raw->span, raw->threads, shift);
        }
        // a lone small test: one element per thread, in a cluster from n = 2^9
        // on (M2_PATH_SMALL and the hints speak of the one-CTA kernel, which the
        // shared launches of batches and the server run too)
        const bool lone = o.path == M2_PATH_AUTO && !o.wg && !o.carry_pairs && !o.fused_middle && raw->carry_threads > 0;
        raw->cluster = lone && m2k::cluster_supported(lh, raw->span, gf61);
        raw->lane = lone && !raw->cluster && m2k::lane_supported((unsigned)h, raw->span, raw->carry_threads);
    } else {
        const m2k::LargePlan& P = raw->plan;
        raw->plan.mode = mode;
        raw->plan.gf61 = gf61 ? 1u : 0u;
        raw->bufs = m2k::LargeBufs{raw->d_digits, raw->d_carries, raw->d_za, raw->d_zb, raw->d_w61, raw->d_w31,
                                   raw->tw.tw4, raw->tw.tc, raw->d_status, raw->d_flags};
        raw->bufs.aux = raw->d_aux;
        if (m2k::large_setup(P) != cudaSuccess) { m2_destroy(c.release()); return M2_EUNSUPPORTED; }
        raw->fused = m2k::cols_mid_supported(P);
        raw->plan.mid_tickets = (raw->fused && !m2k::cols_mid_cooperative(P)) ? 1u : 0u;
        // the phase barrier measured faster with R = 1024 rows only (n = 2^21)
        raw->plan.mid_barrier = (raw->fused && !P.mid_tickets && P.R == 1024u) ? 1u : 0u;
        if (raw->flow) {
            raw->fargs = m2k::FlowArgs{raw->d_digits, raw->d_carries, raw->d_za, raw->d_zb, raw->d_w61, raw->d_w31, raw->d_aux,
                                       raw->tw.tw4, raw->tw.tc, reinterpret_cast<unsigned long long*>(raw->d_flow),
                                       reinterpret_cast<unsigned long long*>(raw->d_flow) + cw,
                                       reinterpret_cast<unsigned*>(raw->d_flow + 8 * (cw + 1)), raw->d_status, 0u,
                                       (unsigned short)(2u * P.C), (unsigned short)0, raw->span, mode};
        }
        // without the fused column kernel; with the fields in turn where those serve the size (m2_pass.cu)
        raw->free_plan = raw->plan;
        raw->free_plan.mid_tickets = raw->free_plan.mid_barrier = 0u;
        raw->free_plan.in_turn = P.R == 256u ? 1u : 0u;
        if (((raw->flow || raw->fused) && m2k::pass_setup(raw->free_plan) != cudaSuccess) || (raw->tide && m2k::normalize_setup() != cudaSuccess)) { m2_destroy(c.release()); return M2_EUNSUPPORTED; }
        raw->bufs.ticket = reinterpret_cast<unsigned long long*>(raw->d_flags + P.G);
        raw->bufs.phase = reinterpret_cast<unsigned long long*>(raw->d_flags + P.G + 2);
    }
    m2k::SmallTest t{};
    t.digits = raw->d_digits; t.w61 = raw->d_w61; t.w31 = raw->d_w31;
    t.tw4 = raw->tw.tw4; t.tc = raw->tw.tc; t.status = raw->d_status;
    t.p = p; t.iters = 0; t.ln = raw->L.ln; t.mode = mode; t.span = raw->span;
    t.carry_threads = raw->carry_threads;
    t.fuse_middle = o.fused_middle ? 1 : 0;
    t.gf61_only = gf61 ? 1 : 0;
    raw->h_test = t;
    if (cudaMemcpyAsync(raw->d_test, &raw->h_test, sizeof(t), cudaMemcpyHostToDevice, raw->stream) != cudaSuccess) {
        m2_destroy(c.release());
        return M2_ECUDA;
    }
    raw->bytes += raw->tw.bytes;
    // shifts, unweighting records and the start state x0, built on the device
    // (tiny exponents, whose first digit may not hold x0, take it from the host)
    const long long x0 = mode == M2_MODE_LL ? 4 : 3;
    const bool host_state = raw->L.q < 4;
    e = m2k::launch_test_init(m2k::TestInit{raw->d_w61, raw->d_w31, raw->d_aux, host_state ? nullptr : raw->d_digits, x0, p, raw->L.ln},
                              raw->stream);
    if (e == cudaSuccess && raw->tide) e = m2k::tide_tables(lh, tide_args(raw), raw->stream);
    if (e == cudaSuccess) e = reset_sync_words(raw);
    if (e != cudaSuccess) { rc = fail_cuda("test setup", e); m2_destroy(c.release()); return rc; }
    if (host_state) {
        const m2::Layout L = m2::make_layout(p, gf61 ? 61 : 92);
        if ((rc = upload_state(raw, L, m2::digits_of_small(L, (u64)x0)))) { m2_destroy(c.release()); return rc; }
    }
    *out = c.release();
    return M2_OK;
}

int m2_iterate(m2_ctx* c, uint32_t k) {
    if (!c) return M2_EINVAL;
    if (k == 0) return M2_OK;
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    const int rc = advance(c, k, alone(c));
    if (!rc) c->iteration += k;
    return rc;
}

int m2_sync(m2_ctx* c) {
    if (!c) return M2_EINVAL;
    return settle(c);
}

int m2_get_digits(m2_ctx* c, uint64_t* out) {
    if (!c || !out) return M2_EINVAL;
    return read_settled(c, [&] {
        m2k::NormArgs a;
        const int rc = device_canonical(c, a);
        if (rc) return rc;
        const cudaError_t e = m2i::read_back(out, c->d_canon, c->L.n * sizeof(u64), c->stream);
        return e == cudaSuccess ? M2_OK : fail_cuda("digits read", e);
    });
}

int m2_set_digits(m2_ctx* c, const uint64_t* digits, uint32_t iteration) {
    if (!c || !digits) return M2_EINVAL;
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) return M2_ECUDA;   // (the old state's owed squarings go with it)
    // canonical input (every digit below 2^width), the usual case: uploaded and
    // balanced on the device, which also checks that it is canonical; anything
    // else is reduced on the host first
    int rc;
    if ((rc = canon_alloc(c))) return rc;
    unsigned* d_bad = reinterpret_cast<unsigned*>(c->d_norm);   // scratch word, free between reads
    unsigned bad = 0;
    cudaError_t e = cudaMemsetAsync(d_bad, 0, sizeof(unsigned), c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d_canon, digits, c->L.n * sizeof(u64), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = m2k::launch_balance(c->d_canon, c->d_digits, c->L.p, c->L.ln, c->L.n, d_bad, c->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, d_bad, sizeof(unsigned), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = reset_sync_words(c);
    if (e == cudaSuccess) e = clear_words(c);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return fail_cuda("state upload", e);
    if (bad) {
        try {
            const m2::Layout L = m2::make_layout(c->L.p, c->gf61 ? 61 : 92);
            rc = upload_state(c, L, m2::canonical_from_unsigned(L, digits));
        } catch (const std::bad_alloc&) {
            rc = M2_ENOMEM;
        } catch (const std::exception&) {
            rc = M2_EINVAL;
        }
        if (rc) return rc;
        cudaMemset(c->d_status, 0, sizeof(int));
    }
    c->iteration = iteration;
    return M2_OK;
}

int m2_res64(m2_ctx* c, uint64_t* out) {
    if (!c || !out) return M2_EINVAL;
    std::vector<u64> head;
    unsigned flags = 0;
    int rc = read_head(c, head, flags);
    if (rc) return rc;
    u64 r = 0;
    for (u64 j = 0; j < head.size() && c->L.bitpos[j] < 64; ++j) r |= head[j] << c->L.bitpos[j];
    *out = r;
    return M2_OK;
}

int m2_verdict(m2_ctx* c, int* is_prime) {
    if (!c || !is_prime) return M2_EINVAL;
    std::vector<u64> head;
    unsigned flags = 0;
    int rc = read_head(c, head, flags);
    if (rc) return rc;
    u64 want = c->mode == M2_MODE_LL ? 0 : (c->mode == M2_MODE_PRP ? 9 : 3);
    if (c->L.p < 64) want %= (u64(1) << c->L.p) - 1;
    // digits from index 8 on are zero when the result was all ones (written as
    // zero) or when no digit there is nonzero
    bool same = (flags & 1u) || !(flags & 2u);
    for (u64 j = 0; j < head.size() && same; ++j) {
        const u64 pos = c->L.bitpos[j], w = c->L.width[j];
        same = head[j] == (pos < 64 ? (want >> pos) & ((u64(1) << w) - 1) : 0);
    }
    *is_prime = same ? 1 : 0;
    return M2_OK;
}

int m2_carry_normalize(uint32_t p, const int64_t* digits, const int64_t* seg_carries, uint32_t seg_digits,
                       uint64_t* out, void* stream) {
    if (p < 3 || !digits || !out) return M2_EINVAL;
    if (m2::transform_log2(p) > 30) return M2_EUNSUPPORTED;
    const int ln = m2::transform_log2(p);
    const u64 n = u64(1) << ln;
    if (seg_carries && (seg_digits == 0 || seg_digits % 8 != 0 || n % seg_digits != 0)) return M2_EINVAL;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return M2_ECUDA;
    cudaMemPool_t mp = ctx_pool(dev);
    if (!mp) return M2_ECUDA;
    cudaStream_t s = (cudaStream_t)stream;
    void* scratch = nullptr;
    const size_t sb = m2k::norm_scratch_bytes(n) + 64;
    cudaError_t e = cudaMallocFromPoolAsync(&scratch, sb, mp, s);
    if (e != cudaSuccess) return fail_cuda("carry scratch", e);
    m2k::NormArgs a{};
    a.digits = reinterpret_cast<const long long*>(digits);
    a.carries = reinterpret_cast<const long long*>(seg_carries);
    a.seg = seg_carries ? seg_digits : 0;
    a.n = n; a.p = p; a.ln = ln;
    a.out = reinterpret_cast<unsigned long long*>(out);
    m2k::norm_bind_scratch(a, scratch);
    a.status = reinterpret_cast<int*>(static_cast<char*>(scratch) + m2k::norm_scratch_bytes(n));
    int st = 0;
    e = cudaMemsetAsync(a.status, 0, sizeof(int), s);
    if (e == cudaSuccess) e = m2k::launch_normalize(a, s);
    if (e == cudaSuccess) e = m2i::read_back(&st, a.status, sizeof(int), s);
    if (e == cudaSuccess) e = cudaFreeAsync(scratch, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail_cuda("carry propagation", e);
    return st ? M2_ESTATE : M2_OK;
}

int m2_test_stall_fused(m2_ctx* c) {
    if (!c) return M2_EINVAL;
    if (c->cluster) { c->stall = true; return M2_OK; }
    if (!c->flow && (!c->fused || !c->d_flags)) return M2_EUNSUPPORTED;
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    if (c->flow) {
        // column group 0 expects a tag that no carry word has
        const unsigned never = 2u;
        cudaError_t e = cudaMemcpyAsync(c->fargs.parity, &never, sizeof(never), cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        return e == cudaSuccess ? M2_OK : fail_cuda("m2_test_stall_fused", e);
    }
    unsigned f0 = 0;
    cudaError_t e = m2i::read_back(&f0, c->d_flags, sizeof(unsigned), c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    f0 += 1u << 20;
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d_flags, &f0, sizeof(unsigned), cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    return e == cudaSuccess ? M2_OK : fail_cuda("m2_test_stall_fused", e);
}

int m2_test_stage(m2_ctx* c, int stage, void* za_out, void* zb_out) {
    if (!c || stage < 0 || stage > 2) return M2_EINVAL;
    if (c->path != M2_PATH_LARGE) return M2_EUNSUPPORTED;
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    if (const int rc = c->flow ? settle(c) : M2_OK) return rc;
    if (c->flow || c->cluster) {
        // what unstage needs, also under a capture
        if (const int rc = canon_alloc(c)) return rc;
        c->staged = true;
    }
    const size_t h = c->L.h;
    cudaError_t e = cudaSuccess;
    // a stage out of order: its kernels poll for elements without tags (m2_pass.cu)
    if (stage != 0 && !c->untagged) {
        e = cudaMemsetAsync(c->d_za, 0, 16 * h, c->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(c->d_zb, 0, 8 * h, c->stream);
    }
    c->untagged = true;
    if (e == cudaSuccess) e = m2k::launch_large_stage(c->plan, c->bufs, stage, c->stream);
    if (e == cudaSuccess && za_out) e = m2i::read_back(za_out, c->d_za, 16 * h, c->stream);
    if (e == cudaSuccess && zb_out) e = m2i::read_back(zb_out, c->d_zb, 8 * h, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return fail_cuda("m2_test_stage", e);
    if (stage == 2) c->iteration += 1;
    return m2_sync(c);
}

int m2_info(m2_ctx* c, m2_info_t* info) {
    if (!c || !info) return M2_EINVAL;
    std::memset(info, 0, sizeof(*info));
    info->p = c->L.p; info->mode = c->mode; info->ln = c->L.ln; info->n = c->L.n;
    info->iteration = c->iteration;
    info->total_iters = total_iters_for(c->L.p, c->mode);
    info->path = c->path;
    info->span = (uint32_t)c->span;
    if (c->path == M2_PATH_LARGE) { info->rows = c->plan.R; info->row_len = c->plan.B; info->cols_per_cta = c->plan.C; }
    else { info->rows = 1; info->row_len = (uint32_t)c->L.h; info->cols_per_cta = (uint32_t)c->threads; }
    info->device_bytes = c->bytes;
    info->fused_cols = c->fused ? 1u : 0u;
    info->fields = c->gf61 ? M2_FIELDS_GF61 : M2_FIELDS_DUAL;
    return M2_OK;
}

void m2_destroy(m2_ctx* c) {
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->run) m2b::Board::of(c->device).remove(c->run);
    if (c->yield) {
        std::lock_guard<std::mutex> lk(g_yield_mu);
        g_yield.push_back(c->yield);
    }
    // stream-ordered frees: they follow the context's queued work and do not
    // wait for other streams; its stream is released once that work is done
    if (c->stream)
        for (void* b : {c->d_slab, c->d_read}) if (b) cudaFreeAsync(b, c->stream);
    for (auto& set : c->graph)
        for (cudaGraphExec_t g : set)
            if (g) cudaGraphExecDestroy(g);
    if (c->own_stream && c->stream) cudaStreamDestroy(c->stream);
    delete c;
}

int m2_profile(m2_ctx* c, uint32_t iters, m2_stage_time* out, int max_stages, int* n_stages) {
    if (!c || !out || max_stages < 1 || iters == 0) return M2_EINVAL;
    if (cudaSetDevice(c->device) != cudaSuccess) return M2_ECUDA;
    // the launch sequence m2_iterate issues for `iters` squarings, one event after each
    std::vector<int> seq;
    if (const int rc = unstage(c)) return rc;
    m2b::Board& board = m2b::Board::of(c->device);
    const m2b::Kind kind = board.begin(*c->run, alone(c));
    const bool free = kind == m2b::FREE && kind != alone(c);
    if (own_kernel(c) && !free) seq.push_back(-1);
    else if (kind == m2b::FUSED) {
        seq = {0, 1};
        for (uint32_t i = 1; i < iters; ++i) { seq.push_back(m2k::STAGE_MID); seq.push_back(1); }
        seq.push_back(2);
    } else {
        for (uint32_t i = 0; i < iters; ++i) for (int st = 0; st < m2k::LARGE_STAGES; ++st) seq.push_back(st);
    }
    std::vector<cudaEvent_t> ev(seq.size() + 1);
    cudaError_t err = cudaSuccess;
    for (auto& e : ev) if (err == cudaSuccess) err = cudaEventCreate(&e);
    if (err == cudaSuccess) err = cudaEventRecord(ev[0], c->stream);
    if (free && c->flow) c->staged = true;
    for (size_t i = 0; i < seq.size() && err == cudaSuccess; ++i) {
        if (seq[i] < 0) err = launch_own(c, iters, false);
        else err = m2k::launch_large_stage(free ? c->free_plan : c->plan, c->bufs, seq[i], c->stream);
        if (err == cudaSuccess) err = cudaEventRecord(ev[i + 1], c->stream);
    }
    if (err == cudaSuccess) err = cudaStreamSynchronize(c->stream);
    board.done(*c->run);
    // per stage (in order of first appearance): total time and launches
    std::vector<int> order;
    std::map<int, std::pair<double, uint64_t>> tot;
    if (err == cudaSuccess) {
        for (size_t i = 0; i < seq.size(); ++i) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev[i], ev[i + 1]);
            if (!tot.count(seq[i])) order.push_back(seq[i]);
            tot[seq[i]].first += ms;
            tot[seq[i]].second += 1;
        }
    }
    for (auto& e : ev) if (e) cudaEventDestroy(e);
    if (err != cudaSuccess) return fail_cuda("m2_profile", err);
    c->iteration += iters;
    if (const int rc = unstage(c)) return rc;
    const int k = std::min((int)order.size(), max_stages);
    for (int i = 0; i < k; ++i) {
        const int st = order[i];
        m2_stage_time& o = out[i];
        std::memset(&o, 0, sizeof(o));
        const char* nm = (st < 0) ? own_kernel_name(c) : m2k::large_stage_name(st);
        std::strncpy(o.name, nm, sizeof(o.name) - 1);
        o.launches = tot[st].second;
        o.ms_per_launch = tot[st].first / (double)o.launches;
        o.iters_per_launch = (st < 0) ? iters : 1u;
        // on chip between squarings (digits in and out), or both hand-overs of
        // every squaring through global memory
        o.bytes_per_launch = (st >= 0) ? m2k::large_stage_bytes(c->plan, st)
                             : c->flow ? (uint64_t)iters * 2 * m2k::large_stage_bytes(c->plan, 1) : 16ull * c->L.n;
    }
    if (n_stages) *n_stages = k;
    return M2_OK;
}

uint64_t m2_launches_for(m2_ctx* c, uint32_t k) {
    if (!c || k == 0) return 0;
    if (own_kernel(c)) return ((uint64_t)k - 1) / iters_per_launch(c) + 1;
    if (!c->fused) return (uint64_t)m2k::LARGE_STAGES * k;
    // graph replays of GRAPH_ITERS[0] then GRAPH_ITERS[1] squarings, then the
    // rest in one sequence
    uint64_t left = k, n = 0;
    for (int i = 0; i < 2 && !c->graph_failed; ++i) {
        const uint64_t chunks = left / GRAPH_ITERS[i];
        n += chunks * (2ull * GRAPH_ITERS[i] + 1);
        left -= chunks * GRAPH_ITERS[i];
    }
    return n + (left ? 2 * left + 1 : 0);
}

int m2_measure_mul_peak(int device, double* products_per_s) {
    if (!products_per_s) return M2_EINVAL;
    const double r = m2k::measure_wide_mul_rate(device);
    if (r <= 0.0) return M2_ECUDA;
    *products_per_s = r;
    return M2_OK;
}

}  // extern "C"

// ---------------- batched engine ----------------
namespace {

// Launch shape of the one-CTA kernel, tuned per (device, h): every
// combination of threads per transform (32 ... 256), carry segments (threads,
// threads / 2, threads / 4, each segment at least span + 1 digits) and the
// fused or separate transform middle runs a GPU-filling sample of the bucket's
// own tests for TUNE_ITERS squarings on scratch copies of their state, and so
// does m2_duo.cu's kernel where it serves all of them; the highest rate of
// test-squarings per second wins.  Cached for the process.
struct Tuned {
    int threads = 0, carry_shift = 0, fuse = 0;
    // the kernel of m2_duo.cu: its middle is fused, its carry has a segment per
    // thread, and its 512 or 1024 threads at h = 4096, 8192 count as 256, the
    // most that a caller may ask for
    bool duo = false;
    double ns_per_test_iter = 0.0, ns_default = 0.0;
    int blocks = 0;            // carry segments of the choice, and digits
    int n = 0;
};
std::mutex g_tune_mu;
// per device, size and whether the tests in flight fill the GPU (a test per SM and
// more): a few tests of n = 512 are faster in the one-CTA kernel, a full GPU of
// them in m2_duo.cu's, so neither's choice is the other's
std::map<std::tuple<int, u64, bool>, Tuned> g_tune;
bool find_tuned(int device, u64 h, bool full, Tuned& out) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune.find({device, h, full});
    if (it == g_tune.end()) return false;
    out = it->second;
    return true;
}
constexpr u32 TUNE_ITERS = 48;

// m2_duo.cu's kernel serves these tests of one size (both fields)
bool duo_for(const std::vector<m2k::SmallTest>& tests) {
    for (const m2k::SmallTest& t : tests)
        if (t.gf61_only || !m2k::duo_supported(1u << (t.ln - 1), t.span, t.carry_threads)) return false;
    return !tests.empty();
}

template <class Item>
int tune_bucket(int device, u64 h, const std::vector<Item>& items, const std::vector<m2k::SmallTest>& tests,
                const long long* d_dig, int sms, size_t total, Tuned& out) {
    const bool fills = total >= (size_t)sms;
    if (find_tuned(device, h, fills, out)) return M2_OK;
    const u64 n = 2 * h;
    // A batch of at least a test per SM is timed as a full GPU, the bucket's tests
    // repeated: a last wave that is not full would count against the kernel with
    // more tests per SM (n = 4096, 498 tests, m2_duo.cu: 143 ns per test-squaring for 118 in full waves).
    const size_t full = (size_t)std::max(sms, 1) * std::min<size_t>(32, std::max<size_t>(1, 232448 / (24 * h)));
    const size_t cap = fills ? full : items.size();
    long long* scratch = nullptr;
    m2k::SmallTest* d_t = nullptr;
    int* d_st = nullptr;
    cudaStream_t st = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    auto cleanup = [&]() {
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (st) cudaStreamDestroy(st);
        cudaFree(scratch); cudaFree(d_t); cudaFree(d_st);
    };
    if (cudaMalloc(&scratch, cap * n * sizeof(i64)) != cudaSuccess || cudaMalloc(&d_t, cap * sizeof(m2k::SmallTest)) != cudaSuccess ||
        cudaMalloc(&d_st, sizeof(int)) != cudaSuccess || cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        cudaGetLastError();
        cleanup();
        return M2_ENOMEM;
    }
    std::vector<m2k::SmallTest> d;
    // ns per test-squaring of `ns` tests by `launch` (from the bucket's own states)
    auto rate = [&](size_t ns, auto launch, double& out_ns) {
        cudaError_t e = cudaSuccess;
        for (size_t t = 0; t < ns; t += items.size())
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(scratch + t * n, d_dig, std::min(items.size(), ns - t) * n * sizeof(i64), cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(d_t, d.data(), ns * sizeof(m2k::SmallTest), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = launch(2u);   // warm-up
        if (e == cudaSuccess) e = cudaEventRecord(e0, st);
        if (e == cudaSuccess) e = launch(TUNE_ITERS);
        if (e == cudaSuccess) e = cudaEventRecord(e1, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        float ms = 0.f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
        out_ns = ms * 1e6 / ((double)ns * TUNE_ITERS);
        return e;
    };
    auto sample = [&](int per_sm) {
        const size_t ns = std::min(cap, (size_t)std::max(per_sm, 1) * (size_t)std::max(sms, 1));
        d.clear();
        for (size_t t = 0; t < ns; ++t) {
            d.push_back(tests[t % tests.size()]);
            d[t].digits = scratch + t * n;
            d[t].status = d_st;
        }
        return ns;
    };
    const int T0 = m2k::small_threads_for((unsigned)h);
    Tuned best;
    best.threads = T0;
    // one combination of the one-CTA kernel
    auto small_rate = [&](int T, int shift, int fuse) {
        const size_t ns = sample(m2k::small_ctas_per_sm((unsigned)h, T, fuse != 0));
        for (size_t t = 0; t < ns; ++t) {
            const Item& it = items[t % items.size()];
            d[t].carry_threads = small_carry_threads(it.L, it.span, T, shift);
            d[t].fuse_middle = fuse;
        }
        double ns_per = 0.0;
        const cudaError_t e = rate(ns, [&](u32 iters) {
            return m2k::launch_small(d_t, (int)ns, (unsigned)h, T, iters, st, fuse != 0);
        }, ns_per);
        if (T == T0 && shift == 0 && fuse == 0) best.ns_default = ns_per;
        if (best.ns_per_test_iter == 0.0 || ns_per < best.ns_per_test_iter) {
            best.threads = T; best.carry_shift = shift; best.fuse = fuse; best.ns_per_test_iter = ns_per;
        }
        return e;
    };
    cudaError_t e = small_rate(T0, 0, 0);
    if (e == cudaSuccess && duo_for(tests) && m2k::duo_ctas_per_sm((unsigned)h) > 0) {
        const size_t ns = sample(m2k::duo_ctas_per_sm((unsigned)h));
        double ns_per = 0.0;
        e = rate(ns, [&](u32 iters) { return m2k::launch_duo(d_t, (int)ns, (unsigned)h, iters, st); }, ns_per);
        if (ns_per < best.ns_per_test_iter) {
            best.threads = std::min(m2k::duo_threads((unsigned)h), 256); best.carry_shift = 0; best.fuse = 1; best.duo = true;
            best.ns_per_test_iter = ns_per;
        }
    }
    // on a full GPU no other combination comes near m2_duo.cu's kernel; a few
    // tests of n = 256 or 512 are 5-13% faster in the one-CTA kernel's best
    for (int T = 32; T <= 256 && !(best.duo && cap == full); T *= 2) {
        for (int shift = 0; shift <= 2; ++shift) {
            // a carry split that the segment length rules out collapses onto a smaller shift: skip repeats
            if (shift > 0 && small_carry_threads(items[0].L, items[0].span, T, shift) ==
                                 small_carry_threads(items[0].L, items[0].span, T, shift - 1))
                continue;
            for (int fuse = 0; fuse <= 1; ++fuse) {
                if (T == T0 && shift == 0 && fuse == 0) continue;   // the default, above
                const double before = best.ns_per_test_iter;
                if (e == cudaSuccess) e = small_rate(T, shift, fuse);
                if (best.ns_per_test_iter < before) best.duo = false;
            }
        }
    }
    if (e != cudaSuccess) { cleanup(); return fail_cuda("batch tuning", e); }
    cleanup();
    best.blocks = small_carry_threads(items[0].L, items[0].span, best.threads, best.carry_shift);
    best.n = (int)n;
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[{device, h, fills}] = best;
    out = best;
    return M2_OK;
}

}  // namespace

// the choice on a full GPU, else the one for fewer tests
static bool tuned_for(int device, int ln, Tuned& t) {
    const u64 h = u64(1) << (ln - 1);
    return find_tuned(device, h, true, t) || find_tuned(device, h, false, t);
}

extern "C" {

int m2_batch_tuned(int device, int ln, int* threads, double* ns_per_test_iter) {
    Tuned t;
    if (ln < 3 || ln > 14 || !tuned_for(device, ln, t)) return M2_EINVAL;
    if (threads) *threads = t.threads;
    if (ns_per_test_iter) *ns_per_test_iter = t.ns_per_test_iter;
    return M2_OK;
}

int m2_batch_tuning(int device, int ln, m2_batch_tuning_t* out) {
    Tuned t;
    if (ln < 3 || ln > 14 || !out || !tuned_for(device, ln, t)) return M2_EINVAL;
    out->threads = t.threads;
    out->carry_blocks = t.blocks;
    out->carry_pairs = t.blocks ? t.n / (2 * t.blocks) : 0;
    out->fused_middle = t.fuse;
    out->ns_per_test_iter = t.ns_per_test_iter;
    out->ns_default = t.ns_default;
    return M2_OK;
}
const char* m2_batch_kernel(int device, int ln) {
    Tuned t;
    if (ln < 3 || ln > 14 || !tuned_for(device, ln, t)) return nullptr;
    return t.duo ? "k_duo" : "k_small";
}

// Tests are bucketed by transform length h; every bucket is one persistent
// launch (CTAs pull test indices from a device counter, longest tests first)
// with its tuned threads per transform, all buckets run concurrently on their
// own streams, and the whole set of launches is captured into one CUDA graph.
int m2_batch_run(const uint32_t* p, const int* modes, const uint32_t* iters, size_t count,
                 uint64_t* res64_out, int* is_prime_out, int device, m2_batch_stats* stats) {
    if (!p || count == 0) return M2_EINVAL;
    if (cudaSetDevice(device) != cudaSuccess) { cudaGetLastError(); return M2_EINVAL; }
    struct Item { size_t idx; m2::Layout L; int mode; u32 iters; int span; };
    std::map<u64, std::vector<Item>> buckets;
    for (size_t i = 0; i < count; ++i) {
        const int mode = modes ? modes[i] : M2_MODE_PRP;
        if (p[i] < 3 || mode < M2_MODE_LL || mode > M2_MODE_PRP3) return M2_EINVAL;
        if (m2::transform_log2(p[i]) > 14) return M2_EUNSUPPORTED;   // h <= 8192
        Item it;
        it.idx = i; it.L = m2::make_layout(p[i], 92, 0); it.mode = mode;
        it.iters = iters ? iters[i] : total_iters_for(p[i], mode);
        it.span = m2::carry_span(it.L);
        buckets[it.L.h].push_back(std::move(it));
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // device memory from the stream-ordered pool: a call neither waits for nor
    // holds up other work on the device.  What the pool grew by goes back at the
    // end, but for 256 MiB that the next call finds ready (the tests of a full GPU
    // take 10 to 50 MB).
    cudaMemPool_t mp = ctx_pool(device);
    if (!mp) return M2_ECUDA;
    struct Trim {
        cudaMemPool_t mp;
        uint64_t keep = 0;
        explicit Trim(cudaMemPool_t pool) : mp(pool) {
            if (cudaMemPoolGetAttribute(mp, cudaMemPoolAttrReservedMemCurrent, &keep) != cudaSuccess) cudaGetLastError();
            keep = std::max<uint64_t>(keep, 256ull << 20);
        }
        ~Trim() {
            uint64_t now = 0;
            if (cudaMemPoolGetAttribute(mp, cudaMemPoolAttrReservedMemCurrent, &now) != cudaSuccess) cudaGetLastError();
            if (now > keep && cudaMemPoolTrimTo(mp, keep) != cudaSuccess) cudaGetLastError();
        }
    } trim(mp);
    struct Dev {
        std::vector<void*> allocs;
        std::vector<cudaStream_t> streams;
        std::vector<cudaEvent_t> events;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        ~Dev() {
            if (!streams.empty() && streams[0]) {
                for (auto a : allocs) cudaFreeAsync(a, streams[0]);
                cudaStreamSynchronize(streams[0]);
            }
            if (exec) cudaGraphExecDestroy(exec);
            if (graph) cudaGraphDestroy(graph);
            for (auto e : events) if (e) cudaEventDestroy(e);
            for (auto s : streams) if (s) cudaStreamDestroy(s);
        }
    } dv;
    const size_t nb = buckets.size();
    struct Turn {   // in flight from here to the end of the call
        m2b::Board& board;
        std::shared_ptr<m2b::Run> run = std::make_shared<m2b::Run>();
        explicit Turn(int device) : board(m2b::Board::of(device)) {
            board.add(run);
            board.begin(*run, m2b::BATCH);
        }
        ~Turn() {
            board.done(*run);
            board.remove(run);
        }
    } turn(device);
    dv.streams.resize(nb + 1, nullptr);
    for (auto& s : dv.streams) if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return M2_ECUDA;
    dv.events.resize(nb + 3, nullptr);
    for (size_t i = 0; i < dv.events.size(); ++i)
        if (cudaEventCreateWithFlags(&dv.events[i], i == 1 || i == 2 ? cudaEventDefault : cudaEventDisableTiming) != cudaSuccess) return M2_ECUDA;
    cudaStream_t s0 = dv.streams[0];
    auto dmal = [&](void** ptr, size_t bytes) -> int {
        if (cudaMallocFromPoolAsync(ptr, bytes, mp, s0) != cudaSuccess) { cudaGetLastError(); return M2_ENOMEM; }
        dv.allocs.push_back(*ptr);
        return M2_OK;
    };
    // test descriptors, results and one {queue, status} pair per bucket, in bucket order
    int rc;
    m2k::SmallTest* d_all = nullptr; m2k::TestInit* d_init = nullptr; unsigned long long* d_res = nullptr; int *d_prime = nullptr, *d_q = nullptr;
    if ((rc = dmal((void**)&d_all, count * sizeof(m2k::SmallTest))) || (rc = dmal((void**)&d_init, count * sizeof(m2k::TestInit))) ||
        (rc = dmal((void**)&d_res, count * sizeof(u64))) || (rc = dmal((void**)&d_prime, count * sizeof(int))) ||
        (rc = dmal((void**)&d_q, 2 * nb * sizeof(int))))
        return rc;
    struct Launch { u64 h; int ln, threads, ntests, grid; size_t first; long long* d_dig; std::vector<Item>* items; bool fuse, duo; };
    std::vector<Launch> launches;
    std::vector<m2k::SmallTest> tests(count);
    std::vector<m2k::TestInit> init(count);
    uint64_t squarings = 0;
    size_t first = 0;
    for (auto& kv : buckets) {
        const u64 h = kv.first, n = 2 * h;
        std::vector<Item>& items = kv.second;
        std::sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.iters > b.iters; });
        const size_t nt = items.size();
        TwTables tw;
        if ((rc = get_twiddles(device, h, tw))) return rc;
        long long* d_dig = nullptr; unsigned char* d_w = nullptr;
        if ((rc = dmal((void**)&d_dig, nt * n * sizeof(i64))) || (rc = dmal((void**)&d_w, nt * n * 2))) return rc;
        for (size_t t = 0; t < nt; ++t) {
            const Item& it = items[t];
            m2k::SmallTest& T = tests[first + t];
            T.digits = d_dig + t * n; T.w61 = d_w + t * 2 * n; T.w31 = d_w + t * 2 * n + n;
            T.tw4 = tw.tw4; T.tc = tw.tc; T.status = d_q + 2 * launches.size() + 1;
            T.p = it.L.p; T.iters = it.iters; T.ln = it.L.ln; T.mode = it.mode; T.span = it.span;
            T.carry_threads = small_carry_threads(it.L, it.span, m2k::small_threads_for((unsigned)h));
            T.gf61_only = 0; T.fuse_middle = 0;
            const u64 x0 = it.mode == M2_MODE_LL ? 4 : 3;
            const bool host_state = it.L.q < 4;   // tiny: the first digit may not hold x0
            init[first + t] = m2k::TestInit{d_w + t * 2 * n, d_w + t * 2 * n + n, nullptr, host_state ? nullptr : T.digits, (long long)x0, it.L.p, it.L.ln};
            if (host_state) {
                const m2::Layout L = m2::make_layout(it.L.p);
                const std::vector<i64> b = m2::balanced_digits(L, m2::digits_of_small(L, x0));
                if (cudaMemcpyAsync(T.digits, b.data(), n * sizeof(i64), cudaMemcpyHostToDevice, s0) != cudaSuccess) return M2_ECUDA;
            }
            squarings += it.iters;
        }
        launches.push_back(Launch{h, items[0].L.ln, 0, (int)nt, 0, first, d_dig, &items, false, false});
        first += nt;
    }
    cudaError_t e = cudaMemsetAsync(d_q, 0, 2 * nb * sizeof(int), s0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_init, init.data(), count * sizeof(m2k::TestInit), cudaMemcpyHostToDevice, s0);
    if (e == cudaSuccess) e = m2k::launch_test_init(d_init, (int)count, s0);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s0);   // the tuner reads the start states on a stream of its own
    if (e != cudaSuccess) return fail_cuda("batch setup", e);
    for (Launch& l : launches) {
        std::vector<Item>& items = *l.items;
        Tuned tn;
        const std::vector<m2k::SmallTest> mine(tests.begin() + l.first, tests.begin() + l.first + l.ntests);
        if ((rc = tune_bucket(device, l.h, items, mine, l.d_dig, sms, count, tn))) return rc;
        // the choice is cached per size: these tests may have one it does not serve
        l.duo = tn.duo && duo_for(mine);
        l.threads = tn.threads;
        l.fuse = tn.fuse != 0;
        for (int t = 0; t < l.ntests; ++t) {
            tests[l.first + t].carry_threads = small_carry_threads(items[t].L, items[t].span, tn.threads, tn.carry_shift);
            tests[l.first + t].fuse_middle = tn.fuse;
        }
        const int per_sm = l.duo ? m2k::duo_ctas_per_sm((unsigned)l.h) : m2k::small_ctas_per_sm((unsigned)l.h, l.threads, l.fuse);
        l.grid = (int)std::min<size_t>((size_t)l.ntests, (size_t)per_sm * (size_t)std::max(sms, 1));
    }
    if (cudaMemcpyAsync(d_all, tests.data(), count * sizeof(m2k::SmallTest), cudaMemcpyHostToDevice, s0) != cudaSuccess) return M2_ECUDA;
    // capture: fork from stream 0 to one stream per bucket, join back
    if (cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return M2_ECUDA;
    cudaEventRecord(dv.events[0], s0);
    for (size_t b = launches.size(); b-- > 0;) {   // the largest size first
        cudaStream_t sb = dv.streams[b + 1];
        cudaStreamWaitEvent(sb, dv.events[0], 0);
        const Launch& l = launches[b];
        if (l.duo) m2k::launch_duo(d_all + l.first, l.ntests, (unsigned)l.h, 0u, sb, d_q + 2 * b, l.grid);
        else m2k::launch_small_persistent(d_all + l.first, l.ntests, (unsigned)l.h, l.threads, d_q + 2 * b, l.grid, sb, l.fuse);
        cudaEventRecord(dv.events[b + 3], sb);
        cudaStreamWaitEvent(s0, dv.events[b + 3], 0);
    }
    if (cudaStreamEndCapture(s0, &dv.graph) != cudaSuccess) return M2_ECUDA;
    if (cudaGraphInstantiate(&dv.exec, dv.graph, 0) != cudaSuccess) return M2_ECUDA;
    cudaEvent_t t0 = dv.events[1], t1 = dv.events[2];
    cudaEventRecord(t0, s0);
    if (cudaGraphLaunch(dv.exec, s0) != cudaSuccess) return M2_ECUDA;
    cudaEventRecord(t1, s0);
    for (const Launch& l : launches)
        if (e == cudaSuccess) e = m2k::launch_results(d_all + l.first, l.ntests, l.ln, d_res + l.first, d_prime + l.first, s0);
    std::vector<u64> res(count);
    std::vector<int> prime(count), q(2 * nb);
    if (e == cudaSuccess) e = m2i::read_back(res.data(), d_res, count * sizeof(u64), s0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(prime.data(), d_prime, count * sizeof(int), cudaMemcpyDeviceToHost, s0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(q.data(), d_q, 2 * nb * sizeof(int), cudaMemcpyDeviceToHost, s0);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s0);
    if (e != cudaSuccess) return fail_cuda("batch run", e);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, t0, t1);
    int status_any = 0;
    for (size_t b = 0; b < launches.size(); ++b) {
        status_any |= q[2 * b + 1];
        const Launch& l = launches[b];
        for (int t = 0; t < l.ntests; ++t) {
            const Item& it = (*l.items)[t];
            if (res64_out) res64_out[it.idx] = res[l.first + t];
            if (is_prime_out) is_prime_out[it.idx] = prime[l.first + t];
        }
    }
    if (stats) {
        stats->seconds = ms * 1e-3;
        stats->squarings = squarings;
        stats->launches = (uint32_t)launches.size();
        stats->buckets = (uint32_t)buckets.size();
    }
    return status_any ? M2_ESTATE : M2_OK;
}

}  // extern "C"

// ---------------- serving engine ----------------
// Lanes run independently: the one-CTA tests of one transform size form one
// lane (one launch advances all of them), every three-pass test is a lane of
// its own (its context's stream).  A step starts the next quantum on every idle
// lane, then waits (bounded) until at least one lane has finished and accounts
// for it, so a long quantum of a large test never holds back small ones.
namespace {

struct SrvItem {
    uint64_t id = 0;
    uint32_t p = 0;
    int mode = 0;
    uint32_t total = 0, done = 0;
    uint32_t inflight = 0;       // squarings launched and not yet accounted
    m2_ctx* ctx = nullptr;
    cudaEvent_t ev = nullptr;    // three-pass tests: end of the quantum in flight
    uint64_t bytes = 0;
    double t_submit = 0, t_admit = 0;
};

struct SrvBucket {
    m2k::SmallTest* d_tests = nullptr;
    m2k::SmallTest* h_tests = nullptr;   // pinned staging of the descriptors
    int* d_status = nullptr;             // status word of each member for this launch
    int* h_status = nullptr;             // pinned copy, read once the launch is done
    size_t cap = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev = nullptr;
    std::vector<uint64_t> members;       // keys of the tests in the launch in flight
    std::vector<uint32_t> ks;
    std::shared_ptr<m2b::Run> run;
    bool busy = false;
    bool whole = false;                  // its CTAs hold whole SMs (srv_launch)
};

// device memory a test will hold (digits, weights, status, descriptor; the
// element arrays and carries of the three-pass path); twiddles are shared
uint64_t srv_estimate(uint32_t p) {
    const int ln = m2::transform_log2(p);
    const uint64_t n = uint64_t(1) << ln, h = n / 2;
    uint64_t b = 10 * n + 512;
    if (h > 8192) b += 24 * h + 8 * (h / 4) + 4096;
    return b;
}

// longest a step waits for a lane to finish before reporting M2_ETIMEOUT
constexpr double SRV_WAIT_LIMIT_S = 600.0;

}  // namespace

struct m2_server {
    int device = 0;
    uint64_t budget = 0;
    uint32_t quantum = 1000;
    int sms = 1;
    size_t smem_sm = 0;                   // shared memory of an SM
    std::deque<SrvItem> queue;
    std::map<uint64_t, SrvItem> active;   // key: admission order
    uint64_t next_key = 0;
    std::deque<m2_srv_result> finished;
    std::map<u64, SrvBucket> buckets;
    // the one-CTA tests' contexts share a stream (they only set up and read
    // back on it; their squarings run in the buckets' launches, which wait for
    // small_ready): a stream per test makes every allocation slower
    cudaStream_t small_stream = nullptr;
    cudaEvent_t small_ready = nullptr;
    uint64_t resident = 0, squarings = 0, completed = 0;
    uint32_t steps = 0, launches = 0;
    std::chrono::steady_clock::time_point t0;
    double now() const { return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count(); }
};

namespace {

void srv_retire(m2_server* s, SrvItem& it, int status) {
    m2_srv_result r{};
    r.id = it.id; r.p = it.p; r.mode = it.mode; r.iters = it.done; r.status = status;
    r.t_submit = it.t_submit; r.t_admit = it.t_admit;
    if (it.ctx) {
        r.n = it.ctx->L.n;
        if (status == M2_OK) {
            int rc = m2_res64(it.ctx, &r.res64);
            if (rc == M2_OK) rc = m2_verdict(it.ctx, &r.is_prime);
            r.status = rc;
        }
        m2_destroy(it.ctx);
        it.ctx = nullptr;
    }
    if (it.ev) { cudaEventDestroy(it.ev); it.ev = nullptr; }
    r.t_done = s->now();
    s->resident -= it.bytes;
    s->completed++;
    s->finished.push_back(r);
}

int srv_bucket_reserve(SrvBucket& b, size_t need) {
    cudaError_t e;
    int lo = 0, hi = 0;   // before the larger lanes' CTAs (srv_launch)
    cudaDeviceGetStreamPriorityRange(&lo, &hi);
    if (!b.stream && (e = cudaStreamCreateWithPriority(&b.stream, cudaStreamNonBlocking, hi)) != cudaSuccess)
        return fail_cuda("server stream", e);
    if (!b.ev && (e = cudaEventCreateWithFlags(&b.ev, cudaEventDisableTiming)) != cudaSuccess)
        return fail_cuda("server event", e);
    if (b.cap >= need) return M2_OK;
    cudaFree(b.d_tests); cudaFree(b.d_status); cudaFreeHost(b.h_tests); cudaFreeHost(b.h_status);
    b.d_tests = nullptr; b.d_status = nullptr; b.h_tests = nullptr; b.h_status = nullptr;
    const size_t cap = std::max<size_t>({need, 2 * b.cap, 64});
    if ((e = cudaMalloc(&b.d_tests, cap * sizeof(m2k::SmallTest))) != cudaSuccess ||
        (e = cudaMalloc(&b.d_status, cap * sizeof(int))) != cudaSuccess ||
        (e = cudaMallocHost(&b.h_tests, cap * sizeof(m2k::SmallTest))) != cudaSuccess ||
        (e = cudaMallocHost(&b.h_status, cap * sizeof(int))) != cudaSuccess) {
        b.cap = 0;
        return fail_cuda("server descriptors", e);
    }
    b.cap = cap;
    return M2_OK;
}

// starts a quantum on every idle lane
int srv_launch(m2_server* s) {
    std::map<u64, std::vector<uint64_t>> small;
    size_t total = 0;
    bool waits = false;   // a lane's column CTAs wait for each other
    for (auto& kv : s->active) {
        SrvItem& it = kv.second;
        if (it.ctx->path == M2_PATH_SMALL) ++total;
        else if (it.ctx->fused) waits = true;
        if (it.inflight) continue;
        if (it.ctx->path == M2_PATH_SMALL) {
            auto b = s->buckets.find(it.ctx->L.h);
            if (b == s->buckets.end() || !b->second.busy) small[it.ctx->L.h].push_back(kv.first);
            continue;
        }
        const uint32_t k = std::min(s->quantum, it.total - it.done);
        // CTAs that wait for each other need room for all of them
        if (it.ctx->fused)
            for (auto& b : s->buckets)
                if (b.second.busy && b.second.whole && cudaStreamWaitEvent(it.ctx->stream, b.second.ev, 0) != cudaSuccess)
                    return fail_cuda("server lane order", cudaGetLastError());
        int rc = m2_iterate(it.ctx, k);
        if (rc) return rc;
        cudaError_t e = cudaEventRecord(it.ev, it.ctx->stream);
        if (e != cudaSuccess) return fail_cuda("server event record", e);
        it.inflight = k;
        s->launches += (uint32_t)m2_launches_for(it.ctx, k);
    }
    // A one-CTA test is one serial chain: among the larger lanes' warps it gets a
    // warp's share of an SM and a request of a second takes two.  While the
    // one-CTA tests would fill at most half the SMs, each asks for the shared
    // memory of a whole one, so that nothing else joins it there; more of them
    // share in proportion (20 s of a mix: tests of n = 2^8 ... 2^12 12-45k ->
    // 19-67k squarings/s each, p99 9.5 -> 5.9 s, all tests 227k -> 232k).
    // Not beside column CTAs that wait for each other (n = 2^21 and up).
    const size_t per_sm = (2 * total + (size_t)s->sms - 1) / (size_t)s->sms;
    const size_t min_smem = per_sm && !waits ? s->smem_sm / per_sm : 0;
    for (auto& kv : small) {
        SrvBucket& b = s->buckets[kv.first];
        const size_t cnt = kv.second.size();
        int rc = srv_bucket_reserve(b, cnt);
        if (rc) return rc;
        b.members = kv.second;
        b.ks.resize(cnt);
        // one launch per transform size: the batch autotuner's shape for it when
        // cached, else the first member's; every member gets the launch's variant
        const m2_ctx* c0 = s->active[kv.second[0]].ctx;
        Tuned tn;
        const bool tuned = find_tuned(s->device, kv.first, total >= (size_t)s->sms, tn);
        bool duo = !tuned || tn.duo;
        for (size_t j = 0; j < cnt && duo; ++j) duo = duo_for({s->active[kv.second[j]].ctx->h_test});
        const int threads = tuned ? tn.threads : c0->threads;
        const bool fuse = tuned ? tn.fuse != 0 : c0->h_test.fuse_middle != 0;
        for (size_t j = 0; j < cnt; ++j) {
            SrvItem& it = s->active[kv.second[j]];
            b.ks[j] = std::min(s->quantum, it.total - it.done);
            m2k::SmallTest t = it.ctx->h_test;
            t.iters = b.ks[j];
            t.fuse_middle = fuse ? 1 : 0;
            if (tuned) t.carry_threads = small_carry_threads(it.ctx->L, it.ctx->span, threads, tn.carry_shift);
            t.status = b.d_status + j;
            b.h_tests[j] = t;
        }
        cudaError_t e = cudaStreamWaitEvent(b.stream, s->small_ready, 0);
        if (e == cudaSuccess) e = cudaMemsetAsync(b.d_status, 0, cnt * sizeof(int), b.stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(b.d_tests, b.h_tests, cnt * sizeof(m2k::SmallTest), cudaMemcpyHostToDevice, b.stream);
        if (e != cudaSuccess) return fail_cuda("server descriptor upload", e);
        m2b::Board& board = m2b::Board::of(s->device);
        if (!b.run) {
            b.run = std::make_shared<m2b::Run>();
            b.run->stream = b.stream;
            board.add(b.run);
        }
        board.begin(*b.run, m2b::FREE);
        e = duo ? m2k::launch_duo(b.d_tests, (int)cnt, (unsigned)kv.first, 0u, b.stream, nullptr, 0, min_smem)
                : m2k::launch_small(b.d_tests, (int)cnt, (unsigned)kv.first, threads, 0u, b.stream, fuse, false, min_smem);
        const cudaError_t er = board.end(*b.run);
        if (e == cudaSuccess) e = er;
        if (e != cudaSuccess)
            return fail_cuda("server small-test launch", e);
        e = cudaMemcpyAsync(b.h_status, b.d_status, cnt * sizeof(int), cudaMemcpyDeviceToHost, b.stream);
        if (e == cudaSuccess) e = cudaEventRecord(b.ev, b.stream);
        if (e != cudaSuccess) return fail_cuda("server status readback", e);
        for (size_t j = 0; j < cnt; ++j) s->active[kv.second[j]].inflight = b.ks[j];
        b.busy = true;
        b.whole = min_smem != 0;
        s->launches++;
    }
    return M2_OK;
}

// accounts for every lane whose quantum has finished; *lanes = how many
int srv_harvest(m2_server* s, int* lanes, bool* busy_left) {
    *lanes = 0;
    *busy_left = false;
    for (auto& kv : s->buckets) {
        SrvBucket& b = kv.second;
        if (!b.busy) continue;
        const cudaError_t e = cudaEventQuery(b.ev);
        if (e == cudaErrorNotReady) { *busy_left = true; continue; }
        if (e != cudaSuccess) return fail_cuda("server small-test wait", e);
        b.busy = false;
        ++*lanes;
        for (size_t j = 0; j < b.members.size(); ++j) {
            auto f = s->active.find(b.members[j]);
            SrvItem& it = f->second;
            const uint32_t k = b.ks[j];
            it.inflight = 0;
            it.done += k;
            it.ctx->iteration += k;
            s->squarings += k;
            const int st = b.h_status[j] ? M2_ESTATE : M2_OK;
            if (st != M2_OK || it.done >= it.total) { srv_retire(s, it, st); s->active.erase(f); }
        }
        b.members.clear();
    }
    for (auto f = s->active.begin(); f != s->active.end();) {
        SrvItem& it = f->second;
        if (it.ctx->path != M2_PATH_LARGE || !it.inflight) { ++f; continue; }
        const cudaError_t e = cudaEventQuery(it.ev);
        if (e == cudaErrorNotReady) { *busy_left = true; ++f; continue; }
        if (e != cudaSuccess) return fail_cuda("server large-test wait", e);
        ++*lanes;
        it.done += it.inflight;
        s->squarings += it.inflight;
        it.inflight = 0;
        const int st = m2_sync(it.ctx);
        if (st != M2_OK || it.done >= it.total) { srv_retire(s, it, st); f = s->active.erase(f); }
        else ++f;
    }
    return M2_OK;
}

}  // namespace

extern "C" {

int m2_srv_create(m2_server** out, int device, uint64_t budget_bytes, uint32_t quantum) {
    if (!out || budget_bytes == 0) return M2_EINVAL;
    if (cudaSetDevice(device) != cudaSuccess) { cudaGetLastError(); return M2_EINVAL; }
    m2_server* s = new (std::nothrow) m2_server();
    if (!s) return M2_ENOMEM;
    s->device = device;
    s->budget = budget_bytes;
    s->quantum = quantum ? quantum : 1000;
    int smem = 0;
    if (cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || s->sms < 1) s->sms = 1;
    if (cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device) == cudaSuccess) s->smem_sm = (size_t)smem;
    cudaGetLastError();
    if (cudaStreamCreateWithFlags(&s->small_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&s->small_ready, cudaEventDisableTiming) != cudaSuccess) {
        m2_srv_destroy(s);
        return M2_ECUDA;
    }
    s->t0 = std::chrono::steady_clock::now();
    *out = s;
    return M2_OK;
}

int m2_srv_submit(m2_server* s, uint64_t id, uint32_t p, int mode, uint32_t iters) {
    if (!s || p < 3 || mode < M2_MODE_LL || mode > M2_MODE_PRP3) return M2_EINVAL;
    if (m2::transform_log2(p) > 30) return M2_EUNSUPPORTED;
    SrvItem it;
    it.id = id; it.p = p; it.mode = mode;
    const uint32_t full = total_iters_for(p, mode);
    it.total = iters ? std::min(iters, full) : full;
    it.bytes = srv_estimate(p);
    if (it.bytes > s->budget) return M2_ENOMEM;   // could never be admitted: refused, not queued
    it.t_submit = s->now();
    s->queue.push_back(it);
    return M2_OK;
}

int m2_srv_step(m2_server* s) {
    if (!s) return M2_EINVAL;
    if (cudaSetDevice(s->device) != cudaSuccess) return M2_ECUDA;
    // admission: FIFO while the next test fits the budget
    while (!s->queue.empty() && s->resident + s->queue.front().bytes <= s->budget) {
        SrvItem it = s->queue.front();
        s->queue.pop_front();
        m2_opts o{};
        o.device = s->device;
        // up to h = 8192 a test joins its size's shared one-CTA launch
        o.path = (m2::transform_log2(it.p) <= 14) ? M2_PATH_SMALL : M2_PATH_LARGE;
        if (o.path == M2_PATH_SMALL) o.stream = s->small_stream;
        const int rc = m2_create(&it.ctx, it.p, it.mode, &o);
        // lanes share the GPU: the passes with the fields in turn, whose CTAs
        // wait for nothing (us a squaring, 8 tests of n = 2^19 25.9 -> 23.6, 4 of
        // 2^20 58.4 -> 52.4, one test alone 44.2 -> 36.6 and 79 -> 66.6)
        if (rc == M2_OK && it.ctx->path == M2_PATH_LARGE && it.ctx->plan.R == 256u && it.ctx->fused) {
            it.ctx->plan.in_turn = 1u;
            it.ctx->fused = false;
        }
        it.t_admit = s->now();
        s->resident += it.bytes;
        if (rc != M2_OK) { it.ctx = nullptr; srv_retire(s, it, rc); continue; }
        // from now on the test holds what its context allocated (shared tables excluded)
        const uint64_t own = it.ctx->bytes - it.ctx->tw.bytes;
        s->resident = s->resident - it.bytes + own;
        it.bytes = own;
        if (it.total == 0) { srv_retire(s, it, M2_OK); continue; }
        if (it.ctx->path == M2_PATH_LARGE) {
            const cudaError_t e = cudaEventCreateWithFlags(&it.ev, cudaEventDisableTiming);
            if (e != cudaSuccess) { srv_retire(s, it, fail_cuda("server event", e)); continue; }
        }
        s->active.emplace(s->next_key++, it);
    }
    if (s->active.empty()) return M2_OK;
    s->steps++;
    const cudaError_t er = cudaEventRecord(s->small_ready, s->small_stream);
    if (er != cudaSuccess) return fail_cuda("server setup event", er);
    int rc = srv_launch(s);
    if (rc) return rc;
    // wait until a lane finishes (polling; bounded)
    const auto t_start = std::chrono::steady_clock::now();
    for (;;) {
        int lanes = 0;
        bool busy = false;
        if ((rc = srv_harvest(s, &lanes, &busy))) return rc;
        if (lanes > 0 || !busy) return M2_OK;
        if (std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count() > SRV_WAIT_LIMIT_S) {
            std::snprintf(g_last_error, sizeof(g_last_error), "m2_srv_step: no lane finished within %.0f s", SRV_WAIT_LIMIT_S);
            return M2_ETIMEOUT;
        }
        std::this_thread::sleep_for(std::chrono::microseconds(50));
    }
}

int m2_srv_poll(m2_server* s, m2_srv_result* out, int max, int* n_out) {
    if (!s || (!out && max > 0)) return M2_EINVAL;
    int n = 0;
    while (n < max && !s->finished.empty()) { out[n++] = s->finished.front(); s->finished.pop_front(); }
    if (n_out) *n_out = n;
    return M2_OK;
}

int m2_srv_stats_get(m2_server* s, m2_srv_stats* st) {
    if (!s || !st) return M2_EINVAL;
    st->queued = (uint32_t)s->queue.size();
    st->active = (uint32_t)s->active.size();
    st->resident_bytes = s->resident;
    st->budget_bytes = s->budget;
    st->squarings = s->squarings;
    st->completed = s->completed;
    st->steps = s->steps;
    st->launches = s->launches;
    return M2_OK;
}

int m2_srv_active_get(m2_server* s, m2_srv_progress* out, int max, int* n_out) {
    if (!s || (!out && max > 0)) return M2_EINVAL;
    int n = 0;
    for (const auto& kv : s->active) {
        if (n >= max) break;
        const SrvItem& it = kv.second;
        m2_srv_progress& g = out[n++];
        g.id = it.id; g.p = it.p; g.done = it.done; g.total = it.total; g.inflight = it.inflight;
        g.n = it.ctx ? it.ctx->L.n : 0;
        g.device_bytes = it.bytes;
        g.t_submit = it.t_submit; g.t_admit = it.t_admit;
    }
    if (n_out) *n_out = n;
    return M2_OK;
}

void m2_srv_destroy(m2_server* s) {
    if (!s) return;
    cudaSetDevice(s->device);
    for (auto& kv : s->buckets)
        if (kv.second.stream) cudaStreamSynchronize(kv.second.stream);
    for (auto& kv : s->active) {
        if (kv.second.ctx) { m2_sync(kv.second.ctx); m2_destroy(kv.second.ctx); }
        if (kv.second.ev) cudaEventDestroy(kv.second.ev);
    }
    for (auto& kv : s->buckets) {
        SrvBucket& b = kv.second;
        if (b.run) m2b::Board::of(s->device).remove(b.run);
        cudaFree(b.d_tests); cudaFree(b.d_status); cudaFreeHost(b.h_tests); cudaFreeHost(b.h_status);
        if (b.ev) cudaEventDestroy(b.ev);
        if (b.stream) cudaStreamDestroy(b.stream);
    }
    if (s->small_ready) cudaEventDestroy(s->small_ready);
    if (s->small_stream) cudaStreamDestroy(s->small_stream);
    delete s;
}

}  // extern "C"
