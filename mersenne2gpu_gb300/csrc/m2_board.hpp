// m2_board.hpp -- what the contexts, servers and batches of this process have in
// flight on a device, and which kernels a new run takes beside it.
//
// How kernels share the GPU, as measured on a GB300:
//  - A cooperative grid starts all its CTAs at one instant, once there is room
//    for all (128 CTAs beside 100 CTAs that ended one by one: none before the
//    76th had).  Runs of one-launch kernels (m2_flow.cu, m2_tide.cu) on several
//    streams therefore alternate launch by launch by themselves: 2000
//    squarings of n = 2^21 beside 20000 are done after 0.42 of 2.28 s.
//  - Kernels that wait for nothing get on beside a one-launch kernel on the 24
//    SMs that m2_flow.cu leaves (2000 squarings of n = 2^16: 60 ms for 36), but
//    m2_tide.cu leaves none: one pass of three per launch of 26 ms and more.
//  - A batch holds its SMs to its end: beside 100 of them a one-launch kernel
//    of n = 2^16 does not begin (2.6 s), 500 squarings in passes take 11 ms.
//  - The fused column kernels spin on CTAs that may not have started, with a limit:
//    never beside a one-launch kernel.
//  - Tests of n <= 2^18 are faster together in passes once there are three: us a
//    squaring in all, 4 and 16 tests, one-launch in turns against passes:
//    2^15 8.3, 8.3 / 4.4, 1.8; 2^16 9.3, 9.3 / 5.4, 3.0; 2^17 9.7, 9.7 / 8.2,
//    6.0; 2^18 15.3, 15.3 / 13.0, 11.1; two tests 8.3 / 8.3, 9.3 / 9.5, 9.7 /
//    11.4, 15.3 / 17.8; n = 2^19 and 2^20 within 8% either way.
#pragma once
#include <chrono>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include <cuda_runtime_api.h>

namespace m2b {

// ONE: one-launch kernels; FUSED: passes with CTAs that wait for each other; FREE:
// kernels that wait for nothing; BATCH: persistent CTAs for seconds and minutes
enum Kind { ONE, FUSED, FREE, BATCH };

struct Run {
    int device = 0;
    cudaStream_t stream = nullptr;    // runs on one stream follow each other
    bool large = false;               // a context of n >= 2^14
    bool whole = false;               // its one-launch kernel takes every SM
    bool crowds = false;              // faster in passes beside two others (n <= 2^18)
    volatile unsigned* yield = nullptr;   // host word that calls off its queued one-launch kernels
    // under the board's lock:
    const void* group = nullptr;      // runs of one group follow each other too, by their owner's events
    unsigned kinds = 0;               // of what it may have in flight: bits 1 << Kind
    int starting = 0;                 // calls between begin and end
    bool recorded = false;            // `end` follows its last run
    cudaEvent_t end = nullptr;
};

class Board {
public:
    static Board& of(int device) {
        static std::mutex mu;
        static std::map<int, std::unique_ptr<Board>> all;
        std::lock_guard<std::mutex> lk(mu);
        std::unique_ptr<Board>& b = all[device];
        if (!b) b.reset(new Board());
        return *b;
    }
    void add(const std::shared_ptr<Run>& r) {
        std::lock_guard<std::mutex> lk(mu_);
        runs_.push_back(r);
        left_.reserve(runs_.size());
    }
    // its owner goes; work still in flight counts until it is done
    void remove(const std::shared_ptr<Run>& r) {
        Relaxed x;
        std::lock_guard<std::mutex> lk(mu_);
        r->stream = nullptr;
        r->group = nullptr;
        r->starting = 0;
        left_.push_back(r);
        for (size_t i = 0; i < left_.size();) {
            if (in_flight(*left_[i])) { ++i; continue; }
            if (left_[i]->end) cudaEventDestroy(left_[i]->end);
            for (size_t k = 0; k < runs_.size(); ++k)
                if (runs_[k] == left_[i]) { runs_[k] = runs_.back(); runs_.pop_back(); break; }
            left_[i] = left_.back();
            left_.pop_back();
        }
    }
    void group(Run& a, Run& b, const void* id) {
        std::lock_guard<std::mutex> lk(mu_);
        a.group = b.group = id;
    }
    // The kernels a run takes that would take `want` alone.  It counts as in
    // flight from here on; again() looks anew for the rest of a long call.
    Kind begin(Run& r, Kind want) {
        Relaxed x;
        std::lock_guard<std::mutex> lk(mu_);
        if (!r.starting) in_flight(r);   // drops the kinds of runs that are done
        ++r.starting;
        return choose(r, want);
    }
    Kind again(Run& r, Kind want) {
        Relaxed x;
        std::lock_guard<std::mutex> lk(mu_);
        return choose(r, want);
    }
    // its work is on the stream (the event is recorded outside the lock: a full
    // stream would block every other context)
    cudaError_t end(Run& r) {
        cudaError_t e = cudaSuccess;
        {
            Relaxed x;
            if (!r.end) e = cudaEventCreateWithFlags(&r.end, cudaEventDisableTiming);
        }
        if (e == cudaSuccess) e = cudaEventRecord(r.end, r.stream);
        std::lock_guard<std::mutex> lk(mu_);
        --r.starting;
        r.recorded = e == cudaSuccess;
        return e;
    }
    void done(Run& r) {   // nothing of it is in flight any more
        std::lock_guard<std::mutex> lk(mu_);
        --r.starting;
    }

private:
    // events may be asked about and made while another thread captures a stream
    struct Relaxed {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
        ~Relaxed() {
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (cudaPeekAtLastError() == cudaErrorNotReady) cudaGetLastError();
        }
    };
    static bool in_flight(Run& o) {
        if (o.starting) return true;
        if (o.recorded && cudaEventQuery(o.end) != cudaErrorNotReady) o.recorded = false;
        if (!o.recorded) o.kinds = 0;
        return o.recorded;
    }
    Kind choose(Run& r, Kind want) {
        using clock = std::chrono::steady_clock;
        int one = 0, fused = 0, free_large = 0, free_small = 0, batch = 0;
        for (const auto& p : runs_) {
            Run& o = *p;
            if (&o == &r || (o.stream && o.stream == r.stream) || (o.group && o.group == r.group)) continue;
            if (want == FREE && !(o.kinds & 1u << ONE)) continue;
            if (!in_flight(o)) continue;
            if (o.kinds & 1u << ONE) ++one;
            else if (o.kinds & 1u << BATCH) ++batch;
            else if (o.kinds & 1u << FUSED) ++fused;
            else ++(o.large ? free_large : free_small);
        }
        Kind k = want;
        if (want == ONE) {
            // (three at once a moment ago: a program with many contexts, whose next round begins)
            if (r.crowds && one + fused + free_large >= 2) crowded_until_ = clock::now() + std::chrono::milliseconds(200);
            if (fused || batch || free_large || (r.whole && free_small) || (r.crowds && clock::now() < crowded_until_)) k = FREE;
        } else if (want == FUSED && (one || batch)) {
            k = FREE;
        }
        r.kinds |= 1u << k;
        if (k == ONE) {
            if (r.yield) *r.yield = 0;
        } else if (one) {
            // queued one-launch kernels would keep this run off the GPU
            for (const auto& p : runs_)
                if ((p->kinds & 1u << ONE) && p->yield && p.get() != &r && (p->whole || r.large || k == BATCH) &&
                    !(p->stream && p->stream == r.stream) && !(p->group && p->group == r.group))
                    *p->yield = 1;
        }
        return k;
    }
    std::mutex mu_;
    std::vector<std::shared_ptr<Run>> runs_, left_;
    std::chrono::steady_clock::time_point crowded_until_{};
};

}  // namespace m2b
