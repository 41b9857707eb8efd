// capi_internal.h -- what the C ABI's translation units share: error
// reporting, the device guard, host record transfers, scene constants, the
// task-size autotuner and the batch handle (capi.cu: simulator and scene
// builders; capi_batch.cu: batches; capi_adjoint.cu: differentiation).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/mpm.h"
#include "mpm_internal.h"
#include "sorted_engine.h"

namespace mpm {

// The message mpm_last_error() returns (capi.cu).
void set_last_error(const std::string& msg);

inline int fail(int code, const std::string& msg) {
    set_last_error(msg);
    return code;
}

inline int cuda_fail(cudaError_t e, const char* what) {
    return fail(MPM_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define MPM_CUDA(call)                                   \
    do {                                                 \
        cudaError_t e_ = (call);                         \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call); \
    } while (0)

// Switches to the handle's device for the duration of a call.
struct DeviceGuard {
    int prev = -1;
    bool ok = true;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) { ok = false; return; }
        if (prev != dev && cudaSetDevice(dev) != cudaSuccess) ok = false;
    }
    ~DeviceGuard() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

// Host 80-byte records <-> device particle streams through a staging buffer
// (capi.cu).
cudaError_t upload_records(const Particles& dst, const float* host, int n, float* stage,
                           cudaStream_t st);
cudaError_t download_records(const Particles& src, float* host, int n, float* stage,
                             cudaStream_t st);

// WGSL i32(f32): truncation toward zero, saturating, NaN -> 0 (capi.cu).
int f2i_trunc_sat(float x);
// mls-mpm.ts:229 gridCount (capi.cu).
long long grid_count_of(const float b[3]);
// SimConsts of one scene; MPM_OK or an error for an unusable description
// (capi_batch.cu).
int scene_consts(const mpm_scene_desc& d, SimConsts& k);

// Times `substeps` sorted-engine substeps for each combination of z-pair
// threshold, task-kernel block size, task size and lane-table threshold from
// the same saved state; then, over five times as many, the fastest of them and
// the other lane-table thresholds of the fastest of those, and keeps the fastest
// by that timing.  Each candidate first runs once untimed, so that
// the CUDA graphs the timed run replays are captured outside it.  The state
// after the call is the state before it (particles, posvel, counters, grid).
template <class StepFn>
int tune_engine(SortedEngine* e, ParticleStore& ps, int n, float4* posvel,
                unsigned long long* counters, int substeps, cudaStream_t st, StepFn step,
                int* chosen, int* chosen_lane, double* ms_out, int* chosen_threads = nullptr) {
    static const int kPairs[] = {0, 256, 512, 1 << 30};
    static const int kThreads[] = {128, 256, 512};
    static const int kCaps[] = {128, 256, 512, 1024};
    static const int kLanes[] = {32, 128, 512, 1 << 30};  // 1 << 30: no lane table
    Particles save{};
    float4* pv = nullptr;
    unsigned long long cnt[2] = {0, 0};
    cudaEvent_t a = nullptr, b = nullptr;
    auto cleanup = [&]() {
        cudaFree(save.p0); cudaFree(save.p1); cudaFree(save.p2); cudaFree(save.p3);
        cudaFree(pv);
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    };
    cudaError_t err = cudaSuccess;
    float4** sp[4] = {&save.p0, &save.p1, &save.p2, &save.p3};
    for (int q = 0; q < 4 && err == cudaSuccess; ++q) err = cudaMalloc(sp[q], sizeof(float4) * (size_t)(n ? n : 1));
    if (err == cudaSuccess) err = cudaMalloc(&pv, sizeof(float4) * 2 * (size_t)(n ? n : 1));
    if (err == cudaSuccess) err = cudaEventCreate(&a);
    if (err == cudaSuccess) err = cudaEventCreate(&b);
    if (err == cudaSuccess) err = cudaMemcpy(cnt, counters, sizeof(cnt), cudaMemcpyDeviceToHost);
    // canonical snapshot of the state
    if (err == cudaSuccess) {
        const int c = ps.cur;
        if (ps.canonical) {
            const float4* src[4] = {ps.P[c].p0, ps.P[c].p1, ps.P[c].p2, ps.P[c].p3};
            for (int q = 0; q < 4 && err == cudaSuccess; ++q)
                err = cudaMemcpyAsync(*sp[q], src[q], sizeof(float4) * (size_t)n, cudaMemcpyDeviceToDevice, st);
        } else {
            launch_canonicalize(ps.P[c], ps.id[c], save, nullptr, n, st);
            err = cudaGetLastError();
        }
    }
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(pv, posvel, sizeof(float4) * 2 * (size_t)n, cudaMemcpyDeviceToDevice, st);
    auto restore = [&]() -> cudaError_t {
        ps.cur = 0;
        ps.canonical = true;
        const float4* src[4] = {save.p0, save.p1, save.p2, save.p3};
        float4* dst[4] = {ps.P[0].p0, ps.P[0].p1, ps.P[0].p2, ps.P[0].p3};
        for (int q = 0; q < 4; ++q) {
            cudaError_t e2 = cudaMemcpyAsync(dst[q], src[q], sizeof(float4) * (size_t)n, cudaMemcpyDeviceToDevice, st);
            if (e2 != cudaSuccess) return e2;
        }
        launch_iota(ps.id[0], n, st);
        sorted_invalidate(e);
        return cudaGetLastError();
    };
    struct Choice {
        int pair, threads, cap, lane;
        float ms;
    };
    // Time of `windows` calls in a row from the saved state, after an untimed
    // pass that captures their graphs; false: not a choice, or an error (err).
    auto time_choice = [&](Choice& c, int windows) {
        if (sorted_set_pair_max(e, c.pair) != 0 || sorted_set_threads(e, c.threads) != 0 ||
            sorted_set_task_cap(e, c.cap) != 0 || sorted_set_lane_table_min(e, c.lane) != 0)
            return false;
        for (int timed = 0; timed < 2; ++timed) {
            if ((err = restore()) != cudaSuccess) return false;
            if (step(1) != 0) { err = cudaErrorLaunchFailure; return false; }  // primes
            cudaEventRecord(a, st);
            for (int w = 0; w < windows; ++w)
                if (step(substeps) != 0) { err = cudaErrorLaunchFailure; return false; }
            cudaEventRecord(b, st);
        }
        if ((err = cudaEventSynchronize(b)) != cudaSuccess) return false;
        cudaEventElapsedTime(&c.ms, a, b);
        return true;
    };
    // Every combination over one window; then the fastest of them (with their
    // best lane-table threshold) over five, because what suits the state of the
    // moment may not suit the next ones: a million particles falling from a
    // lattice, 128 threads and tasks of 1,024 are the fastest over 8 substeps,
    // when there are no more tasks than CTAs, and 509 us a frame against 416 over
    // the next 20 frames.
    constexpr int kWindows = 5;
    constexpr size_t kFinalists = 12;
    const auto faster = [](const Choice& x, const Choice& y) { return x.ms < y.ms; };
    std::vector<Choice> found;
    for (int pair : kPairs)
    for (int th : kThreads)
    for (int cap : kCaps) {
        Choice best_of{0, 0, 0, 0, 0.f};
        for (int lane : kLanes) {
            if (err != cudaSuccess) break;
            Choice c{pair, th, cap, lane, 0.f};
            if (time_choice(c, 1) && (!best_of.cap || faster(c, best_of))) best_of = c;
        }
        if (best_of.cap) found.push_back(best_of);
    }
    std::stable_sort(found.begin(), found.end(), faster);
    if (found.size() > kFinalists) found.resize(kFinalists);
    Choice best{0, 0, 0, 0, 0.f};
    auto keep_faster = [&](Choice c) {
        if (err == cudaSuccess && time_choice(c, kWindows) && (!best.cap || faster(c, best))) best = c;
    };
    for (const Choice& c : found) keep_faster(c);
    // the lane-table threshold too by the longer timing
    const Choice first = best;
    for (int lane : kLanes)
        if (first.cap && lane != first.lane) keep_faster({first.pair, first.threads, first.cap, lane, 0.f});
    if (err == cudaSuccess) err = restore();
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(posvel, pv, sizeof(float4) * 2 * (size_t)n, cudaMemcpyDeviceToDevice, st);
    if (err == cudaSuccess) err = cudaMemcpyAsync(counters, cnt, sizeof(cnt), cudaMemcpyHostToDevice, st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(st);
    cleanup();
    if (err != cudaSuccess) return cuda_fail(err, "autotune");
    if (best.cap) {
        sorted_set_pair_max(e, best.pair);
        sorted_set_threads(e, best.threads);
        sorted_set_task_cap(e, best.cap);
        sorted_set_lane_table_min(e, best.lane);
    }
    if (chosen) *chosen = best.cap;
    if (chosen_lane) *chosen_lane = best.lane;
    if (chosen_threads) *chosen_threads = best.threads;
    if (ms_out) *ms_out = (double)best.ms / kWindows;
    return MPM_OK;
}

}  // namespace mpm

struct mpm_batch {
    int device = 0;
    std::vector<mpm_scene_desc> desc;
    std::vector<mpm::SimConsts> consts;
    std::vector<long long> first;  // first particle of each scene
    int n = 0;
    mpm::ParticleStore ps{};
    float4* posvel = nullptr;
    unsigned long long* counters = nullptr;  // [0] out-of-range, [1] non-finite scratch
    mpm::SortedEngine* sorted = nullptr;
    bool graph = true;
    bool stepped = false;
    // order between scenes' new constants, copied on the null stream, and work on
    // other streams: work that a copy has to wait for, copies that work has to
    // wait for, and whether steps were captured (their replays are not seen here)
    bool in_flight = false, copies = false, captured = false;
    mpm::LaunchProfiler prof;
};

namespace mpm {
int check_batch(const mpm_batch* b);  // capi_batch.cu
cudaError_t after_scene_copies(mpm_batch* b, cudaStream_t st);
}  // namespace mpm
