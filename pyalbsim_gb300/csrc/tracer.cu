// Tracer kernels: one wave of warps, each keeping its lanes supplied with photons of its share.
#include <algorithm>

#include "device_common.cuh"
#include "internal.h"
#include "tracer.cuh"
#include "tracer_fast.cuh"

namespace alb {

constexpr int kTraceThreads = 128;
// Lanes of a warp whose photons are done wait until `refill` of them take new photons together, and
// lanes at a surface or seafloor crossing until `batch` of them cross together. One photon per lane
// and launch left 10 of 32 lanes active: a photon makes 38 events on average and three times that
// at the longest of 32, and a warp met a crossing, most of the code, in nearly every step with one
// or two lanes. Forward trace of 1e6 photons of the large scene: 2.96 -> 1.76 ms, 17 lanes active
// (refill 8, batch 4; batch 6: 1.77, 8: 1.79; refill 12: 1.87).
struct LaneRule {
    int refill, batch;
};

// One warp's photons [next, end).
template <class Lane>
ALB_DEVICE void trace_warp(Lane& lane, uint64_t next, uint64_t end, LaneRule rule) {
    constexpr unsigned kAll = 0xffffffffu;
    int mode = kLaneDone;
    uint64_t mine = 0;
    while (true) {
        const unsigned idle = __ballot_sync(kAll, mode == kLaneDone);
        if (next < end && __popc(idle) >= rule.refill) {
            const uint64_t i = next + __popc(idle & lanemask_lt());
            if (mode == kLaneDone && i < end) {
                mine = i;
                mode = lane.start(i);
                if (mode == kLaneDone) lane.finish(i);
            }
            next += __popc(idle);
            __syncwarp();
        } else if (idle == kAll) {
            break;  // nothing is left: with photons to take, 32 idle lanes refill
        }
        // a kind of crossing runs once enough lanes wait for it, or when no lane is under way
        const bool stuck = !__any_sync(kAll, mode == kLaneRun) && !(next < end && __popc(__ballot_sync(kAll, mode == kLaneDone)) >= rule.refill);
        auto cross = [&](int kind, auto&& handler) {
            const unsigned b = __ballot_sync(kAll, mode == kind);
            if (b && (stuck || __popc(b) >= rule.batch)) {
                if (mode == kind) {
                    mode = handler();
                    if (mode == kLaneDone) lane.finish(mine);
                }
                __syncwarp();
            }
        };
        cross(kLaneAir, [&]() { return lane.air(); });
        cross(kLaneExit, [&]() { return lane.exit(); });
        cross(kLaneFloor, [&]() { return lane.floor(); });
        if (mode == kLaneRun) {
            mode = lane.run();
            if (mode == kLaneDone) lane.finish(mine);
        }
        __syncwarp();
    }
}

ALB_DEVICE void warp_range(uint64_t n, uint64_t& r0, uint64_t& r1) {
    const uint64_t warps = (uint64_t)gridDim.x * (kTraceThreads / 32), w = (uint64_t)blockIdx.x * (kTraceThreads / 32) + threadIdx.x / 32;
    r0 = n * w / warps;
    r1 = n * (w + 1) / warps;
}

// warp-reduce the event counters, one atomic per warp
ALB_DEVICE void count_events(const TraceOut& out, unsigned long long events, unsigned long long done) {
    for (int o = 16; o > 0; o >>= 1) {
        events += __shfl_xor_sync(0xffffffffu, events, o);
        done += __shfl_xor_sync(0xffffffffu, done, o);
    }
    if ((threadIdx.x & 31) == 0 && out.stats) {
        atomicAdd(out.stats, events);
        atomicAdd(out.stats + 1, done);
    }
}

template <int PASS, bool REPLAY>
__global__ void __launch_bounds__(kTraceThreads) k_trace(const __grid_constant__ SceneDev sc,
                                                         const __grid_constant__ TraceOut out, uint64_t n, uint64_t first,
                                                         uint32_t k0, uint32_t k1, const int64_t* __restrict__ offs,
                                                         const double* __restrict__ vals,
                                                         const float* __restrict__ taus, LaneRule rule) {
    uint64_t r0, r1;
    warp_range(n, r0, r1);
    if (REPLAY) {
        PreciseLane<PASS, ReplaySrc> lane{sc, out, first, offs, ReplaySrc{vals, taus, 0, 0, out.err}};
        trace_warp(lane, r0, r1, rule);
        count_events(out, lane.events, lane.done);
    } else {
        PreciseLane<PASS, PhiloxSrc> lane{sc, out, first, offs, PhiloxSrc{k0, k1, 0u, 0u, (uint32_t)PASS, 0u}};
        trace_warp(lane, r0, r1, rule);
        count_events(out, lane.events, lane.done);
    }
}

template <int PASS>
__global__ void __launch_bounds__(kTraceThreads) k_trace_fast(const __grid_constant__ SceneDev sc,
                                                              const __grid_constant__ FastScene fs,
                                                              const __grid_constant__ TraceOut out, uint64_t n,
                                                              uint64_t first, uint32_t k0, uint32_t k1, LaneRule rule) {
    uint64_t r0, r1;
    warp_range(n, r0, r1);
    FastLane<PASS> lane{sc, fs, out, first, PhiloxSrc{k0, k1, 0u, 0u, (uint32_t)PASS, 0u}};
    trace_warp(lane, r0, r1, rule);
    count_events(out, lane.events, lane.done);
}

// Tables of one layer's phase function at u = j / kInvCdf: theta(u) (numpy.interp restated) for the
// float32 tracer, and the interval of the CDF table that holds u.
__global__ void k_phase_tables(const double* __restrict__ cdf, const double* __restrict__ theta,
                               const double* __restrict__ slope, float* inv, uint16_t* guide) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j > kInvCdf) return;
    const int n = ALB_PHASE_DIVISIONS;
    const double u = (double)j / kInvCdf;
    int lo = 0, hi = n - 1;
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (cdf[mid] <= u) lo = mid; else hi = mid;
    }
    double t;
    if (u < cdf[0]) t = theta[0];
    else if (u >= cdf[n - 1]) t = theta[n - 1];
    else t = (u == cdf[lo]) ? theta[lo] : fma(slope[lo], u - cdf[lo], theta[lo]);
    inv[j] = (float)t;
    guide[j] = (uint16_t)lo;
}

void launch_phase_tables(const double* cdf, const double* theta, const double* slope, float* inv, uint16_t* guide,
                         cudaStream_t st) {
    k_phase_tables<<<(kInvCdf + 256) / 256, 256, 0, st>>>(cdf, theta, slope, inv, guide);
    note_launch();
}

// Logarithms of the exponential profiles' ends, as the device forms them.
__global__ void k_profile_logs(SceneDev sc, double* out) {
    const int l = threadIdx.x;
    if (l >= sc.n_layers) return;
    const double nl = log(sc.layer_n0[l]), al = log(sc.layer_a0[l]);
    out[4 * l] = nl;
    out[4 * l + 1] = log(sc.layer_n1[l]) - nl;
    out[4 * l + 2] = al;
    out[4 * l + 3] = log(sc.layer_a1[l]) - al;
}

void launch_profile_logs(const SceneDev& sc, double* out, cudaStream_t st) {
    k_profile_logs<<<1, 32, 0, st>>>(sc, out);
    note_launch();
}

void launch_trace(const SceneDev& sc, const TraceOut& out, int pass, uint64_t n, uint64_t first_photon,
                  uint64_t seed, const AlbReplay* rp, int* launches, cudaStream_t st, const FastScene* fast) {
    if (n == 0) return;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // One wave of resident blocks, each warp with its share of the photons. The float64 tracer and
    // depth-profiled water (a float64 table lookup per step) keep the two FP64 lanes of an SM busy
    // with a few warps: fewer, fuller warps spend fewer instructions (200 000 photons of the large
    // scene, float64, two launches: 2 blocks per SM 24.4 ms, 3 25.5, 4 26.8, all 27.8; 200 003 photons
    // of profiled water: 4 blocks 10.0 ms, all 12.6). Profiled water makes a hundred steps per
    // crossing, so waiting for a crossing costs more there.
    bool profiled = false;
    for (int l = 0; l < sc.n_layers; ++l) profiled = profiled || sc.layer_prof[l];
    const bool f32 = fast && !rp;
    const int most = !f32 ? 2 : (profiled ? 4 : 32);
    const LaneRule rule = profiled ? LaneRule{4, 2} : LaneRule{8, 4};
    auto grid = [&](auto kernel) {
        int per_sm = 2;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTraceThreads, 0);
        const uint64_t want = (n + kTraceThreads - 1) / kTraceThreads;
        return (unsigned)std::min(want, (uint64_t)sms * std::max(std::min(per_sm, most), 1));
    };
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
    if (f32) {
        if (pass == ALB_FORWARD) k_trace_fast<ALB_FORWARD><<<grid(k_trace_fast<ALB_FORWARD>), kTraceThreads, 0, st>>>(sc, *fast, out, n, first_photon, k0, k1, rule);
        else k_trace_fast<ALB_BACKWARD><<<grid(k_trace_fast<ALB_BACKWARD>), kTraceThreads, 0, st>>>(sc, *fast, out, n, first_photon, k0, k1, rule);
        note_launch();
        if (launches) ++*launches;
        return;
    }
    const int64_t* offs = rp ? rp->offsets : nullptr;
    const double* vals = rp ? rp->values : nullptr;
    const float* taus = rp ? rp->tau : nullptr;
    if (pass == ALB_FORWARD) {
        if (rp) k_trace<ALB_FORWARD, true><<<grid(k_trace<ALB_FORWARD, true>), kTraceThreads, 0, st>>>(sc, out, n, first_photon, k0, k1, offs, vals, taus, rule);
        else k_trace<ALB_FORWARD, false><<<grid(k_trace<ALB_FORWARD, false>), kTraceThreads, 0, st>>>(sc, out, n, first_photon, k0, k1, offs, vals, taus, rule);
    } else {
        if (rp) k_trace<ALB_BACKWARD, true><<<grid(k_trace<ALB_BACKWARD, true>), kTraceThreads, 0, st>>>(sc, out, n, first_photon, k0, k1, offs, vals, taus, rule);
        else k_trace<ALB_BACKWARD, false><<<grid(k_trace<ALB_BACKWARD, false>), kTraceThreads, 0, st>>>(sc, out, n, first_photon, k0, k1, offs, vals, taus, rule);
    }
    note_launch();
    if (launches) ++*launches;
}

}  // namespace alb
