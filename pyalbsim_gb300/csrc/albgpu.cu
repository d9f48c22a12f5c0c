// C ABI of the GB300 photon-tracing / photon-mapping engine (declared in include/albgpu.h).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <unordered_set>
#include <vector>

#include "albgpu.h"
#include "internal.h"
#include "tracer_fast.cuh"

using namespace alb;

#include <atomic>
static std::atomic<long long> g_launches{0};
namespace alb {
void set_global_error(const std::string& msg);
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
long long launches_total() { return g_launches.load(); }
}  // namespace alb

// ------------------------------------------------------------------------------------------
// Workspace
// ------------------------------------------------------------------------------------------

// Device memory of every context comes from one pool per device, stream ordered, so that a context
// made for one run and destroyed after it (run_linear, the batch's workers) does not map and unmap
// its gigabytes each time and never stalls the device for another worker's stream. The pool
// keeps at most an eighth of the device that nobody holds; what is over goes back to the driver at
// the next synchronisation, alb_trim_memory gives back the rest, and so does a cudaMalloc that would
// fail otherwise (measured: 160 GB beside 160 GB idle in the pool). Blocks over kDirect are cudaMalloc's: a pool
// maps 16 GB in 13 ms, cudaMalloc in 1 ms, and so large a block would not be kept anyway.
constexpr uint64_t kDirect = 16ull << 30;
// In a batch's worker threads: blocks over 1 GB. Workers fill the device with instances of many sizes, and
// a pool's blocks of one size do not serve the next (2 of 128 instances of the sweep ran out of memory).
constexpr uint64_t kDirectBatch = 1ull << 30;
static thread_local uint64_t t_direct = kDirect;

static std::mutex g_direct_mu;
static std::unordered_set<void*> g_direct;

static cudaMemPool_t device_pool() {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> g(mu);
    if (!pools[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        size_t idle = 0, all = 0;
        cudaMemGetInfo(&idle, &all);
        uint64_t keep = all / 8;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        pools[dev] = pool;
    }
    return pools[dev];
}

// Bytes the device's pool holds that nobody uses.
static uint64_t pool_idle() {
    uint64_t reserved = 0, used = 0;
    const cudaMemPool_t pool = device_pool();
    if (!pool || cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return reserved - used;
}

extern "C" int alb_trim_memory(int device) {
    int before = 0;
    if (cudaGetDevice(&before) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        set_global_error("alb_trim_memory: no such device");
        return ALB_ERR_INVALID;
    }
    const cudaMemPool_t pool = device_pool();
    const bool ok = pool && cudaMemPoolTrimTo(pool, 0) == cudaSuccess;
    cudaSetDevice(before);
    if (ok) return ALB_OK;
    cudaGetLastError();
    set_global_error("alb_trim_memory: the pool could not be trimmed");
    return ALB_ERR_CUDA;
}

namespace alb {
void* dev_alloc(uint64_t bytes, cudaStream_t st) {
    const cudaMemPool_t pool = device_pool();
    if (!pool) return nullptr;
    if (bytes == 0) bytes = 16;
    for (int attempt = 0; attempt < 3; ++attempt) {
        void* p = nullptr;
        if (bytes > t_direct) {
            if (cudaMalloc(&p, bytes) == cudaSuccess) {
                std::lock_guard<std::mutex> g(g_direct_mu);
                g_direct.insert(p);
                return p;
            }
        } else if (cudaMallocFromPoolAsync(&p, bytes, pool, st) == cudaSuccess) return p;
        cudaGetLastError();
        // again with every idle block given back to the driver: this stream's, then every stream's
        if (attempt == 0) cudaStreamSynchronize(st);
        else if (attempt == 1) cudaDeviceSynchronize();
        if (attempt < 2) cudaMemPoolTrimTo(pool, 0);
    }
    return nullptr;
}

void dev_free(void* p, cudaStream_t st) {
    if (!p) return;
    {
        std::unique_lock<std::mutex> g(g_direct_mu);
        if (g_direct.erase(p)) {
            g.unlock();
            cudaStreamSynchronize(st);
            cudaFree(p);
            return;
        }
    }
    cudaFreeAsync(p, st);
}
}  // namespace alb

template <class T>
static bool take(T*& p, uint64_t bytes, cudaStream_t st) {
    p = (T*)dev_alloc(bytes, st);
    return p != nullptr;
}

template <class T>
static void drop(T*& p, cudaStream_t st) {
    dev_free(p, st);
    p = nullptr;
}

Workspace::~Workspace() {
    for (void* p : temps_) dev_free(p, st_);
    dev_free(box_, st_);
}

void* Workspace::take_bytes(uint64_t bytes) {
    void* p = dev_alloc(bytes, st_);
    if (!p) {
        failed_ = true;
        return nullptr;
    }
    temps_.push_back(p);
    return p;
}

void Workspace::release(size_t m) {
    while (temps_.size() > m) {
        dev_free(temps_.back(), st_);
        temps_.pop_back();
    }
}

unsigned* Workspace::scratch_box() {
    if (!box_ && !(box_ = (unsigned*)dev_alloc(64 * sizeof(unsigned), st_))) failed_ = true;
    return box_;
}

static void* grow(void* old, uint64_t& cap, uint64_t n, size_t elem, bool& failed, cudaStream_t st) {
    if (cap >= n && old) return old;
    dev_free(old, st);
    uint64_t want = std::max<uint64_t>(n + n / 32, 256);
    void* p = dev_alloc(want * elem, st);
    if (!p) {
        failed = true;
        cap = 0;
        return nullptr;
    }
    cap = want;
    return p;
}

void* Workspace::alloc_persistent(void* old, uint64_t& cap, uint64_t n) { return grow(old, cap, n, 16, failed_, st_); }
void* Workspace::alloc_persistent_u32(void* old, uint64_t& cap, uint64_t n) { return grow(old, cap, n, 4, failed_, st_); }

// ------------------------------------------------------------------------------------------
// Context
// ------------------------------------------------------------------------------------------

struct AlbCtx {
    int device = 0;
    cudaStream_t st = 0;
    bool callers_stream = false;  // st came with ALB_OPT_STREAM
    SceneDev sc{};
    FastScene fast{};
    std::vector<void*> tables;
    Workspace ws;
    // forward records
    RecordStore rec[ALB_CHANNELS];
    uint64_t rec_id_cap[ALB_CHANNELS] = {0};
    uint64_t fwi_cap[ALB_CHANNELS] = {0}, sfi_cap[ALB_CHANNELS] = {0}, b_cap[ALB_CHANNELS] = {0};
    // one control block: record counts [0, 4), query counts [4, 7), error word and crowded channels [7], counters [8, 40),
    // counters kept across a retried trace [41, 43), the gathers' work counters [43, 47)
    unsigned long long* ctl = nullptr;
    unsigned long long* d_rec_count = nullptr;
    uint64_t h_rec_count[ALB_CHANNELS] = {0};
    double rec_rate[ALB_CHANNELS] = {2.0, 8.0, 1.05, 1.05};
    MapIndex map[ALB_CHANNELS];
    bool maps_built = false;
    // records of a channel live either in its append store or, once indexed, only in the
    // index (the store is released to make room; restored if more records are appended)
    bool rec_released[ALB_CHANNELS] = {false, false, false, false};
    // backward queries
    float4* qa[3] = {nullptr, nullptr, nullptr};
    float4* qb[3] = {nullptr, nullptr, nullptr};
    float4* qc[3] = {nullptr, nullptr, nullptr};
    uint32_t* qid[3] = {nullptr, nullptr, nullptr};
    float4* qs[3] = {nullptr, nullptr, nullptr};  // adjoint query scores
    uint32_t* qperm[3] = {nullptr, nullptr, nullptr};
    double* qrk[3][2] = {{nullptr, nullptr}, {nullptr, nullptr}, {nullptr, nullptr}};
    uint64_t qcap[3] = {0, 0, 0}, qcap_b[3] = {0}, qcap_c[3] = {0}, qid_cap[3] = {0}, qperm_cap[3] = {0};
    uint64_t qrk_cap[3][2] = {{0}};
    unsigned long long* d_q_count = nullptr;
    uint64_t h_q_count[3] = {0, 0, 0};
    double q_rate[3] = {2.0, 8.0, 1.05};
    bool rec_rate_known = false, q_rate_known = false;  // measured by a trace of this scene's context
    // accumulators
    unsigned long long* wf = nullptr;  // lo words then hi words, [2][channels][nbins]
    unsigned long long* hm = nullptr;  // sampled heatmaps, [2 maps][2 words][bins*bins]
    unsigned *hm_radius = nullptr, *hm_radius_bak = nullptr;  // the copies: before the call, before its second part
    // adjoint Jacobian: lo words then hi words, [2][kJacParams][channels][nbins]
    unsigned long long* jac = nullptr;
    // sums of one gather by exponent class (every gather leaves them zero)
    unsigned long long *cls = nullptr, *jac_cls = nullptr, *heat_cls = nullptr;
    int64_t cls_bins = 0, jac_cls_bins = 0, heat_cls_cells = 0;
    int64_t wf_bins = 0, jac_bins = 0, hm_cells = 0, hm_radius_cells = 0;  // accumulator capacities
    // per-layer scene tables (device), reused when the context takes a new scene
    struct LayerTables {
        void *th = nullptr, *cdf = nullptr, *sl = nullptr, *w = nullptr, *dlw = nullptr, *dsg = nullptr, *inv = nullptr,
             *guide = nullptr;
    } lt[ALB_MAX_LAYERS];
    bool keep_records = false;  // keep the append stores after indexing (batched runs)
    // exit states
    double* ex_pos = nullptr;
    double* ex_dir = nullptr;
    float* ex_f = nullptr;
    uint64_t ex_cap = 0, ex_n = 0;
    // misc
    int* d_err = nullptr;
    unsigned long long* d_stats = nullptr;
    int keep_exit = 0, keep_ids = 0, precise = 1, sort_q = 1;
    int64_t map_cap_hint = 0;
    int launches = 0;
    std::string err;
    // phase timing (CUDA events on the context's stream)
    double phase_ms[ALB_PHASES] = {0};
    int64_t phase_calls[ALB_PHASES] = {0};
    int64_t gathered[ALB_CHANNELS] = {0};
    // recorded phases whose times are read at the next synchronisation, and idle events
    struct Phase {
        int phase;
        cudaEvent_t e0, e1;
    };
    std::vector<Phase> pending;
    std::vector<cudaEvent_t> events;
    // streams of the small gathers, forked from and joined to st
    cudaStream_t side[3] = {};
    cudaEvent_t fork = nullptr, join[3] = {};
};

static cudaEvent_t take_event(AlbCtx* c) {
    cudaEvent_t e = nullptr;
    if (!c->events.empty()) {
        e = c->events.back();
        c->events.pop_back();
    } else {
        cudaEventCreate(&e);
    }
    return e;
}

// Time one phase between two events on its stream; the times are folded into the accumulators
// once the stream has drained (fold_phases).
struct PhaseTimer {
    AlbCtx* c;
    AlbCtx::Phase p;
    bool stopped = false;
    PhaseTimer(AlbCtx* ctx, int phase, cudaStream_t st) : c(ctx), p{phase, take_event(ctx), take_event(ctx)} {
        cudaEventRecord(p.e0, st);
    }
    PhaseTimer(AlbCtx* ctx, int phase) : PhaseTimer(ctx, phase, ctx->st) {}
    PhaseTimer(const PhaseTimer&) = delete;
    ~PhaseTimer() {  // a phase left on an error counts for nothing
        if (!stopped) c->events.insert(c->events.end(), {p.e0, p.e1});
    }
    void stop(cudaStream_t st) {
        cudaEventRecord(p.e1, st);
        c->phase_calls[p.phase] += 1;
        c->pending.push_back(p);
        stopped = true;
    }
    void stop() { stop(c->st); }
};

static void fold_phases(AlbCtx* c) {
    for (const auto& p : c->pending) {
        float ms = 0.f;
        if (cudaEventSynchronize(p.e1) == cudaSuccess && cudaEventElapsedTime(&ms, p.e0, p.e1) == cudaSuccess)
            c->phase_ms[p.phase] += ms;
        c->events.push_back(p.e0);
        c->events.push_back(p.e1);
    }
    c->pending.clear();
}

static int fail(AlbCtx* c, int code, const std::string& msg) {
    if (c) {
        c->err = msg;
        c->ws.clear_failed();  // this call has reported it
    }
    return code;
}

#define CK(call)                                                                                  \
    do {                                                                                          \
        cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess) return fail(ctx, ALB_ERR_CUDA, std::string(#call ": ") + cudaGetErrorString(e_)); \
    } while (0)

// Waits for the context's stream and reports what failed on it; counts (nullable) receives the
// record and query counts, crowded (nullable) the channels whose searches left queries.
static int check_device(AlbCtx* ctx, const char* where, unsigned long long* counts = nullptr, uint32_t* crowded = nullptr) {
    unsigned long long ctl[8] = {0};
    cudaError_t e = cudaMemcpyAsync(ctl, ctx->ctl, sizeof ctl, cudaMemcpyDeviceToHost, ctx->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->st);
    if (e == cudaSuccess) e = cudaGetLastError();
    fold_phases(ctx);
    if (e != cudaSuccess) return fail(ctx, ALB_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
    if (ctx->ws.failed()) {
        ctx->ws.clear_failed();
        return fail(ctx, ALB_ERR_CUDA, std::string(where) + ": device allocation failed");
    }
    if (counts) std::memcpy(counts, ctl, 7 * 8);
    const int h = (int)(uint32_t)ctl[7];
    if (crowded) *crowded = (uint32_t)(ctl[7] >> 32);
    if (ctl[7] != 0) {
        CK(cudaMemsetAsync(ctx->d_err, 0, 8, ctx->st));
        CK(cudaStreamSynchronize(ctx->st));
    }
    if (h != 0) {
        const char* what = h == ALB_ERR_ITER_CAP ? "a device loop hit its iteration cap"
                           : h == ALB_ERR_REPLAY ? "a replay stream ran out of variates"
                           : h == ALB_ERR_TOO_FEW ? "a photon map holds fewer records than k"
                           : h == ALB_ERR_CAPACITY ? "a waveform bin index fell outside the waveform"
                           : h == ALB_ERR_INVALID ? "a neighbour search admitted fewer than k finite points "
                                                    "(NaN or infinite coordinates)"
                                                   : "device error";
        return fail(ctx, h, std::string(where) + ": " + what);
    }
    return ALB_OK;
}

static thread_local std::string g_create_error;

namespace alb {
// message of a failure that has no context (alb_create, alb_knn_noalloc)
void set_global_error(const std::string& msg) { g_create_error = msg; }
}  // namespace alb

extern "C" const char* alb_last_error(const AlbCtx* ctx) { return ctx ? ctx->err.c_str() : g_create_error.c_str(); }

static void* table_buf(void*& slot, size_t bytes, cudaStream_t st) {
    if (!slot) slot = dev_alloc(bytes, st);
    return slot;
}

// Scene constants and tables of p into ctx->sc. The per-layer table buffers belong to the
// context and are reused by a later scene (batched runs re-scene one context per stream);
// copies are ordered on the context's stream, drained before the host staging vectors go
// away. Returns "" or why the scene is invalid.
static std::string set_scene(AlbCtx* ctx, const AlbSceneParams* p) {
    if (!(p->dt > 0) || p->steps <= 0 || p->sample_multiplier <= 0) return std::string("bad time step");
    if (p->k < 1 || p->k > 256) return std::string("photon_mapping_k must be in [1, 256]");
    if (p->n_layers < 1 || p->n_layers > ALB_MAX_LAYERS) return std::string("1..8 water layers supported");
    if (!(p->surface_y > p->floor_y)) return std::string("seafloor must lie below the surface");
    const int32_t adjoint = ctx->sc.adjoint;
    if (adjoint)
        for (int l = 0; l < p->n_layers; ++l)
            if (p->layers[l].profiled) return std::string("the adjoint needs constant layers");
    SceneDev& s = ctx->sc;
    s.dt = p->dt;
    s.total_steps = p->steps * (int64_t)p->sample_multiplier;
    s.nbins = 2 * p->steps;
    s.gate_lo = 0;
    s.gated = 0;
    if (p->gate_bins < 0 || p->gate_start < 0) return std::string("gate_start and gate_bins must be >= 0");
    s.stop_step[ALB_FORWARD] = s.stop_step[ALB_BACKWARD] = s.total_steps;
    if (p->gate_bins > 0) {
        if (p->gate_start + p->gate_bins > 2 * p->steps) return std::string("the gate must lie inside the timeline");
        s.nbins = p->gate_bins;
        s.gate_lo = p->gate_start;
        s.gated = 1;
        // With the fixed-radius gather every (query, record) pair contributes on its own. A
        // contribution lands in bin (t_query + t_record) / multiplier. Every photon starts at
        // the origin, |surface_y| above the water, and no record or query is made before it
        // reaches the surface: t >= floor(|surface_y| / (c_air dt)) - 2 steps, less the
        // forward pulse offset (bounded by 7 sigma / effective rate steps). A photon of one
        // pass can therefore stop once its steps exceed the gate's end minus the other
        // pass's earliest time: nothing it would add later can land in the window. (The
        // k-NN estimate is not pairwise: a late record can still be among a query's k
        // nearest and set its radius, so k-NN runs trace the whole timeline.)
        const double step_air = p->speed_air * p->dt;
        const int64_t t_surface = std::max<int64_t>((int64_t)std::floor(-p->surface_y / step_air) - 2, 0);
        const int64_t pulse = (int64_t)std::ceil(7.0 * p->pulse_sigma / (double)(float)p->effective_rate) + 1;
        const int64_t end = (p->gate_start + p->gate_bins + 2) * (int64_t)p->sample_multiplier;
        const int64_t fwd = end - t_surface + pulse + 4;                           // queries start >= t_surface
        const int64_t bwd = end - std::max<int64_t>(t_surface - pulse, 0) + 4;     // records start >= t_surface - pulse
        if (p->gather_radius > 0.0) {
            s.stop_step[ALB_FORWARD] = std::min(s.total_steps, std::max<int64_t>(fwd, 0));
            s.stop_step[ALB_BACKWARD] = std::min(s.total_steps, std::max<int64_t>(bwd, 0));
        }
    }
    s.mult = p->sample_multiplier;
    s.mult32 = (float)p->sample_multiplier;
    s.mult32_inv = 1.0f / s.mult32;
    s.k = p->k;
    s.ys = p->surface_y;
    s.yf = p->floor_y;
    s.v_air = p->speed_air;
    s.n_water = p->n_water;
    s.eta = 1.0 / p->n_water;
    s.f0 = p->f0;
    s.floor_albedo = p->seafloor_albedo;
    s.floor_albedo32 = (float)p->seafloor_albedo;
    s.surface_albedo = p->surface_albedo;
    s.floor_lambert = (float)(p->seafloor_albedo / kPi);
    s.surface_lambert = (float)(p->surface_albedo / kPi);
    s.roughness = p->roughness;
    double ga = p->roughness * p->roughness;
    s.ggx_a2 = (float)(ga * ga);
    for (int i = 0; i < 9; ++i) s.rot_d[i] = (double)p->laser_rot[i];
    s.div = p->divergence;
    s.fov = p->fov;
    s.cos_fov = std::cos(p->fov);
    s.aperture = p->aperture_radius;
    s.pulse_sigma32 = p->pulse_sigma;
    s.eff_rate32 = (double)(float)p->effective_rate;
    s.rayleigh_sigma = p->divergence / 3.0;
    s.rayleigh_mass = -std::expm1(-(p->divergence * p->divergence) / (2.0 * s.rayleigh_sigma * s.rayleigh_sigma));
    s.n_layers = p->n_layers;
    if (!(p->gather_radius >= 0.0)) return std::string("gather_radius must be >= 0 (0 selects the k-NN gather)");
    if (!(p->slope_sigma >= 0.0)) return std::string("slope_sigma must be >= 0");
    s.slope_sigma = p->slope_sigma;
    s.radius = p->gather_radius;
    s.heatmap = p->heatmap_enabled;
    s.hm_bins = p->heatmap_bins;
    s.hm_wext = p->heatmap_water_extent;
    s.hm_fext = p->heatmap_floor_extent;
    s.hm_wbin = 2.0 * p->heatmap_water_extent / p->heatmap_bins;
    s.hm_fbin = 2.0 * p->heatmap_floor_extent / p->heatmap_bins;
    for (int i = 0; i < 3; ++i) {
        s.wc[i] = p->water_center[i];
        s.fc[i] = p->floor_center[i];
    }
    for (int i = 0; i < 2; ++i) {
        const float w = (float)s.wc[2 * i], f = (float)s.fc[2 * i];
        s.hm_wc32[i] = make_float2(w, (float)(s.wc[2 * i] - (double)w));
        s.hm_fc32[i] = make_float2(f, (float)(s.fc[2 * i] - (double)f));
    }
    s.hm_wext32 = (float)s.hm_wext;
    s.hm_fext32 = (float)s.hm_fext;
    const bool small_map = s.hm_bins > 0 && s.hm_bins <= 512;
    s.hm_winv = small_map && s.hm_wbin > 0.0 ? (float)(1.0 / s.hm_wbin) : 0.f;
    s.hm_finv = small_map && s.hm_fbin > 0.0 ? (float)(1.0 / s.hm_fbin) : 0.f;
    s.adjoint = adjoint;
    s.inv_albedo = p->seafloor_albedo > 0.0 ? (float)(1.0 / p->seafloor_albedo) : 0.f;
    s.dla2_drough = (float)(4.0 * p->roughness * p->roughness * p->roughness);
    const int N = ALB_PHASE_DIVISIONS;
    for (int l = 0; l < p->n_layers; ++l) {
        const AlbLayer& L = p->layers[l];
        if (!L.phase_theta || !L.phase_cdf || !L.phase_slope || !L.scatter_weight) return std::string("missing layer table");
        for (int i = 0; i < 3; ++i) {
            s.adj_dla[l][i] = (float)L.dlog_alpha[i];
            s.adj_dls[l][i] = (float)L.dlog_ssa[i];
        }
        s.layer_hg_g[l] = (float)L.hg_g;
        s.layer_dlw_g[l] = nullptr;
        if (L.dlog_weight_g) {
            std::vector<float> d(N);
            for (int i = 0; i < N; ++i) d[i] = (float)L.dlog_weight_g[i];
            float* dd = (float*)table_buf(ctx->lt[l].dlw, N * sizeof(float), ctx->st);
            if (!dd) return std::string("table allocation failed");
            cudaMemcpyAsync(dd, d.data(), N * sizeof(float), cudaMemcpyHostToDevice, ctx->st);
            cudaStreamSynchronize(ctx->st);
            s.layer_dlw_g[l] = dd;
        }
        s.layer_dsg[l] = nullptr;
        if (L.dlog_sample_g) {
            std::vector<float> d(N);
            for (int i = 0; i < N; ++i) d[i] = (float)L.dlog_sample_g[i];
            float* dd = (float*)table_buf(ctx->lt[l].dsg, N * sizeof(float), ctx->st);
            if (!dd) return std::string("table allocation failed");
            cudaMemcpyAsync(dd, d.data(), N * sizeof(float), cudaMemcpyHostToDevice, ctx->st);
            cudaStreamSynchronize(ctx->st);
            s.layer_dsg[l] = dd;
        }
        s.layer_bottom[l] = L.bottom_depth;
        s.layer_speed[l] = L.speed;
        s.layer_alpha[l] = L.alpha;
        s.layer_ssa[l] = L.ssa;
        s.layer_binw[l] = (float)L.bin_width;
        s.layer_binw_inv[l] = 1.0f / s.layer_binw[l];
        s.layer_bottom32[l] = (float)L.bottom_depth;
        s.layer_speed32[l] = (float)L.speed;
        s.layer_floor32[l] = (float)(s.ys - L.bottom_depth);
        s.layer_h[l] = L.height;
        s.layer_hinv[l] = 1.0 / L.height;
        s.layer_top32[l] = L.top32;
        s.layer_prof[l] = L.profiled ? 1 : 0;
        s.layer_lut_n[l] = 0;
        s.layer_lut_z[l] = nullptr;
        s.layer_lut_a[l] = s.layer_lut_s[l] = nullptr;
        s.layer_lut_inv[l] = 0.f;
        s.layer_nkind[l] = s.layer_akind[l] = 0;
        s.layer_n0[l] = s.layer_n1[l] = s.layer_a0[l] = s.layer_a1[l] = 0.0;
        if (L.profiled) {
            if (!L.lut_z || !L.lut_alpha || L.lut_n < 2) return std::string("profiled layer without an attenuation table");
            if (!(L.height > 0.0)) return std::string("profiled layer needs a positive height");
            if (L.n_kind < 0 || L.n_kind > 2 || L.a_kind < 0 || L.a_kind > 2) return std::string("unknown profile kind");
            float* lz;
            double* la;  // values, then slopes
            if (!take(lz, L.lut_n * sizeof(float), ctx->st)) return std::string("table allocation failed");
            ctx->tables.push_back(lz);
            if (!take(la, 2 * L.lut_n * sizeof(double), ctx->st)) return std::string("table allocation failed");
            ctx->tables.push_back(la);
            std::vector<double> slopes(L.lut_n, 0.0);
            for (int i = 0; i + 1 < L.lut_n; ++i)
                slopes[i] = (L.lut_alpha[i + 1] - L.lut_alpha[i]) / ((double)L.lut_z[i + 1] - (double)L.lut_z[i]);
            cudaMemcpyAsync(lz, L.lut_z, L.lut_n * sizeof(float), cudaMemcpyHostToDevice, ctx->st);
            cudaMemcpyAsync(la, L.lut_alpha, L.lut_n * sizeof(double), cudaMemcpyHostToDevice, ctx->st);
            cudaMemcpyAsync(la + L.lut_n, slopes.data(), L.lut_n * sizeof(double), cudaMemcpyHostToDevice, ctx->st);
            cudaStreamSynchronize(ctx->st);
            s.layer_lut_n[l] = L.lut_n;
            s.layer_lut_z[l] = lz;
            s.layer_lut_a[l] = la;
            s.layer_lut_s[l] = la + L.lut_n;
            const double span = (double)L.lut_z[L.lut_n - 1] - (double)L.lut_z[0];
            s.layer_lut_inv[l] = span > 0.0 && L.lut_z[0] == 0.f ? (float)((L.lut_n - 1) / span) : 0.f;
            s.layer_nkind[l] = L.n_kind;
            s.layer_akind[l] = L.a_kind;
            s.layer_n0[l] = L.n_start;
            s.layer_n1[l] = L.n_end;
            s.layer_a0[l] = L.a_start;
            s.layer_a1[l] = L.a_end;
        }
        double* th = (double*)table_buf(ctx->lt[l].th, N * sizeof(double), ctx->st);
        double* cdf = (double*)table_buf(ctx->lt[l].cdf, N * sizeof(double), ctx->st);
        double* sl = (double*)table_buf(ctx->lt[l].sl, N * sizeof(double), ctx->st);
        float* w = (float*)table_buf(ctx->lt[l].w, N * sizeof(float), ctx->st);
        if (!th || !cdf || !sl || !w) return std::string("table allocation failed");
        std::vector<double> slope(N, 0.0);
        std::memcpy(slope.data(), L.phase_slope, (N - 1) * sizeof(double));
        std::vector<float> wf(N);
        for (int i = 0; i < N; ++i) wf[i] = (float)L.scatter_weight[i];
        cudaMemcpyAsync(th, L.phase_theta, N * sizeof(double), cudaMemcpyHostToDevice, ctx->st);
        cudaMemcpyAsync(cdf, L.phase_cdf, N * sizeof(double), cudaMemcpyHostToDevice, ctx->st);
        cudaMemcpyAsync(sl, slope.data(), N * sizeof(double), cudaMemcpyHostToDevice, ctx->st);
        cudaMemcpyAsync(w, wf.data(), N * sizeof(float), cudaMemcpyHostToDevice, ctx->st);
        s.layer_theta[l] = th;
        s.layer_cdf[l] = cdf;
        s.layer_slope[l] = sl;
        s.layer_weight[l] = w;
        float* dinv = (float*)table_buf(ctx->lt[l].inv, (kInvCdf + 1) * sizeof(float), ctx->st);
        uint16_t* guide = (uint16_t*)table_buf(ctx->lt[l].guide, (kInvCdf + 1) * sizeof(uint16_t), ctx->st);
        if (!dinv || !guide) return std::string("table allocation failed");
        launch_phase_tables(cdf, th, sl, dinv, guide, ctx->st);
        s.layer_guide[l] = guide;
        cudaStreamSynchronize(ctx->st);  // the host staging vectors die with this iteration
        ctx->fast.inv_theta[l] = dinv;
    }
    bool logs = false;
    for (int l = 0; l < s.n_layers; ++l) {
        s.layer_nl0[l] = s.layer_ndl[l] = s.layer_al0[l] = s.layer_adl[l] = 0.0;
        logs = logs || s.layer_nkind[l] == 2 || s.layer_akind[l] == 2;
    }
    if (logs) {
        double* d = nullptr;
        double h[4 * ALB_MAX_LAYERS];
        if (!take(d, sizeof h, ctx->st)) return std::string("table allocation failed");
        launch_profile_logs(s, d, ctx->st);
        const cudaError_t e = cudaMemcpyAsync(h, d, sizeof h, cudaMemcpyDeviceToHost, ctx->st);
        cudaStreamSynchronize(ctx->st);
        drop(d, ctx->st);
        if (e != cudaSuccess) return std::string("profile tables failed");
        for (int l = 0; l < s.n_layers; ++l) {
            s.layer_nl0[l] = h[4 * l];
            s.layer_ndl[l] = h[4 * l + 1];
            s.layer_al0[l] = h[4 * l + 2];
            s.layer_adl[l] = h[4 * l + 3];
        }
    }
    return std::string();
}

// Sets of class words for the waveform: one per channel, so that gathers may run side by side, or one for
// all of them where a set is large (128 B per bin).
static int64_t class_sets(int64_t nbins) { return nbins <= (1 << 20) ? ALB_CHANNELS : 1; }

// Bytes of what ensure_accumulators allocates.
static double accumulator_bytes(int64_t nbins, bool adjoint, int64_t heat_cells) {
    const double words = 2.0 * ALB_CHANNELS + 16.0 * class_sets(nbins) + (adjoint ? (2.0 * ALB_CHANNELS + 16.0) * kJacParams : 0.0);
    return 8.0 * words * nbins + heat_cells * (8.0 * (heat_cells <= 512 * 512 ? 4 + 32 : 4) + 3 * 4.0);
}

// Waveform, Jacobian and heatmap accumulators sized for the current scene (grown, never
// shrunk; a grown buffer is zeroed by the next reset).
static std::string ensure_accumulators(AlbCtx* ctx) {
    const SceneDev& s = ctx->sc;
    auto regrow = [&](unsigned long long*& buf, int64_t& have, int64_t need, size_t words_per) -> bool {
        if (buf && have >= need) return true;
        drop(buf, ctx->st);
        if (!take(buf, (size_t)need * words_per * 8, ctx->st)) {
            have = 0;
            return false;
        }
        cudaMemsetAsync(buf, 0, (size_t)need * words_per * 8, ctx->st);
        have = need;
        return true;
    };
    if (!regrow(ctx->wf, ctx->wf_bins, s.nbins, (size_t)2 * ALB_CHANNELS) ||
        !regrow(ctx->cls, ctx->cls_bins, s.nbins * class_sets(s.nbins), 16))
        return "waveform allocation failed";
    if (s.adjoint && (!regrow(ctx->jac, ctx->jac_bins, s.nbins, (size_t)2 * kJacParams * ALB_CHANNELS) ||
                      !regrow(ctx->jac_cls, ctx->jac_cls_bins, s.nbins, (size_t)16 * kJacParams)))
        return "jacobian allocation failed";
    if (s.heatmap) {
        const int64_t hb = (int64_t)s.hm_bins * s.hm_bins;
        if (!regrow(ctx->hm, ctx->hm_cells, hb, 4)) return "heatmap allocation failed";
        // two maps of class words: 10 MB at the default 200 bins; larger maps add directly
        if (s.hm_bins <= 512 && !regrow(ctx->heat_cls, ctx->heat_cls_cells, hb, 32)) return "heatmap allocation failed";
        if (!ctx->hm_radius || ctx->hm_radius_cells < hb) {
            drop(ctx->hm_radius, ctx->st);
            drop(ctx->hm_radius_bak, ctx->st);
            ctx->hm_radius_cells = 0;
            if (!take(ctx->hm_radius, hb * 4, ctx->st) || !take(ctx->hm_radius_bak, 2 * hb * 4, ctx->st))
                return "heatmap allocation failed";
            cudaMemsetAsync(ctx->hm_radius, 0, hb * 4, ctx->st);
            ctx->hm_radius_cells = hb;
        }
    }
    return std::string();
}

static int create_on(const AlbSceneParams* p, int device, cudaStream_t st, AlbCtx** out);

extern "C" int alb_create(const AlbSceneParams* p, int device, AlbCtx** out) { return create_on(p, device, nullptr, out); }

static int create_on(const AlbSceneParams* p, int device, cudaStream_t st, AlbCtx** out) {
    if (!p || !out) return ALB_ERR_INVALID;
    *out = nullptr;
    AlbCtx* ctx = new AlbCtx();
    auto bad = [&](const std::string& m) {
        g_create_error = m;
        alb_destroy(ctx);
        return ALB_ERR_INVALID;
    };
    ctx->device = device;
    if (cudaSetDevice(device) != cudaSuccess) return bad("cudaSetDevice failed");
    ctx->st = st;
    ctx->ws.set_stream(st);
    std::string e = set_scene(ctx, p);
    if (e.empty()) e = ensure_accumulators(ctx);
    if (!e.empty()) return bad(e);
    if (!take(ctx->ctl, 64 * 8, st)) return bad("counter allocation failed");
    ctx->d_rec_count = ctx->ctl;
    ctx->d_q_count = ctx->ctl + 4;
    ctx->d_err = (int*)(ctx->ctl + 7);
    ctx->d_stats = ctx->ctl + 8;
    cudaMemsetAsync(ctx->ctl, 0, 64 * 8, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return bad("device initialisation failed");
    *out = ctx;
    return ALB_OK;
}

extern "C" void alb_destroy(AlbCtx* ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    // a caller's stream may be gone by now: wait for the device and free in the default stream
    if (ctx->callers_stream) {
        cudaDeviceSynchronize();
        ctx->st = nullptr;
        ctx->ws.set_stream(nullptr);
    }
    const cudaStream_t st = ctx->st;
    cudaStreamSynchronize(st);
    for (void* p : ctx->tables) dev_free(p, st);
    for (int c = 0; c < ALB_CHANNELS; ++c) {
        RecordStore& r = ctx->rec[c];
        for (void* p : {(void*)r.a, (void*)r.fwi, (void*)r.sfi, (void*)r.id, (void*)r.sco}) dev_free(p, st);
        release_map_index(ctx->map[c], st);
        dev_free(ctx->map[c].box_lo, st);
        dev_free(ctx->map[c].box_hi, st);
    }
    for (int k = 0; k < 3; ++k)
        for (void* p : {(void*)ctx->qa[k], (void*)ctx->qb[k], (void*)ctx->qc[k], (void*)ctx->qid[k], (void*)ctx->qperm[k],
                        (void*)ctx->qrk[k][0], (void*)ctx->qrk[k][1], (void*)ctx->qs[k]})
            dev_free(p, st);
    for (void* p : {(void*)ctx->wf, (void*)ctx->cls, (void*)ctx->jac_cls, (void*)ctx->heat_cls, (void*)ctx->hm,
                    (void*)ctx->hm_radius, (void*)ctx->hm_radius_bak, (void*)ctx->jac, (void*)ctx->ex_pos,
                    (void*)ctx->ex_dir, (void*)ctx->ex_f, (void*)ctx->ctl})
        dev_free(p, st);
    for (auto& t : ctx->lt)
        for (void* p : {t.th, t.cdf, t.sl, t.w, t.dlw, t.dsg, t.inv, t.guide}) dev_free(p, st);
    for (const auto& p : ctx->pending) {
        cudaEventDestroy(p.e0);
        cudaEventDestroy(p.e1);
    }
    for (cudaEvent_t e : ctx->events) cudaEventDestroy(e);
    if (ctx->fork) cudaEventDestroy(ctx->fork);
    for (cudaEvent_t e : ctx->join)
        if (e) cudaEventDestroy(e);
    for (cudaStream_t x : ctx->side)
        if (x) cudaStreamDestroy(x);
    delete ctx;
    cudaStreamSynchronize(st);  // what the pool does not keep goes back to the driver here
}

extern "C" int alb_set_option(AlbCtx* ctx, int key, int64_t v) {
    if (!ctx) return ALB_ERR_INVALID;
    CK(cudaSetDevice(ctx->device));
    switch (key) {
        case ALB_OPT_KEEP_EXIT_STATES: ctx->keep_exit = (int)v; break;
        case ALB_OPT_KEEP_RECORD_IDS: ctx->keep_ids = (int)v; break;
        case ALB_OPT_PRECISE: ctx->precise = (int)v; break;
        case ALB_OPT_MAP_CAPACITY: ctx->map_cap_hint = v; break;
        case ALB_OPT_SORT_QUERIES: ctx->sort_q = (int)v; break;
        case ALB_OPT_STREAM:
            // every call has waited for its stream, so nothing is pending on the old one
            ctx->st = (cudaStream_t)(intptr_t)v;
            ctx->callers_stream = true;
            ctx->ws.set_stream(ctx->st);
            break;
        case ALB_OPT_ADJOINT: {
            for (int c = 0; c < ALB_CHANNELS; ++c)
                if (ctx->h_rec_count[c]) return fail(ctx, ALB_ERR_STATE, "set ALB_OPT_ADJOINT before the first forward trace");
            if (v) {
                for (int l = 0; l < ctx->sc.n_layers; ++l)
                    if (ctx->sc.layer_prof[l]) return fail(ctx, ALB_ERR_INVALID, "the adjoint needs constant layers");
            }
            ctx->sc.adjoint = v ? 1 : 0;
            if (v) {
                std::string e = ensure_accumulators(ctx);
                if (!e.empty()) return fail(ctx, ALB_ERR_CUDA, e);
                CK(cudaStreamSynchronize(ctx->st));
            }
            break;
        }
        default: return fail(ctx, ALB_ERR_INVALID, "unknown option");
    }
    return ALB_OK;
}

// backward photons traced and gathered per chunk when no per-photon state is exported
constexpr uint64_t kBackwardChunk = 1ull << 22;
// A trace into buffers that turn out too small runs twice. In a scene not traced before, a small forward call
// therefore gets room for kManyRecords scatter records per photon (3 KB per photon, given back when the
// maps are built, or kept with the record stores by a batch's workers), and a large one traces its first kPilot photons into as much and measures: those few
// leave most of the chip idle, 2.7 ms of the float64 tracer's 16.5 for 200 000 photons twice over.
constexpr uint64_t kPilot = 1ull << 14;
constexpr uint64_t kSmallCall = 1ull << 18;
constexpr double kFewRecords = 4.0;  // bottom reflections in that room
constexpr double kManyRecords = 96.0;

// Records per photon that a first small call has room for (alb_trace's and ensure_records' allowances).
static double first_call_records() { return 1.03 * (1.0 + 1.0 / 16.0) * (kFewRecords + kManyRecords + 2.0 * 1.05); }

static void release_records(AlbCtx* ctx, int c) {
    RecordStore& r = ctx->rec[c];
    for (void* p : {(void*)r.a, (void*)r.fwi, (void*)r.sfi, (void*)r.id, (void*)r.sco}) dev_free(p, ctx->st);
    r = RecordStore{};
}

// grow a record store to hold `need` records, preserving the first `keep`
static int ensure_records(AlbCtx* ctx, int c, uint64_t need, uint64_t keep) {
    RecordStore& r = ctx->rec[c];
    bool want_hm = ctx->sc.heatmap != 0;
    bool want_id = ctx->keep_ids != 0;
    bool want_sco = ctx->sc.adjoint != 0;
    if (r.cap >= need && (!want_id || r.id) && (!want_hm || r.fwi) && (!want_sco || r.sco)) return ALB_OK;
    // small stores double (up to 32 MB), so that a pass of many batches does not copy its records for each
    uint64_t cap = std::max<uint64_t>(need + (keep ? std::max<uint64_t>(need / 16, std::min<uint64_t>(need, 1ull << 20)) : need / 16), 1024);
    if (!keep) release_records(ctx, c);  // nothing to copy: the peak is one store
    float4 *a = nullptr, *fwi = nullptr, *sfi = nullptr, *sco = nullptr;
    uint32_t* id = nullptr;
    // every allocation is checked, and a failure frees what this call had taken; the two
    // record halves are interleaved in one allocation (RecordStore)
    bool ok = take(a, cap * 32, ctx->st);
    if (ok && want_hm) ok = take(fwi, cap * 16, ctx->st) && take(sfi, cap * 16, ctx->st);
    if (ok && want_id) ok = take(id, cap * 4, ctx->st);
    if (ok && want_sco) ok = take(sco, cap * 16, ctx->st);
    if (!ok) {
        drop(a, ctx->st); drop(fwi, ctx->st); drop(sfi, ctx->st); drop(id, ctx->st); drop(sco, ctx->st);
        return fail(ctx, ALB_ERR_CUDA, "photon-map store: out of device memory");
    }
    if (keep) {
        CK(cudaMemcpyAsync(a, r.a, keep * 32, cudaMemcpyDeviceToDevice, ctx->st));
        if (want_hm && r.fwi) {
            CK(cudaMemcpyAsync(fwi, r.fwi, keep * 16, cudaMemcpyDeviceToDevice, ctx->st));
            CK(cudaMemcpyAsync(sfi, r.sfi, keep * 16, cudaMemcpyDeviceToDevice, ctx->st));
        }
        if (want_id && r.id) CK(cudaMemcpyAsync(id, r.id, keep * 4, cudaMemcpyDeviceToDevice, ctx->st));
        if (want_sco && r.sco) CK(cudaMemcpyAsync(sco, r.sco, keep * 16, cudaMemcpyDeviceToDevice, ctx->st));
    }
    release_records(ctx, c);
    r.a = a; r.b = a + 1; r.fwi = fwi; r.sfi = sfi; r.id = id; r.sco = sco; r.cap = cap;
    return ALB_OK;
}

// Bring a channel's records back into an append store (from its index) before appending.
static int restore_records(AlbCtx* ctx, int c, uint64_t need) {
    if (!ctx->rec_released[c]) return ALB_OK;
    const uint64_t n = ctx->h_rec_count[c];
    int rc = ensure_records(ctx, c, need, 0);
    if (rc) return rc;
    const MapIndex& m = ctx->map[c];
    RecordStore& r = ctx->rec[c];
    if (n) {
        // the index holds the halves in two arrays; the store interleaves them (32-byte pitch)
        CK(cudaMemcpy2DAsync(r.a, 32, m.a, 16, 16, n, cudaMemcpyDeviceToDevice, ctx->st));
        CK(cudaMemcpy2DAsync(r.b, 32, m.b, 16, 16, n, cudaMemcpyDeviceToDevice, ctx->st));
        if (r.fwi && m.fwi) {
            CK(cudaMemcpyAsync(r.fwi, m.fwi, n * 16, cudaMemcpyDeviceToDevice, ctx->st));
            CK(cudaMemcpyAsync(r.sfi, m.sfi, n * 16, cudaMemcpyDeviceToDevice, ctx->st));
        }
        if (r.id && m.id) CK(cudaMemcpyAsync(r.id, m.id, n * 4, cudaMemcpyDeviceToDevice, ctx->st));
        if (r.sco && m.sco) CK(cudaMemcpyAsync(r.sco, m.sco, n * 16, cudaMemcpyDeviceToDevice, ctx->st));
        CK(cudaStreamSynchronize(ctx->st));
    }
    ctx->rec_released[c] = false;
    return ALB_OK;
}

static int ensure_queries(AlbCtx* ctx, int k, uint64_t need) {
    if (ctx->qcap[k] >= need && (!ctx->keep_ids || ctx->qid[k]) && (!ctx->sc.adjoint || ctx->qs[k])) return ALB_OK;
    uint64_t cap = std::max<uint64_t>(need + need / 4, 1024);
    const cudaStream_t st = ctx->st;
    drop(ctx->qa[k], st); drop(ctx->qb[k], st); drop(ctx->qc[k], st); drop(ctx->qid[k], st); drop(ctx->qperm[k], st);
    drop(ctx->qrk[k][0], st); drop(ctx->qrk[k][1], st); drop(ctx->qs[k], st);
    ctx->qcap[k] = 0;
    bool ok = take(ctx->qa[k], cap * 16, st) && take(ctx->qb[k], cap * 16, st) && take(ctx->qc[k], cap * 16, st) &&
              take(ctx->qperm[k], cap * 4, st);
    if (ok && ctx->keep_ids)
        ok = take(ctx->qid[k], cap * 4, st) && take(ctx->qrk[k][0], cap * 8, st) && take(ctx->qrk[k][1], cap * 8, st);
    if (ok && ctx->sc.adjoint) ok = take(ctx->qs[k], cap * 16, st);
    if (!ok) return fail(ctx, ALB_ERR_CUDA, "gather queries: out of device memory");
    ctx->qcap[k] = cap;
    return ALB_OK;
}

static TraceOut make_out(AlbCtx* ctx) {
    TraceOut o{};
    for (int c = 0; c < ALB_CHANNELS; ++c) {
        o.rec_a[c] = ctx->rec[c].a;
        o.rec_b[c] = ctx->rec[c].b;
        o.rec_fwi[c] = ctx->rec[c].fwi;
        o.rec_sfi[c] = ctx->rec[c].sfi;
        o.rec_id[c] = ctx->rec[c].id;
        o.rec_sco[c] = ctx->sc.adjoint ? ctx->rec[c].sco : nullptr;
        o.rec_cap[c] = ctx->rec[c].cap;
    }
    o.rec_count = ctx->d_rec_count;
    for (int k = 0; k < 3; ++k) {
        o.q_a[k] = ctx->qa[k];
        o.q_b[k] = ctx->qb[k];
        o.q_c[k] = ctx->qc[k];
        o.q_id[k] = ctx->qid[k];
        o.q_s[k] = ctx->sc.adjoint ? ctx->qs[k] : nullptr;
        o.q_cap[k] = ctx->qcap[k];
    }
    o.q_count = ctx->d_q_count;
    o.ex_pos = ctx->keep_exit ? ctx->ex_pos : nullptr;
    o.ex_dir = ctx->ex_dir;
    o.ex_f = ctx->ex_f;
    o.hm_radius = ctx->hm_radius;
    o.err = ctx->d_err;
    o.stats = ctx->d_stats;
    return o;
}

// Q9 of the reference: a gather on a map with fewer than k records raises IndexError.
static int check_map_sizes(AlbCtx* ctx) {
    static const int need[3][2] = {{ALB_BOTTOM_REFLECTION, -1}, {ALB_SCATTER, -1},
                                   {ALB_SURFACE_REFLECTION, ALB_SURFACE_TRANSMISSION_UP}};
    static const char* names[4] = {"BOTTOM_REFLECTION", "SCATTER", "SURFACE_REFLECTION", "SURFACE_TRANSMISSION_UP"};
    for (int k = 0; k < 3; ++k) {
        if (ctx->h_q_count[k] == 0) continue;
        for (int j = 0; j < 2; ++j) {
            int c = need[k][j];
            if (c < 0) continue;
            if (ctx->map[c].n_real < (uint64_t)ctx->sc.k) {
                char buf[256];
                snprintf(buf, sizeof buf, "photon map %s holds %llu records, fewer than k=%d", names[c],
                         (unsigned long long)ctx->map[c].n_real, ctx->sc.k);
                return fail(ctx, ALB_ERR_TOO_FEW, buf);
            }
        }
    }
    return ALB_OK;
}

static const int kGatherKind[4] = {kQueryBottom, kQueryScatter, kQuerySurface, kQuerySurface};
static const int kGatherChannel[4] = {ALB_BOTTOM_REFLECTION, ALB_SCATTER, ALB_SURFACE_REFLECTION, ALB_SURFACE_TRANSMISSION_UP};

// The queries of gather g as left by the last backward trace.
static QueryDev query_dev(AlbCtx* ctx, int g, bool lo_zero) {
    const int k = kGatherKind[g], c = kGatherChannel[g];
    QueryDev q{};
    q.a = ctx->qa[k];
    q.b = ctx->qb[k];
    q.c = ctx->qc[k];
    q.lo_zero = lo_zero;
    q.s = ctx->sc.adjoint ? ctx->qs[k] : nullptr;
    q.perm = ctx->sort_q ? ctx->qperm[k] : nullptr;
    q.n = ctx->h_q_count[k];
    q.rk_out = ctx->keep_ids ? ctx->qrk[k][g == 3 ? 1 : 0] : nullptr;
    q.stats = ctx->d_stats + 4 + 4 * c;  // per channel: leaves, nodes, selects, queries
    q.crowded = (uint32_t*)ctx->d_err + 1;
    q.retries = ctx->d_stats + 30;
    q.n_crowded = ctx->d_stats + 31;
    q.ticket = (uint32_t*)(ctx->ctl + 43 + c);
    return q;
}

// Sorts the queries of the last backward trace and gathers them from their maps, queued on the
// context's stream. side: how many of the context's side streams were given work; they are joined
// to its stream on success only.
static int queue_gathers(AlbCtx* ctx, const Accum& acc, bool lo_zero, int& side) {
    uint64_t total = 0;
    for (int k = 0; k < 3; ++k) {
        const uint64_t nq = ctx->h_q_count[k];
        total += nq;
        if (nq == 0 || !ctx->sort_q) continue;
        PhaseTimer ps(ctx, 3);
        const int rc = sort_queries(ctx->ws, ctx->qa[k], nq, ctx->qperm[k], ctx->st);
        ps.stop();
        if (rc != 0) return fail(ctx, ALB_ERR_CUDA, "query sort: device memory allocation failed");
    }
    // each channel's work items of a fixed-radius gather (8 MB each; without them a query is one warp's)
    uint32_t* work = nullptr;
    const uint64_t words = 2 + 2 * (uint64_t)kRadiusItems;
    if (ctx->sc.radius > 0.0 && !(work = ctx->ws.take_u32(4 * words))) ctx->ws.clear_failed();
    // Few queries leave most of the chip idle in one gather: the planar ones run beside one another on
    // streams forked here and joined below (the Jacobian and the heatmaps sum through words
    // that the channels share, so those runs stay in series). A backward call on the
    // 5 m water scene's maps of 1e5 photons: 1.2 -> 0.9 ms with 5000 photons, 2.0 -> 1.6 ms with 25,000.
    const bool fork = total < (1ull << 20) && !acc.jac_lo && !acc.hw_lo && acc.cls_step;
    if (fork) {
        if (!ctx->fork) {
            CK(cudaEventCreateWithFlags(&ctx->fork, cudaEventDisableTiming));
            for (int i = 0; i < 3; ++i) {
                CK(cudaEventCreateWithFlags(&ctx->join[i], cudaEventDisableTiming));
                CK(cudaStreamCreateWithFlags(&ctx->side[i], cudaStreamNonBlocking));
            }
        }
        CK(cudaEventRecord(ctx->fork, ctx->st));
    }
    static const int sequence[4] = {0, 2, 3, 1};  // the scatter gather's CTAs fill whole SMs: last
    for (int s = 0; s < 4; ++s) {
        const int g = sequence[s], c = kGatherChannel[g];
        QueryDev q = query_dev(ctx, g, lo_zero);
        if (q.n == 0) continue;
        q.work = work ? work + c * words : nullptr;
        const bool aside = fork && c != ALB_SCATTER;
        cudaStream_t st = ctx->st;
        if (aside) {
            st = ctx->side[side++];
            CK(cudaStreamWaitEvent(st, ctx->fork, 0));
        }
        PhaseTimer pg(ctx, 4 + c, st);
        launch_gather(ctx->sc, map_dev(ctx->map[c]), q, c, acc, ctx->d_err, &ctx->launches, st);
        pg.stop(st);
        if (aside) CK(cudaEventRecord(ctx->join[side - 1], st));
        ctx->gathered[c] += (int64_t)q.n;
    }
    for (int i = 0; i < side; ++i) CK(cudaStreamWaitEvent(ctx->st, ctx->join[i], 0));
    return ALB_OK;
}

static int gather_all(AlbCtx* ctx, const Accum& acc, bool lo_zero) {
    const size_t mark = ctx->ws.mark();
    int side = 0;
    const int rc = queue_gathers(ctx, acc, lo_zero, side);
    if (rc) {
        // what is queued still uses the query buffers and the scratch
        for (int i = 0; i < side; ++i) cudaStreamSynchronize(ctx->side[i]);
        cudaStreamSynchronize(ctx->st);
    }
    ctx->ws.release(mark);
    return rc;
}

// What a call takes of the workspace goes back when it returns, on an error too.
struct ScratchScope {
    AlbCtx* ctx;
    size_t mark;
    explicit ScratchScope(AlbCtx* c) : ctx(c), mark(c->ws.mark()) {}
    ScratchScope(const ScratchScope&) = delete;
    ~ScratchScope() { ctx->ws.release(mark); }
};

extern "C" int alb_trace(AlbCtx* ctx, int pass, uint64_t n, uint64_t seed, uint64_t first, const AlbReplay* rp) {
    if (!ctx) return ALB_ERR_INVALID;
    if (pass != ALB_FORWARD && pass != ALB_BACKWARD) return fail(ctx, ALB_ERR_INVALID, "pass must be 0 or 1");
    if (pass == ALB_BACKWARD && !ctx->maps_built) return fail(ctx, ALB_ERR_STATE, "backward trace before alb_build_maps");
    if (first + n > (1ull << 32)) return fail(ctx, ALB_ERR_INVALID, "photon ids are 32-bit per pass");
    if (rp && ctx->sc.slope_sigma > 0.0)
        return fail(ctx, ALB_ERR_INVALID, "surface slopes draw variates the reference never records (Philox only)");
    CK(cudaSetDevice(ctx->device));
    ctx->err.clear();
    // replay streams to the device
    AlbReplay drp{};
    const ScratchScope scratch(ctx);
    if (rp) {
        if (!rp->offsets || !rp->values || !rp->tau) return fail(ctx, ALB_ERR_INVALID, "incomplete replay");
        int64_t* o = (int64_t*)ctx->ws.take_bytes((n + 1) * 8);
        double* v = (double*)ctx->ws.take_bytes(rp->n_values * 8 + 8);
        float* t = (float*)ctx->ws.take_bytes(rp->n_values * 4 + 4);
        if (!o || !v || !t) return fail(ctx, ALB_ERR_CUDA, "replay upload allocation failed");
        CK(cudaMemcpyAsync(o, rp->offsets, (n + 1) * 8, cudaMemcpyHostToDevice, ctx->st));
        CK(cudaMemcpyAsync(v, rp->values, rp->n_values * 8, cudaMemcpyHostToDevice, ctx->st));
        CK(cudaMemcpyAsync(t, rp->tau, rp->n_values * 4, cudaMemcpyHostToDevice, ctx->st));
        drp.offsets = o;
        drp.values = v;
        drp.tau = t;
        drp.n_values = rp->n_values;
    }
    if (ctx->keep_exit) {
        if (ctx->ex_cap < n) {
            drop(ctx->ex_pos, ctx->st); drop(ctx->ex_dir, ctx->st); drop(ctx->ex_f, ctx->st);
            ctx->ex_cap = 0;
            if (!take(ctx->ex_pos, n * 24, ctx->st) || !take(ctx->ex_dir, n * 24, ctx->st) || !take(ctx->ex_f, n * 40, ctx->st))
                return fail(ctx, ALB_ERR_CUDA, "exit states: out of device memory");
            ctx->ex_cap = n;
        }
        ctx->ex_n = n;
    }
    // slots 28/29 keep the last forward trace's events and photons across the backward trace
    CK(cudaMemsetAsync(ctx->d_stats, 0, 28 * 8, ctx->st));
    CK(cudaMemsetAsync(ctx->d_stats + 30, 0, 2 * 8, ctx->st));
    unsigned long long* const stats_bak = ctx->ctl + 41;
    if (pass == ALB_FORWARD) {
        ctx->maps_built = false;
        const size_t hb = ctx->sc.heatmap ? (size_t)ctx->sc.hm_bins * ctx->sc.hm_bins : 0;
        uint64_t before_call[ALB_CHANNELS];
        std::memcpy(before_call, ctx->h_rec_count, sizeof before_call);
        bool saved = false;  // the radius heatmap as it was has been copied
        // photons [p0, p0 + pn) of the call
        auto part = [&](uint64_t p0, uint64_t pn) -> int {
            unsigned* const radius_bak = ctx->hm_radius_bak + (p0 ? hb : 0);
            uint64_t before[ALB_CHANNELS];
            std::memcpy(before, ctx->h_rec_count, sizeof before);
            CK(cudaMemcpyAsync(stats_bak, ctx->d_stats, 2 * 8, cudaMemcpyDeviceToDevice, ctx->st));
            if (hb) CK(cudaMemcpyAsync(radius_bak, ctx->hm_radius, hb * 4, cudaMemcpyDeviceToDevice, ctx->st));
            saved = true;
            for (int attempt = 0; attempt < 3; ++attempt) {
                for (int c = 0; c < ALB_CHANNELS; ++c) {
                    uint64_t est = (uint64_t)(ctx->rec_rate[c] * (double)pn * 1.03) + 4096;
                    if (ctx->map_cap_hint > 0) est = std::max<uint64_t>(est, (uint64_t)ctx->map_cap_hint);
                    int rc = ctx->rec_released[c] ? restore_records(ctx, c, before[c] + est)
                                                   : ensure_records(ctx, c, before[c] + est, before[c]);
                    if (rc && !ctx->rec_rate_known && attempt == 0 && ctx->rec_rate[ALB_SCATTER] == kManyRecords) {
                        // no room for so many: as few as a retry can correct
                        ctx->rec_rate[ALB_BOTTOM_REFLECTION] = 2.0;
                        ctx->rec_rate[ALB_SCATTER] = 8.0;
                        ctx->err.clear();
                        c = -1;
                        continue;
                    }
                    if (rc) return rc;
                }
                TraceOut o = make_out(ctx);
                PhaseTimer pt(ctx, 0);
                launch_trace(ctx->sc, o, ALB_FORWARD, pn, first + p0, seed, rp ? &drp : nullptr, &ctx->launches, ctx->st,
                             ctx->precise ? nullptr : &ctx->fast);
                pt.stop();
                CK(cudaMemcpyAsync(ctx->d_stats + 28, ctx->d_stats, 2 * 8, cudaMemcpyDeviceToDevice, ctx->st));
                unsigned long long cnt[7];
                int rc = check_device(ctx, "forward trace", cnt);
                if (rc) return rc;
                bool overflow = false;
                for (int c = 0; c < ALB_CHANNELS; ++c) {
                    uint64_t added = cnt[c] - before[c];
                    const double rate = (double)added / (double)std::max<uint64_t>(pn, 1);
                    if (ctx->rec_rate_known) ctx->rec_rate[c] = pn ? std::max(ctx->rec_rate[c] * 0.5, rate) : ctx->rec_rate[c];
                    else if (pn >= 1024) ctx->rec_rate[c] = rate;  // fewer photons measure too little
                    if (cnt[c] > ctx->rec[c].cap) overflow = true;
                }
                if (!overflow) {
                    for (int c = 0; c < ALB_CHANNELS; ++c) ctx->h_rec_count[c] = cnt[c];
                    if (pn >= 1024) ctx->rec_rate_known = true;
                    return ALB_OK;
                }
                // undo and retry with the measured sizes
                CK(cudaMemcpyAsync(ctx->d_stats, stats_bak, 2 * 8, cudaMemcpyDeviceToDevice, ctx->st));
                CK(cudaMemcpyAsync(ctx->d_rec_count, before, sizeof before, cudaMemcpyHostToDevice, ctx->st));
                if (hb) CK(cudaMemcpyAsync(ctx->hm_radius, radius_bak, hb * 4, cudaMemcpyDeviceToDevice, ctx->st));
                CK(cudaStreamSynchronize(ctx->st));
                for (int c = 0; c < ALB_CHANNELS; ++c) ctx->rec_rate[c] = (double)(cnt[c] - before[c]) / (double)pn;
            }
            return fail(ctx, ALB_ERR_CAPACITY, "photon-map capacity could not be established");
        };
        const uint64_t pilot = !ctx->rec_rate_known && n > kSmallCall && !rp && !ctx->keep_exit ? kPilot : 0;
        if (!ctx->rec_rate_known && (pilot || n <= kSmallCall)) {
            ctx->rec_rate[ALB_BOTTOM_REFLECTION] = kFewRecords;
            ctx->rec_rate[ALB_SCATTER] = kManyRecords;
        }
        int rc = pilot ? part(0, pilot) : ALB_OK;
        if (!rc) rc = part(pilot, n - pilot);
        if (rc) {
            // the call as a whole leaves nothing: no records (a pilot's included) and no crossings
            std::memcpy(ctx->h_rec_count, before_call, sizeof before_call);
            cudaMemcpyAsync(ctx->d_rec_count, before_call, sizeof before_call, cudaMemcpyHostToDevice, ctx->st);
            if (hb && saved) cudaMemcpyAsync(ctx->hm_radius, ctx->hm_radius_bak, hb * 4, cudaMemcpyDeviceToDevice, ctx->st);
            cudaStreamSynchronize(ctx->st);
        }
        return rc;
    }
    // backward: trace -> queries -> gathers. Without per-photon exports the photons go in
    // chunks, so that query buffers stay bounded whatever n is (the waveform sums are
    // integer and order independent, so chunking cannot change the result).
    Accum acc{};
    acc.wf_lo = ctx->wf;
    acc.wf_hi = ctx->wf + (size_t)ALB_CHANNELS * ctx->sc.nbins;
    acc.cls = ctx->cls;
    acc.cls_step = class_sets(ctx->sc.nbins) > 1 ? (uint64_t)16 * ctx->sc.nbins : 0;
    acc.nbins = ctx->sc.nbins;
    if (ctx->sc.adjoint) {
        acc.jac_lo = ctx->jac;
        acc.jac_hi = ctx->jac + (size_t)kJacParams * ALB_CHANNELS * ctx->sc.nbins;
        acc.jac_cls = ctx->jac_cls;
    }
    if (ctx->sc.heatmap) {
        size_t hb = (size_t)ctx->sc.hm_bins * ctx->sc.hm_bins;
        acc.hw_lo = ctx->hm;
        acc.hw_hi = ctx->hm + hb;
        acc.hf_lo = ctx->hm + 2 * hb;
        acc.hf_hi = ctx->hm + 3 * hb;
        acc.heat_cls = ctx->sc.hm_bins <= 512 ? ctx->heat_cls : nullptr;
    }
    const bool chunked = !ctx->keep_exit && !ctx->keep_ids && !rp;
    const uint64_t chunk = chunked ? kBackwardChunk : std::max<uint64_t>(n, 1);
    // traces photons [c0, c0 + nc) into the query buffers, which may turn out too small
    auto trace = [&](uint64_t c0, uint64_t nc, bool& overflow) -> int {
        for (int k = 0; k < 3; ++k) {
            uint64_t est = (uint64_t)(ctx->q_rate[k] * (double)nc * 1.1) + 4096;
            int rc = ensure_queries(ctx, k, est);
            if (rc) return rc;
        }
        CK(cudaMemsetAsync(ctx->d_q_count, 0, 3 * 8, ctx->st));
        CK(cudaMemcpyAsync(stats_bak, ctx->d_stats, 2 * 8, cudaMemcpyDeviceToDevice, ctx->st));
        TraceOut o = make_out(ctx);
        PhaseTimer pt(ctx, 2);
        launch_trace(ctx->sc, o, ALB_BACKWARD, nc, first + c0, seed, rp ? &drp : nullptr, &ctx->launches, ctx->st,
                     ctx->precise ? nullptr : &ctx->fast);
        pt.stop();
        unsigned long long cnt[7];
        int rc = check_device(ctx, "backward trace", cnt);
        if (rc) return rc;
        overflow = false;
        for (int k = 0; k < 3; ++k) {
            ctx->h_q_count[k] = cnt[4 + k];
            if (nc > 0) ctx->q_rate[k] = std::max(ctx->q_rate[k] * 0.5, (double)cnt[4 + k] / (double)nc);
            if (cnt[4 + k] > ctx->qcap[k]) overflow = true;
        }
        if (overflow)
            for (int k = 0; k < 3; ++k) ctx->q_rate[k] = (double)cnt[4 + k] / (double)nc;
        ctx->q_rate_known = ctx->q_rate_known || nc > 0;
        return ALB_OK;
    };
    auto untrace = [&]() -> int {  // the counters as before the trace
        CK(cudaMemcpyAsync(ctx->d_stats, stats_bak, 2 * 8, cudaMemcpyDeviceToDevice, ctx->st));
        return ALB_OK;
    };
    // a scene's backward photons make queries as its forward photons make records (within 2% in every
    // workload here), so the forward rates size the first buffers; a trace into too small ones runs twice
    if (!ctx->q_rate_known && ctx->rec_rate_known) {
        ctx->q_rate[kQueryBottom] = ctx->rec_rate[ALB_BOTTOM_REFLECTION];
        ctx->q_rate[kQueryScatter] = ctx->rec_rate[ALB_SCATTER];
        ctx->q_rate[kQuerySurface] = std::max(ctx->rec_rate[ALB_SURFACE_REFLECTION], 1.0);
        ctx->q_rate_known = true;
    }
    for (uint64_t c0 = 0; c0 == 0 || c0 < n; c0 += chunk) {
        const uint64_t nc = std::min<uint64_t>(chunk, n - c0);
        bool overflow = false;
        int rc = ALB_OK;
        if (!ctx->q_rate_known && nc > 4 * kPilot && chunked) {
            rc = trace(c0, kPilot, overflow);
            if (!rc) rc = untrace();
            if (rc) return rc;
        }
        for (int attempt = 0; attempt < 3; ++attempt) {
            rc = trace(c0, nc, overflow);
            if (rc) return rc;
            if (!overflow) break;
            rc = untrace();
            if (rc) return rc;
            if (attempt == 2) return fail(ctx, ALB_ERR_CAPACITY, "query capacity could not be established");
        }
        rc = ctx->sc.radius > 0.0 ? ALB_OK : check_map_sizes(ctx);  // k-NN needs k records
        if (rc) return rc;
        const bool lo_zero = !ctx->precise && !rp;
        uint32_t crowded = 0;
        rc = gather_all(ctx, acc, lo_zero);
        if (!rc) rc = check_device(ctx, "gather", nullptr, &crowded);
        if (!rc && crowded) {
            for (int g = 0; g < 4; ++g) {
                const int c = kGatherChannel[g];
                if (!(crowded >> c & 1u)) continue;
                PhaseTimer pg(ctx, 4 + c);
                launch_gather_crowded(ctx->sc, map_dev(ctx->map[c]), query_dev(ctx, g, lo_zero), c, acc, ctx->d_err, ctx->st);
                pg.stop();
            }
            rc = check_device(ctx, "gather");
        }
        if (rc) return rc;
        if (n == 0) break;
    }
    return ALB_OK;
}

extern "C" int alb_build_maps(AlbCtx* ctx) {
    if (!ctx) return ALB_ERR_INVALID;
    CK(cudaSetDevice(ctx->device));
    PhaseTimer pt(ctx, 1);
    static const char* const failed = "photon-map index build failed (device memory or partition)";
    // every channel's build is queued before the first is waited for
    RecordStore rec[ALB_CHANNELS];
    bool todo[ALB_CHANNELS];
    for (int c = 0; c < ALB_CHANNELS; ++c) {
        todo[c] = !ctx->rec_released[c];  // else indexed already, nothing appended since
        if (!todo[c]) continue;
        rec[c] = ctx->rec[c];
        if (!ctx->sc.adjoint) rec[c].sco = nullptr;  // a store kept from an adjoint run: no scores now
        if (start_map_index(ctx->ws, rec[c], ctx->h_rec_count[c], ctx->map[c], c, ctx->st) != 0)
            return fail(ctx, ALB_ERR_CAPACITY, failed);
        // a large store is released before the next channel's index is allocated
        if (ctx->h_rec_count[c] > (1ull << 26)) {
            if (finish_map_index(ctx->ws, rec[c], ctx->map[c], c, ctx->st) != 0) return fail(ctx, ALB_ERR_CAPACITY, failed);
            todo[c] = false;
            if (!ctx->keep_records) {
                release_records(ctx, c);
                ctx->rec_released[c] = true;
            }
        }
    }
    for (int c = 0; c < ALB_CHANNELS; ++c) {
        if (!todo[c]) continue;
        if (finish_map_index(ctx->ws, rec[c], ctx->map[c], c, ctx->st) != 0) return fail(ctx, ALB_ERR_CAPACITY, failed);
        if (ctx->keep_records) continue;  // the store stays for the next simulation
        release_records(ctx, c);
        ctx->rec_released[c] = true;
    }
    pt.stop();
    int rc = check_device(ctx, "map build");
    if (rc) return rc;
    ctx->maps_built = true;
    return ALB_OK;
}

extern "C" int alb_map_size(AlbCtx* ctx, int c, uint64_t* out) {
    if (!ctx || !out || c < 0 || c >= ALB_CHANNELS) return ALB_ERR_INVALID;
    *out = ctx->h_rec_count[c];
    return ALB_OK;
}

extern "C" int alb_export_map(AlbCtx* ctx, int c, float* pos, float* dir, float* energy, float* time,
                              float* fwi, float* sfi, int64_t* pid, size_t n) {
    if (!ctx || c < 0 || c >= ALB_CHANNELS) return ALB_ERR_INVALID;
    uint64_t m = ctx->h_rec_count[c];
    if (n < m) return fail(ctx, ALB_ERR_INVALID, "export buffer smaller than the map");
    if (m == 0) return ALB_OK;
    const float4 *a, *b, *fw, *sf;
    const uint32_t* id;
    size_t pitch;  // bytes between consecutive records' a (and b) halves
    // records in append order (the interleaved store), or in index order once the channel
    // has been indexed
    if (ctx->rec_released[c]) {
        const MapIndex& mi = ctx->map[c];
        a = mi.a; b = mi.b; id = mi.id; fw = mi.fwi; sf = mi.sfi;
        pitch = 16;
    } else {
        a = ctx->rec[c].a; b = ctx->rec[c].b; id = ctx->rec[c].id; fw = ctx->rec[c].fwi; sf = ctx->rec[c].sfi;
        pitch = 32;
    }
    std::vector<float4> ha(m), hb(m), hf, hs;
    CK(cudaMemcpy2D(ha.data(), 16, a, pitch, 16, m, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy2D(hb.data(), 16, b, pitch, 16, m, cudaMemcpyDeviceToHost));
    if (fw && (fwi || sfi)) {
        hf.resize(m);
        hs.resize(m);
        CK(cudaMemcpy(hf.data(), fw, m * 16, cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(hs.data(), sf, m * 16, cudaMemcpyDeviceToHost));
    }
    std::vector<uint32_t> hid;
    if (pid && id) {
        hid.resize(m);
        CK(cudaMemcpy(hid.data(), id, m * 4, cudaMemcpyDeviceToHost));
    }
    const float qnan = std::nanf("");
    for (uint64_t i = 0; i < m; ++i) {
        if (pos) { pos[3 * i] = ha[i].x; pos[3 * i + 1] = ha[i].y; pos[3 * i + 2] = ha[i].z; }
        if (energy) energy[i] = ha[i].w;
        if (dir) { dir[3 * i] = hb[i].x; dir[3 * i + 1] = hb[i].y; dir[3 * i + 2] = hb[i].z; }
        if (time) time[i] = hb[i].w;
        if (fwi) {
            fwi[3 * i] = hf.empty() ? qnan : hf[i].x;
            fwi[3 * i + 1] = hf.empty() ? qnan : hf[i].y;
            fwi[3 * i + 2] = hf.empty() ? qnan : hf[i].z;
        }
        if (sfi) {
            sfi[3 * i] = hs.empty() ? qnan : hs[i].x;
            sfi[3 * i + 1] = hs.empty() ? qnan : hs[i].y;
            sfi[3 * i + 2] = hs.empty() ? qnan : hs[i].z;
        }
        if (pid) pid[i] = hid.empty() ? -1 : (int64_t)hid[i];
    }
    return ALB_OK;
}

extern "C" int alb_get_heatmaps(AlbCtx* ctx, double* water, double* seafloor, float* radius, size_t bins2) {
    if (!ctx) return ALB_ERR_INVALID;
    if (!ctx->sc.heatmap) return fail(ctx, ALB_ERR_STATE, "heatmaps are disabled in this scene");
    size_t hb = (size_t)ctx->sc.hm_bins * ctx->sc.hm_bins;
    if (bins2 < hb) return fail(ctx, ALB_ERR_INVALID, "heatmap buffer too small");
    std::vector<unsigned long long> h(4 * hb);
    CK(cudaMemcpy(h.data(), ctx->hm, 4 * hb * 8, cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < hb; ++i) {
        if (water) water[i] = fix_to_double(h[i], (long long)h[hb + i]);
        if (seafloor) seafloor[i] = fix_to_double(h[2 * hb + i], (long long)h[3 * hb + i]);
    }
    if (radius) {
        std::vector<unsigned> r(hb);
        CK(cudaMemcpy(r.data(), ctx->hm_radius, hb * 4, cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < hb; ++i) radius[i] = (float)r[i];
    }
    return ALB_OK;
}

// n 128-bit words of an accumulator to the host as float64 or float32, converted on the device.
template <class T>
static int read_fixed(AlbCtx* ctx, const unsigned long long* lo, const unsigned long long* hi, int64_t n, T* out) {
    CK(cudaSetDevice(ctx->device));
    const size_t mark = ctx->ws.mark();
    T* d = (T*)ctx->ws.take_bytes((size_t)n * sizeof(T));
    if (!d) return fail(ctx, ALB_ERR_CUDA, "read-back buffer: out of device memory");
    launch_fix_to_float(lo, hi, n, d, ctx->st);
    const cudaError_t e = cudaMemcpyAsync(out, d, (size_t)n * sizeof(T), cudaMemcpyDeviceToHost, ctx->st);
    ctx->ws.release(mark);
    CK(e);
    CK(cudaStreamSynchronize(ctx->st));
    return ALB_OK;
}

template <class T>
static int read_wf(AlbCtx* ctx, int c, T* out) {
    const int64_t nb = ctx->sc.nbins;
    return read_fixed(ctx, ctx->wf + (size_t)c * nb, ctx->wf + (size_t)(ALB_CHANNELS + c) * nb, nb, out);
}

extern "C" int alb_get_waveform(AlbCtx* ctx, int c, float* out, size_t nbins) {
    if (!ctx || !out || c < 0 || c >= ALB_CHANNELS) return ALB_ERR_INVALID;
    if (nbins < (size_t)ctx->sc.nbins) return fail(ctx, ALB_ERR_INVALID, "waveform buffer too small");
    return read_wf(ctx, c, out);
}

extern "C" int alb_get_waveform_f64(AlbCtx* ctx, int c, double* out, size_t nbins) {
    if (!ctx || !out || c < 0 || c >= ALB_CHANNELS) return ALB_ERR_INVALID;
    if (nbins < (size_t)ctx->sc.nbins) return fail(ctx, ALB_ERR_INVALID, "waveform buffer too small");
    return read_wf(ctx, c, out);
}

extern "C" int alb_get_jacobian(AlbCtx* ctx, int param, int c, double* out, size_t nbins) {
    if (!ctx || !out || c < 0 || c >= ALB_CHANNELS) return ALB_ERR_INVALID;
    if (param == 0)
        return fail(ctx, ALB_ERR_INVALID, "the depth column is a host-side central difference (no score form)");
    if (param < 1 || param >= ALB_ADJ_PARAMS) return fail(ctx, ALB_ERR_INVALID, "unknown adjoint parameter");
    if (!ctx->jac) return fail(ctx, ALB_ERR_STATE, "ALB_OPT_ADJOINT is not enabled");
    const int64_t nb = ctx->sc.nbins;
    if (nbins < (size_t)nb) return fail(ctx, ALB_ERR_INVALID, "jacobian buffer too small");
    const size_t off = ((size_t)(param - 1) * ALB_CHANNELS + c) * nb;
    const size_t half = (size_t)kJacParams * ALB_CHANNELS * nb;
    return read_fixed(ctx, ctx->jac + off, ctx->jac + half + off, nb, out);
}

extern "C" int alb_adjoint(AlbCtx* ctx, const double* dL_dw, size_t nbins, double* grad) {
    if (!ctx || !dL_dw || !grad) return ALB_ERR_INVALID;
    const int64_t nb = ctx->sc.nbins;
    if (nbins != (size_t)nb) return fail(ctx, ALB_ERR_INVALID, "dL_dw must hold channels * nbins values");
    grad[0] = std::nan("");
    std::vector<double> j(nb);
    for (int p = 1; p < ALB_ADJ_PARAMS; ++p) {
        double acc = 0.0;
        for (int c = 0; c < ALB_CHANNELS; ++c) {
            int rc = alb_get_jacobian(ctx, p, c, j.data(), nb);
            if (rc) return rc;
            for (int64_t i = 0; i < nb; ++i) acc += dL_dw[(size_t)c * nb + i] * j[i];
        }
        grad[p] = acc;
    }
    return ALB_OK;
}

extern "C" int alb_export_map_scores(AlbCtx* ctx, int c, float* scores, size_t n) {
    if (!ctx || !scores || c < 0 || c >= ALB_CHANNELS) return ALB_ERR_INVALID;
    if (!ctx->sc.adjoint) return fail(ctx, ALB_ERR_STATE, "ALB_OPT_ADJOINT is not enabled");
    const uint64_t m = ctx->h_rec_count[c];
    if (n < m) return fail(ctx, ALB_ERR_INVALID, "export buffer smaller than the map");
    if (m == 0) return ALB_OK;
    const float4* s = ctx->rec_released[c] ? ctx->map[c].sco : ctx->rec[c].sco;
    if (!s) return fail(ctx, ALB_ERR_STATE, "records carry no scores");
    CK(cudaMemcpy(scores, s, m * 16, cudaMemcpyDeviceToHost));
    return ALB_OK;
}

extern "C" int alb_reset_waveform(AlbCtx* ctx) {
    if (!ctx) return ALB_ERR_INVALID;
    CK(cudaSetDevice(ctx->device));
    CK(cudaMemsetAsync(ctx->wf, 0, (size_t)2 * ALB_CHANNELS * ctx->sc.nbins * 8, ctx->st));
    if (ctx->hm) CK(cudaMemsetAsync(ctx->hm, 0, (size_t)4 * ctx->sc.hm_bins * ctx->sc.hm_bins * 8, ctx->st));
    if (ctx->jac)
        CK(cudaMemsetAsync(ctx->jac, 0, (size_t)2 * kJacParams * ALB_CHANNELS * ctx->sc.nbins * 8, ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
    return ALB_OK;
}

extern "C" int alb_reset(AlbCtx* ctx) {
    if (!ctx) return ALB_ERR_INVALID;
    CK(cudaSetDevice(ctx->device));
    CK(cudaMemsetAsync(ctx->d_rec_count, 0, ALB_CHANNELS * 8, ctx->st));
    CK(cudaMemsetAsync(ctx->d_q_count, 0, 3 * 8, ctx->st));
    if (ctx->hm_radius)
        CK(cudaMemsetAsync(ctx->hm_radius, 0, (size_t)ctx->sc.hm_bins * ctx->sc.hm_bins * 4, ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
    for (int c = 0; c < ALB_CHANNELS; ++c) {
        ctx->h_rec_count[c] = 0;
        release_map_index(ctx->map[c], ctx->st);  // an empty simulation holds no index memory
        ctx->map[c].n = 0;
        ctx->map[c].n_real = 0;
        ctx->rec_released[c] = false;
    }
    for (int k = 0; k < 3; ++k) ctx->h_q_count[k] = 0;
    ctx->maps_built = false;
    ctx->ex_n = 0;
    return alb_reset_waveform(ctx);
}

extern "C" int alb_export_exit_states(AlbCtx* ctx, double* pos, double* dir, float* energy, float* tau,
                                      float* tau_target, float* time, float* fwi, float* sfi, size_t n) {
    if (!ctx) return ALB_ERR_INVALID;
    if (!ctx->keep_exit || ctx->ex_n == 0) return fail(ctx, ALB_ERR_STATE, "no exit states kept");
    if (n < ctx->ex_n) return fail(ctx, ALB_ERR_INVALID, "exit-state buffer too small");
    uint64_t m = ctx->ex_n;
    std::vector<float> f(10 * m);
    if (pos) CK(cudaMemcpy(pos, ctx->ex_pos, m * 24, cudaMemcpyDeviceToHost));
    if (dir) CK(cudaMemcpy(dir, ctx->ex_dir, m * 24, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(f.data(), ctx->ex_f, m * 40, cudaMemcpyDeviceToHost));
    for (uint64_t i = 0; i < m; ++i) {
        const float* r = f.data() + 10 * i;
        if (energy) energy[i] = r[0];
        if (tau) tau[i] = r[1];
        if (tau_target) tau_target[i] = r[2];
        if (time) time[i] = r[3];
        for (int j = 0; j < 3; ++j) {
            if (fwi) fwi[3 * i + j] = r[4 + j];
            if (sfi) sfi[3 * i + j] = r[7 + j];
        }
    }
    return ALB_OK;
}

extern "C" int alb_query_count(AlbCtx* ctx, int kind, uint64_t* out) {
    if (!ctx || !out || kind < 0 || kind > 2) return ALB_ERR_INVALID;
    *out = ctx->h_q_count[kind];
    return ALB_OK;
}

extern "C" int alb_export_queries(AlbCtx* ctx, int kind, double* pos, float* dir, float* energy, float* time,
                                  int64_t* pid, double* rk, double* rk2, size_t n) {
    if (!ctx || kind < 0 || kind > 2) return ALB_ERR_INVALID;
    uint64_t m = ctx->h_q_count[kind];
    if (n < m) return fail(ctx, ALB_ERR_INVALID, "query buffer too small");
    if (m == 0) return ALB_OK;
    std::vector<float4> a(m), b(m), c(m);
    CK(cudaMemcpy(a.data(), ctx->qa[kind], m * 16, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(b.data(), ctx->qb[kind], m * 16, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(c.data(), ctx->qc[kind], m * 16, cudaMemcpyDeviceToHost));
    std::vector<uint32_t> id;
    if (ctx->qid[kind]) {
        id.resize(m);
        CK(cudaMemcpy(id.data(), ctx->qid[kind], m * 4, cudaMemcpyDeviceToHost));
    }
    if (rk && ctx->qrk[kind][0]) CK(cudaMemcpy(rk, ctx->qrk[kind][0], m * 8, cudaMemcpyDeviceToHost));
    if (rk2 && ctx->qrk[kind][1]) CK(cudaMemcpy(rk2, ctx->qrk[kind][1], m * 8, cudaMemcpyDeviceToHost));
    for (uint64_t i = 0; i < m; ++i) {
        if (pos) {
            pos[3 * i] = (double)a[i].x + (double)c[i].x;
            pos[3 * i + 1] = (double)a[i].y + (double)c[i].y;
            pos[3 * i + 2] = (double)a[i].z + (double)c[i].z;
        }
        if (dir) { dir[3 * i] = b[i].x; dir[3 * i + 1] = b[i].y; dir[3 * i + 2] = b[i].z; }
        if (energy) energy[i] = a[i].w;
        if (time) time[i] = b[i].w;
        if (pid) pid[i] = id.empty() ? -1 : (int64_t)id[i];
    }
    return ALB_OK;
}

extern "C" int alb_knn(AlbCtx* ctx, const float* pts, uint64_t m, const double* qs, uint64_t nq, int k,
                       int32_t* idx, double* dist) {
    if (!ctx || !pts || !qs || !idx || !dist || k < 1 || k > 256) return ALB_ERR_INVALID;
    if (m < (uint64_t)k) return fail(ctx, ALB_ERR_TOO_FEW, "fewer points than k");
    CK(cudaSetDevice(ctx->device));
    // the record's w lane carries its original index (bit pattern) through the sort
    RecordStore r{};
    const size_t mark = ctx->ws.mark();
    r.a = (float4*)ctx->ws.take_bytes(m * 32);  // interleaved store (RecordStore)
    r.b = r.a ? r.a + 1 : nullptr;
    float* dp = (float*)ctx->ws.take_bytes(m * 12);
    double* dq = (double*)ctx->ws.take_bytes(nq * 24);
    float4* qa = (float4*)ctx->ws.take_bytes(nq * 16);
    uint32_t* perm = ctx->ws.take_u32(nq);
    int32_t* di = (int32_t*)ctx->ws.take_bytes(nq * k * 4);
    double* dd = (double*)ctx->ws.take_bytes(nq * k * 8);
    MapIndex mi;
    auto done = [&](int rc) {
        release_map_index(mi, ctx->st);
        dev_free(mi.box_lo, ctx->st);
        dev_free(mi.box_hi, ctx->st);
        ctx->ws.release(mark);
        return rc;
    };
    if (!r.a || !dp || !dq || !qa || !perm || !di || !dd) return done(fail(ctx, ALB_ERR_CUDA, "knn allocation failed"));
    auto ok = [&](cudaError_t e) { return e == cudaSuccess; };
    if (!ok(cudaMemcpyAsync(dp, pts, m * 12, cudaMemcpyHostToDevice, ctx->st)) ||
        !ok(cudaMemcpyAsync(dq, qs, nq * 24, cudaMemcpyHostToDevice, ctx->st)))
        return done(fail(ctx, ALB_ERR_CUDA, "knn upload failed"));
    pack_knn_points(dp, m, r.a, ctx->st);
    if (start_map_index(ctx->ws, r, m, mi, 0, ctx->st) != 0 || finish_map_index(ctx->ws, r, mi, 0, ctx->st) != 0)
        return done(fail(ctx, ALB_ERR_CAPACITY, "knn index build failed"));
    if (nq) pack_knn_queries(dq, nq, qa, ctx->st);
    if (sort_queries(ctx->ws, qa, nq, perm, ctx->st) != 0) return done(fail(ctx, ALB_ERR_CUDA, "knn query sort failed"));
    launch_knn(map_dev(mi), dq, perm, nq, k, di, dd, ctx->d_err, (uint32_t*)ctx->d_err + 1, ctx->st);
    uint32_t crowded = 0;
    int rc = check_device(ctx, "knn", nullptr, &crowded);
    if (!rc && crowded) {
        launch_knn_crowded(map_dev(mi), dq, nq, k, di, dd, ctx->d_err, ctx->st);
        rc = check_device(ctx, "knn");
    }
    if (rc) return done(rc);
    if (!ok(cudaMemcpyAsync(idx, di, nq * k * 4, cudaMemcpyDeviceToHost, ctx->st)) ||
        !ok(cudaMemcpyAsync(dist, dd, nq * k * 8, cudaMemcpyDeviceToHost, ctx->st)) ||
        !ok(cudaStreamSynchronize(ctx->st)))
        return done(fail(ctx, ALB_ERR_CUDA, "knn download failed"));
    return done(ALB_OK);
}

extern "C" int alb_stats(AlbCtx* ctx, int64_t* out, int n) {
    if (!ctx || !out) return ALB_ERR_INVALID;
    unsigned long long s[32];
    CK(cudaMemcpy(s, ctx->d_stats, sizeof s, cudaMemcpyDeviceToHost));
    for (int i = 0; i < n && i < 32; ++i) out[i] = (int64_t)s[i];
    if (n > 2) out[2] = launches_total();
    return ALB_OK;
}

extern "C" int alb_phase_times(AlbCtx* ctx, double* ms, int64_t* calls, int64_t* gathers, int reset) {
    if (!ctx) return ALB_ERR_INVALID;
    for (int i = 0; i < ALB_PHASES; ++i) {
        if (ms) ms[i] = ctx->phase_ms[i];
        if (calls) calls[i] = ctx->phase_calls[i];
    }
    if (gathers)
        for (int c = 0; c < ALB_CHANNELS; ++c) gathers[c] = ctx->gathered[c];
    if (reset) {
        for (int i = 0; i < ALB_PHASES; ++i) {
            ctx->phase_ms[i] = 0.0;
            ctx->phase_calls[i] = 0;
        }
        for (int c = 0; c < ALB_CHANNELS; ++c) ctx->gathered[c] = 0;
    }
    return ALB_OK;
}

// ------------------------------------------------------------------------------------------
// Batched instances (extension)
// ------------------------------------------------------------------------------------------

// Empty the context for the next instance without releasing device memory: stream-ordered
// memsets only, so the other workers' streams keep running.
static int soft_reset(AlbCtx* ctx) {
    const size_t nb = (size_t)ctx->sc.nbins;
    CK(cudaMemsetAsync(ctx->d_rec_count, 0, ALB_CHANNELS * 8, ctx->st));
    CK(cudaMemsetAsync(ctx->d_q_count, 0, 3 * 8, ctx->st));
    CK(cudaMemsetAsync(ctx->wf, 0, 2 * ALB_CHANNELS * nb * 8, ctx->st));
    if (ctx->jac) CK(cudaMemsetAsync(ctx->jac, 0, (size_t)2 * kJacParams * ALB_CHANNELS * nb * 8, ctx->st));
    if (ctx->sc.heatmap) {
        const size_t hb = (size_t)ctx->sc.hm_bins * ctx->sc.hm_bins;
        CK(cudaMemsetAsync(ctx->hm, 0, 4 * hb * 8, ctx->st));
        CK(cudaMemsetAsync(ctx->hm_radius, 0, hb * 4, ctx->st));
    }
    CK(cudaStreamSynchronize(ctx->st));
    for (int c = 0; c < ALB_CHANNELS; ++c) {
        ctx->h_rec_count[c] = 0;
        ctx->map[c].n = 0;
        ctx->map[c].n_real = 0;
        ctx->map[c].nlevels = 0;
    }
    for (int k = 0; k < 3; ++k) ctx->h_q_count[k] = 0;
    ctx->maps_built = false;
    ctx->ex_n = 0;
    return ALB_OK;
}

static int run_instance(AlbCtx* ctx, AlbBatchInstance& I, int adjoint) {
    int rc = alb_trace(ctx, ALB_FORWARD, I.n_forward, I.seed, 0, nullptr);
    if (!rc) rc = alb_build_maps(ctx);
    if (!rc) rc = alb_trace(ctx, ALB_BACKWARD, I.n_backward, I.seed, 0, nullptr);
    if (rc) return rc;
    const int64_t nb = ctx->sc.nbins;
    for (int c = 0; c < ALB_CHANNELS && !rc; ++c)
        if (I.waveform) rc = read_wf(ctx, c, I.waveform + (size_t)c * nb);
    if (!rc && adjoint && I.jacobian)
        for (int p = 1; p < ALB_ADJ_PARAMS && !rc; ++p)
            for (int c = 0; c < ALB_CHANNELS && !rc; ++c)
                rc = alb_get_jacobian(ctx, p, c, I.jacobian + ((size_t)(p - 1) * ALB_CHANNELS + c) * nb, nb);
    return rc;
}

extern "C" int alb_batch_run(AlbBatchInstance* inst, uint64_t n, const AlbBatchOptions* opt) {
    if (!inst || !opt) return ALB_ERR_INVALID;
    if (opt->streams < 1 || opt->streams > 64) {
        g_create_error = "streams must be in [1, 64]";
        return ALB_ERR_INVALID;
    }
    for (uint64_t i = 0; i < n; ++i)
        if (!inst[i].scene) {
            g_create_error = "instance without a scene";
            return ALB_ERR_INVALID;
        }
    // the work queue: largest instances first, so the uneven tail is short
    std::vector<uint64_t> order(n);
    for (uint64_t i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](uint64_t a, uint64_t b) {
        return inst[a].n_forward + inst[a].n_backward > inst[b].n_forward + inst[b].n_backward;
    });
    int64_t max_bins = 0, max_cells = 0;
    for (uint64_t i = 0; i < n; ++i) {
        const AlbSceneParams* sp = inst[i].scene;
        max_bins = std::max<int64_t>(max_bins, sp->gate_bins > 0 ? sp->gate_bins : 2 * sp->steps);
        if (sp->heatmap_enabled) max_cells = std::max<int64_t>(max_cells, (int64_t)sp->heatmap_bins * sp->heatmap_bins);
    }
    std::atomic<uint64_t> next{0};
    std::mutex msg_mu;
    std::string last_msg;
    // Device-memory admission. A context keeps the buffers of the largest instance it ran,
    // so each worker holds an estimate of that footprint against a budget (80% of the free
    // memory at the start); a worker whose next instance needs more waits until the pool
    // has room or it is the only one running, and a worker dropping to instances a quarter
    // of its footprint releases its context. Footprint = forward photons x records per
    // photon (the largest seen so far x 1.5, 200 before any instance finished) x bytes per
    // record (append store, index, build temporaries; scores with the adjoint), + the room that a
    // context's first small call takes beyond those records and keeps (kManyRecords), + the sums of
    // the longest timeline and the largest heatmap (ensure_accumulators), + 64 MiB.
    cudaSetDevice(opt->device);
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const double budget = 0.8 * ((double)free_b + (double)pool_idle());
    const double bytes_per_record = opt->adjoint ? 162.0 : 130.0;
    std::mutex mem_mu;
    std::condition_variable mem_cv;
    double held_total = 0.0, rpp_seen = 0.0;
    int running = 0;
    int exclusive = 0;  // workers waiting to rerun an instance alone; the others hold no memory then
    const double sums = accumulator_bytes(max_bins, opt->adjoint != 0, max_cells) + 64.0 * 1048576.0;
    auto need_of = [&](const AlbBatchInstance& I) {
        const double rpp = rpp_seen > 0.0 ? 1.5 * rpp_seen : 200.0;
        const double spare = I.n_forward <= kSmallCall ? std::max(0.0, first_call_records() - rpp) : 0.0;
        const double bytes_per_spare = 32.0 + (opt->adjoint ? 16.0 : 0.0) + (max_cells ? 32.0 : 0.0);
        return (double)I.n_forward * (rpp * bytes_per_record + spare * bytes_per_spare) + sums;
    };
    auto worker = [&]() {
        cudaSetDevice(opt->device);
        t_direct = kDirectBatch;
        double held = 0.0;
        cudaStream_t st = nullptr;
        if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) st = nullptr;
        AlbCtx* ctx = nullptr;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        bool alone = false;  // the retry of an instance that ran out of memory beside others
        for (uint64_t t = next.fetch_add(1); t < n; t = alone ? t : next.fetch_add(1)) {
            AlbBatchInstance& I = inst[order[t]];
            I.device_ms = 0.f;
            int rc = ALB_OK;
            std::string msg;
            bool shared = false;  // other instances were running when this one started
            {
                std::unique_lock<std::mutex> g(mem_mu);
                const double need = need_of(I);
                auto drop_ctx = [&]() {  // release this worker's context and its device memory
                    g.unlock();
                    alb_destroy(ctx);
                    ctx = nullptr;
                    g.lock();
                    held_total -= held;
                    held = 0.0;
                    mem_cv.notify_all();
                };
                while (true) {
                    if (!alone && exclusive > 0) {  // another worker reruns an instance alone
                        if (ctx) drop_ctx();
                        mem_cv.wait(g, [&] { return exclusive == 0; });
                        continue;
                    }
                    if (ctx && held > (double)(1 << 30) && 4.0 * need < held) drop_ctx();  // small tail
                    const double grow = std::max(0.0, need - held);
                    mem_cv.wait(g, [&] {
                        if (!alone && exclusive > 0) return true;
                        // a rerun alone waits until no instance runs and every other worker
                        // has released its context (a worker that has just finished an
                        // instance still holds its buffers until it comes back here); this
                        // worker's own holding does not count
                        return alone ? (running == 0 && held_total - held <= 0.5)
                                     : (held_total + grow <= budget || running == 0);
                    });
                    if (!alone && exclusive > 0) continue;
                    held_total += grow;
                    held += grow;
                    shared = running > 0;
                    ++running;
                    break;
                }
            }
            if (!ctx) {
                rc = create_on(I.scene, opt->device, st, &ctx);
                if (rc) {
                    msg = g_create_error;
                    ctx = nullptr;
                } else {
                    alb_set_option(ctx, ALB_OPT_PRECISE, opt->precise ? 1 : 0);
                    ctx->keep_records = true;
                    if (opt->adjoint) rc = alb_set_option(ctx, ALB_OPT_ADJOINT, 1);
                    if (!rc) {  // accumulators for the longest instance: no regrowth later
                        const int64_t own = ctx->sc.nbins;
                        ctx->sc.nbins = max_bins;
                        std::string e = ensure_accumulators(ctx);
                        ctx->sc.nbins = own;
                        if (!e.empty()) rc = fail(ctx, ALB_ERR_CUDA, e);
                        else if (cudaStreamSynchronize(ctx->st) != cudaSuccess) rc = fail(ctx, ALB_ERR_CUDA, "reserve");
                    }
                    if (rc) msg = ctx->err;
                }
            } else {
                std::string e = set_scene(ctx, I.scene);
                if (e.empty()) e = ensure_accumulators(ctx);
                if (!e.empty()) {
                    rc = ALB_ERR_INVALID;
                    msg = e;
                } else {
                    rc = soft_reset(ctx);
                    if (rc) msg = ctx->err;
                }
            }
            // with the adjoint option, an instance without a Jacobian buffer runs plain
            const int adj = opt->adjoint && I.jacobian ? 1 : 0;
            if (!rc && ctx && ctx->sc.adjoint != adj) {
                rc = alb_set_option(ctx, ALB_OPT_ADJOINT, adj);
                if (rc) msg = ctx->err;
            }
            if (!rc && ctx) {
                cudaEventRecord(e0, ctx->st);
                rc = run_instance(ctx, I, adj);
                cudaEventRecord(e1, ctx->st);
                cudaEventSynchronize(e1);
                cudaEventElapsedTime(&I.device_ms, e0, e1);
                if (rc) msg = ctx->err;
            }
            {
                std::lock_guard<std::mutex> g(mem_mu);
                if (!rc && ctx && I.n_forward > 0) {
                    uint64_t recs = 0;
                    for (int c = 0; c < ALB_CHANNELS; ++c) recs += ctx->h_rec_count[c];
                    rpp_seen = std::max(rpp_seen, (double)recs / (double)I.n_forward);
                }
                --running;
                mem_cv.notify_all();
            }
            I.status = rc;
            if (rc) {
                std::lock_guard<std::mutex> g(msg_mu);
                last_msg = msg;
                if (ctx && (rc == ALB_ERR_CUDA || rc == ALB_ERR_ITER_CAP || rc == ALB_ERR_CAPACITY)) {
                    alb_destroy(ctx);  // start the next instance clean
                    ctx = nullptr;
                }
                if (!ctx) {  // no context (destroyed, or never created): this worker holds nothing
                    std::lock_guard<std::mutex> m(mem_mu);
                    held_total -= held;
                    held = 0.0;
                    mem_cv.notify_all();
                }
            }
            // Device memory is admitted on an estimate: an instance that failed for memory
            // (an allocation or a map build) while others were running is run once more,
            // alone, once every other worker has released its context.
            const bool memory = rc == ALB_ERR_CUDA || rc == ALB_ERR_CAPACITY;
            const bool was_alone = alone;
            alone = memory && shared && !alone && cudaGetLastError() != cudaErrorIllegalAddress;
            if (alone || was_alone) {
                std::lock_guard<std::mutex> m(mem_mu);
                exclusive += alone ? 1 : -1;
                mem_cv.notify_all();
            }
        }
        if (ctx) alb_destroy(ctx);
        {
            std::lock_guard<std::mutex> g(mem_mu);
            held_total -= held;
            mem_cv.notify_all();
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (st) cudaStreamDestroy(st);
    };
    std::vector<std::thread> pool;
    const int K = (int)std::min<uint64_t>((uint64_t)opt->streams, std::max<uint64_t>(n, 1));
    for (int w = 0; w < K; ++w) pool.emplace_back(worker);
    for (auto& th : pool) th.join();
    g_create_error = last_msg;
    return ALB_OK;
}
