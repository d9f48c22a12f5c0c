// A CUDA runtime of host memory for the library's host code: linked with albgpu.cu and noalloc.cu in place of
// libcudart and of the units that launch kernels, so that what the host does on an error or with several
// devices runs without a GPU. Two devices; a device's memory has a limit that a test sets; a traced photon
// leaves a fixed number of records and queries. Every launch, memset and free is checked: memory on the
// device that is current, nothing freed while another stream still works.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>

#include "fake_cuda.h"

namespace {

constexpr int kDevices = 2;
struct Block {
    uint64_t bytes;
    int device;
};
struct State {
    std::map<uintptr_t, Block> blocks;
    std::map<cudaEvent_t, cudaStream_t> events;  // the stream an event was last recorded on
    std::set<cudaStream_t> busy;
    uint64_t used[kDevices] = {0, 0}, limit[kDevices] = {~0ull, ~0ull}, peak[kDevices] = {0, 0};
    double rec[4] = {1, 8, 1, 1}, query[3] = {1, 8, 1};
    int fail_record = 0;  // the n-th event record from now fails (0: none)
    uint64_t traced = 0;  // photons of every trace
    int trace_ms = 0, trace_error = 0;
    int trims[kDevices] = {0, 0};
    int violations = 0;
    std::string what;
};
std::recursive_mutex mu;
State* g = new State;
thread_local int current = 0;
using Lock = std::lock_guard<std::recursive_mutex>;

void violation(const std::string& s) {
    ++g->violations;
    g->what += s + "\n";
}

const Block* block_of(const void* p) {
    auto it = g->blocks.upper_bound((uintptr_t)p);
    if (it == g->blocks.begin()) return nullptr;
    --it;
    return (uintptr_t)p < it->first + it->second.bytes ? &it->second : nullptr;
}

}  // namespace

void fake::on_device(const void* p, const char* where) {
    Lock l(mu);
    const Block* b = p ? block_of(p) : nullptr;
    if (p && !b) violation(std::string(where) + ": not device memory");
    else if (b && b->device != current) violation(std::string(where) + ": memory of another device than the current one");
}

void fake::launched(cudaStream_t st) {
    Lock l(mu);
    g->busy.insert(st);
}
void fake::traced(uint64_t photons) {
    std::this_thread::sleep_for(std::chrono::milliseconds(g->trace_ms));
    Lock l(mu);
    g->traced += photons;
}
double fake::record_rate(int channel) { return g->rec[channel]; }
double fake::query_rate(int kind) { return g->query[kind]; }
int fake::trace_error() {
    const int e = g->trace_error;
    g->trace_error = 0;
    return e;
}

namespace {

cudaError_t allocate(void** p, uint64_t bytes, int device) {
    Lock l(mu);
    if (g->used[device] + bytes > g->limit[device]) return cudaErrorMemoryAllocation;
    *p = calloc(bytes + 32, 1);
    g->blocks[(uintptr_t)*p] = Block{bytes + 32, device};
    g->used[device] += bytes + 32;
    if (g->used[device] > g->peak[device]) g->peak[device] = g->used[device];
    return cudaSuccess;
}

cudaError_t release(void* p, cudaStream_t st, bool waits) {
    Lock l(mu);
    if (!p) return cudaSuccess;
    auto it = g->blocks.find((uintptr_t)p);
    if (it == g->blocks.end()) {
        violation("free of what is no block");
        return cudaErrorInvalidValue;
    }
    for (cudaStream_t s : g->busy)
        if (!waits && s != st) violation("free while another stream works");
    g->used[it->second.device] -= it->second.bytes;
    g->blocks.erase(it);
    free(p);
    return cudaSuccess;
}

}  // namespace

extern "C" {

void fake_reset() {
    Lock l(mu);
    for (auto& b : g->blocks) free((void*)b.first);
    *g = State();
    current = 0;
}
void fake_limit(int device, uint64_t bytes) { g->limit[device] = bytes; }
uint64_t fake_used(int device) { return g->used[device]; }
uint64_t fake_peak(int device) { return g->peak[device]; }
uint64_t fake_traced() { return g->traced; }
void fake_rates(const double* rec, const double* query) {
    memcpy(g->rec, rec, sizeof g->rec);
    memcpy(g->query, query, sizeof g->query);
}
void fake_trace_ms(int ms) { g->trace_ms = ms; }
void fake_fail_trace(int code) { g->trace_error = code; }
void fake_fail_record(int n) { g->fail_record = n; }
int fake_violations(char* out, int n) {
    snprintf(out, n, "%s", g->what.c_str());
    return g->violations;
}
int fake_trims(int device) { return g->trims[device]; }
int fake_events() { return (int)g->events.size(); }
int fake_busy() { return (int)g->busy.size(); }

void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}

cudaError_t cudaGetDevice(int* d) {
    *d = current;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d >= kDevices) return cudaErrorInvalidDevice;
    current = d;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceSynchronize() {
    Lock l(mu);
    g->busy.clear();
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n, current); }
cudaError_t cudaFree(void* p) { return release(p, nullptr, true); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
    return allocate(p, n, (int)(uintptr_t)pool - 1);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t st) { return release(p, st, false); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    Lock l(mu);
    *t = g->limit[current] == ~0ull ? 1ull << 40 : g->limit[current];
    *f = *t - g->used[current];
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps* props) {
    *pool = (cudaMemPool_t)(uintptr_t)(props->location.id + 1);
    return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) {
    *(uint64_t*)v = 0;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t) {
    Lock l(mu);
    ++g->trims[(uintptr_t)pool - 1];
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
    for (size_t i = 0; i < h; ++i) memmove((char*)d + i * dp, (const char*)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind k, cudaStream_t) {
    return cudaMemcpy2D(d, dp, s, sp, w, h, k);
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    Lock l(mu);
    fake::on_device(d, "memset");
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    Lock l(mu);
    g->busy.erase(s);
    free((void*)s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    Lock l(mu);
    g->busy.erase(s);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    Lock l(mu);
    const cudaStream_t from = g->events[e];
    if (from != s && g->busy.erase(from)) g->busy.insert(s);  // s goes on when that stream's work is done
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    Lock l(mu);
    *e = (cudaEvent_t)malloc(1);
    g->events[*e] = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    Lock l(mu);
    g->events.erase(e);
    free((void*)e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    Lock l(mu);
    if (g->fail_record && --g->fail_record == 0) return cudaErrorInvalidResourceHandle;
    g->events[e] = s;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}

}  // extern "C"
