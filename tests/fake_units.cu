// Stand-ins of the units that launch kernels (tracer, map build, gather) for the host code on fake_runtime.cpp.
#include "albgpu.h"
#include "fake_cuda.h"
#include "internal.h"
#include "tracer_fast.cuh"

namespace alb {

void launch_trace(const SceneDev&, const TraceOut& out, int pass, uint64_t n, uint64_t, uint64_t, const AlbReplay*, int*,
                  cudaStream_t st, const FastScene*) {
    fake::on_device(out.rec_count, "trace");
    fake::launched(st);
    fake::traced(n);  // takes the time that a test sets
    if (const int e = fake::trace_error()) *out.err = e;
    if (pass == ALB_FORWARD && out.hm_radius) out.hm_radius[0] += (unsigned)n;
    if (pass == ALB_FORWARD)
        for (int c = 0; c < 4; ++c) out.rec_count[c] += (unsigned long long)(fake::record_rate(c) * (double)n);
    else
        for (int k = 0; k < 3; ++k) out.q_count[k] += (unsigned long long)(fake::query_rate(k) * (double)n);
}
void launch_phase_tables(const double* cdf, const double*, const double*, float*, uint16_t*, cudaStream_t st) {
    fake::on_device(cdf, "phase tables");
    fake::launched(st);
}
void launch_profile_logs(const SceneDev&, double* out, cudaStream_t st) {
    fake::on_device(out, "profile logs");
    fake::launched(st);
}
void launch_gather(const SceneDev&, const MapDev& m, const QueryDev& q, int, const Accum& acc, int*, int*, cudaStream_t st) {
    fake::on_device(m.a, "gather");
    fake::on_device(q.a, "gather");
    fake::on_device(acc.wf_lo, "gather");
    fake::on_device(acc.cls, "gather");
    fake::on_device(acc.jac_lo, "gather");
    fake::on_device(acc.jac_cls, "gather");
    fake::launched(st);
}
template <class T>
static void fix_to_float(const unsigned long long* lo, const unsigned long long* hi, int64_t n, T* out, cudaStream_t st) {
    fake::on_device(lo, "read-back");
    fake::on_device(hi, "read-back");
    fake::on_device(out, "read-back");
    fake::launched(st);
    for (int64_t i = 0; i < n; ++i) out[i] = (T)fix_to_double(lo[i], (long long)hi[i]);
}
void launch_fix_to_float(const unsigned long long* lo, const unsigned long long* hi, int64_t n, float* out, cudaStream_t st) {
    fix_to_float(lo, hi, n, out, st);
}
void launch_fix_to_float(const unsigned long long* lo, const unsigned long long* hi, int64_t n, double* out, cudaStream_t st) {
    fix_to_float(lo, hi, n, out, st);
}
void launch_knn(const MapDev&, const double*, const uint32_t*, uint64_t, int, int32_t*, double*, int*, uint32_t*, cudaStream_t) {}
void launch_knn_crowded(const MapDev&, const double*, uint64_t, int, int32_t*, double*, int*, cudaStream_t) {}
void launch_gather_crowded(const SceneDev&, const MapDev&, const QueryDev&, int, const Accum&, int*, cudaStream_t) {}
void launch_knn_brute(const float*, uint32_t, const double*, uint64_t, int, int32_t*, double*, cudaStream_t) {}
void pack_knn_points(const float*, uint64_t, float4*, cudaStream_t) {}
void pack_knn_queries(const double*, uint64_t, float4*, cudaStream_t) {}

int start_map_index(Workspace& ws, const RecordStore& rec, uint64_t n, MapIndex& m, int, cudaStream_t st) {
    m.n = m.n_real = n;
    m.nlevels = n ? 1 : 0;
    if (!n) return 0;
    fake::on_device(rec.a, "map build");
    m.a = (float4*)ws.alloc_persistent(m.a, m.a_cap, n);
    m.b = (float4*)ws.alloc_persistent(m.b, m.b_cap, n);
    if (!m.a || !m.b) return -1;
    fake::launched(st);
    for (uint64_t i = 0; i < n; ++i) {
        m.a[i] = rec.a[2 * i];
        m.b[i] = rec.b[2 * i];
    }
    return 0;
}
int finish_map_index(Workspace&, const RecordStore&, MapIndex&, int, cudaStream_t st) {
    return cudaStreamSynchronize(st) == cudaSuccess ? 0 : -1;
}
void release_map_index(MapIndex& m, cudaStream_t st) {
    dev_free(m.a, st);
    dev_free(m.b, st);
    m.a = m.b = nullptr;
    m.a_cap = m.b_cap = 0;
}
int sort_queries(Workspace& ws, const float4* qa, uint64_t n, uint32_t* perm, cudaStream_t st) {
    if (!n) return 0;
    fake::on_device(qa, "query sort");
    fake::on_device(perm, "query sort");
    const size_t mark = ws.mark();
    const bool ok = ws.take_u32(n) != nullptr;
    ws.release(mark);
    fake::launched(st);
    return ok ? 0 : -1;
}

}  // namespace alb
