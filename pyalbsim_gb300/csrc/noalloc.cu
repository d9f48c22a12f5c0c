// alb_knn_noalloc: k-nearest-neighbour queries that allocate no device memory.
//
// Some callers of this library cannot call cudaMalloc: code running while a stream is
// being captured into a CUDA graph (a cudaMalloc there breaks the capture), a real-time
// acquisition loop that may only allocate at start-up, or a process whose device memory is
// owned by another framework's pool (a second allocator would exceed its budget). They
// already hold the input and output buffers, and this entry point works in those alone: one
// kernel screens every point for every query (k_knn_brute), which for at most
// ALB_NOALLOC_MAX_POINTS points costs what a search over an index does, without the index.
// Nothing is shared between calls: calls on different streams or from several host threads
// may overlap.
#include <string>

#include "albgpu.h"
#include "internal.h"

namespace alb {
void set_global_error(const std::string& msg);
}  // namespace alb

using namespace alb;

extern "C" int alb_knn_noalloc(const float* points_dev, uint64_t m, const double* queries_dev, uint64_t q, int k,
                               int32_t* idx_dev, double* dist_dev, void* stream) {
    if (!points_dev || !queries_dev || !idx_dev || !dist_dev) {
        set_global_error("alb_knn_noalloc: null buffer");
        return ALB_ERR_INVALID;
    }
    if (k < 1 || k > 256) {
        set_global_error("alb_knn_noalloc: k must be in [1, 256]");
        return ALB_ERR_INVALID;
    }
    if (m > ALB_NOALLOC_MAX_POINTS) {
        set_global_error("alb_knn_noalloc: at most " + std::to_string(ALB_NOALLOC_MAX_POINTS) + " points per call (got " +
                         std::to_string(m) + ")");
        return ALB_ERR_INVALID;
    }
    if (m < (uint64_t)k) {
        set_global_error("alb_knn_noalloc: fewer points than k");
        return ALB_ERR_TOO_FEW;
    }
    if (q == 0) return ALB_OK;
    int dev = 0;
    const cudaError_t ge = cudaGetDevice(&dev);
    if (ge != cudaSuccess) {
        set_global_error(std::string("alb_knn_noalloc: no usable current device: ") + cudaGetErrorString(ge));
        return ALB_ERR_CUDA;
    }
    launch_knn_brute(points_dev, (uint32_t)m, queries_dev, q, k, idx_dev, dist_dev, (cudaStream_t)stream);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_global_error(std::string("alb_knn_noalloc: launch failed: ") + cudaGetErrorString(e));
        return ALB_ERR_CUDA;
    }
    return ALB_OK;
}
