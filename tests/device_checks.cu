// Device functions of the library, called on arrays (test_gpu_device_functions.py).
#include <cstdint>

#include "tracer.cuh"
#include "word_cache.cuh"

using namespace alb;

// One warp adds v[j] to word i[j] with the given key base; out: words `first` and `second` after the flush.
__global__ void k_word_cache(unsigned long long* words, const uint64_t* i, const uint32_t* base, const long long* v, int n, int on,
                             unsigned long long* first, uint32_t n_first, unsigned long long* second) {
    __shared__ WordCache<8> cache;
    cache_clear(cache);
    __syncthreads();
    if ((int)threadIdx.x < n)
        word_add(cache, on != 0, words, i[threadIdx.x], base[threadIdx.x], (uint32_t)i[threadIdx.x], v[threadIdx.x]);
    __syncthreads();
    cache_flush(cache, first, n_first, second);
}

extern "C" int check_word_cache(void* words, const void* i, const void* base, const void* v, int n, int on, void* first,
                                uint32_t n_first, void* second) {
    k_word_cache<<<1, 32>>>((unsigned long long*)words, (const uint64_t*)i, (const uint32_t*)base, (const long long*)v, n, on,
                            (unsigned long long*)first, n_first, (unsigned long long*)second);
    return (int)cudaDeviceSynchronize();
}

// Whether the step counts of the float64 tracer are the smallest n with y0 + n sy <= lim (down) or > lim (up), or
// nmax + 1 where no n <= nmax is: bad[0] counts the others.
__global__ void k_steps(const double* y0, const double* sy, const double* lim, int64_t n, int64_t nmax, unsigned long long* bad) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const bool down = sy[i] < 0.0;
        const int64_t m = down ? first_at_or_below(y0[i], sy[i], lim[i], nmax) : first_above(y0[i], sy[i], lim[i], nmax);
        auto past = [&](int64_t k) {
            const double y = fma((double)k, sy[i], y0[i]);
            return down ? y <= lim[i] : y > lim[i];
        };
        const bool ok = m >= 1 && m <= nmax + 1 && (m == nmax + 1 || past(m)) && (m == 1 || !past(m - 1));
        if (!ok) atomicAdd(bad, 1ull);
    }
}

extern "C" int check_steps(const void* y0, const void* sy, const void* lim, int64_t n, int64_t nmax, void* bad) {
    k_steps<<<512, 256>>>((const double*)y0, (const double*)sy, (const double*)lim, n, nmax, (unsigned long long*)bad);
    return (int)cudaDeviceSynchronize();
}

// Quotients by a constant against the division operator: bad[0] counts float32 ones, bad[1] float64 ones.
__global__ void k_quotients(const double* x, const double* b, int64_t n, unsigned long long* bad) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float xf = (float)x[i], bf = (float)b[i];
        if (div_by(xf, bf, __fdiv_rn(1.0f, bf)) != __fdiv_rn(xf, bf)) atomicAdd(bad, 1ull);
        if (div64_by(x[i], b[i], __drcp_rn(b[i])) != __ddiv_rn(x[i], b[i])) atomicAdd(bad + 1, 1ull);
    }
}

extern "C" int check_quotients(const void* x, const void* b, int64_t n, void* bad) {
    k_quotients<<<512, 256>>>((const double*)x, (const double*)b, n, (unsigned long long*)bad);
    return (int)cudaDeviceSynchronize();
}
