// Device functions of the library, called on arrays (test_gpu_device_functions.py).
#include <cstdint>

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
