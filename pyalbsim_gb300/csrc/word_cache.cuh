// Sums of 64-bit words in global memory, some of them held in a CTA's shared memory (included by gather.cu).
#pragma once
#include "device_common.cuh"

namespace alb {

// Per-CTA cache of class words for gathers whose neighbours share a few of them: adds to the same sector
// of L2 come one per cycle, and one slice took 1.4 a nanosecond of the scatter gather of the default
// scene, whose first-water cells lie in one narrow beam. With heatmaps, 6.2e5 queries: 4.4 -> 3.9 ms; a
// waveform of 126 bins, 3.1e5 queries: 4.7 -> 2.7; the Jacobian of the gradient's surface gather, 2.5e5
// queries: 7.9 -> 3.5. Direct-mapped, a slot claimed once by CAS on its
// tag; a word is held as two 32-bit ones, which shared memory adds natively. Key: the word's number in
// its array, plus `base` for the second of the two arrays that cache_flush writes. on == false: arrays
// whose keys would not fit 32 bits, every add goes straight to its word.
template <int N>
struct WordCache {
    static constexpr int kSlots = N;
    uint32_t tag[N], lo[N], hi[N];
};
struct NoCache {};
ALB_DEVICE void word_add(NoCache&, bool, unsigned long long* words, uint64_t i, uint32_t, uint32_t, long long v) {
    atomicAdd(words + i, (unsigned long long)v);
}
template <int N>
ALB_DEVICE void word_add(WordCache<N>& wc, bool on, unsigned long long* words, uint64_t i, uint32_t base, uint32_t hash,
                         long long v) {
    const uint32_t slot = hash % N, key = base + (uint32_t)i;
    uint32_t t = on ? wc.tag[slot] : ~key;
    if (on && t == 0xffffffffu) {
        t = atomicCAS(&wc.tag[slot], 0xffffffffu, key);
        if (t == 0xffffffffu) t = key;
    }
    if (t == key) {
        const uint32_t lo = (uint32_t)v, old = atomicAdd(&wc.lo[slot], lo);
        const uint32_t up = (uint32_t)((unsigned long long)v >> 32) + (old + lo < old ? 1u : 0u);
        if (up) atomicAdd(&wc.hi[slot], up);
    } else {
        atomicAdd(words + i, (unsigned long long)v);
    }
}
ALB_DEVICE void cache_clear(NoCache&) {}
template <int N>
ALB_DEVICE void cache_clear(WordCache<N>& wc) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        wc.tag[i] = 0xffffffffu;
        wc.lo[i] = wc.hi[i] = 0u;
    }
}
// (after a block barrier)
ALB_DEVICE void cache_flush(const NoCache&, unsigned long long*, uint32_t, unsigned long long*) {}
template <int N>
ALB_DEVICE void cache_flush(const WordCache<N>& wc, unsigned long long* first, uint32_t n, unsigned long long* second) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const uint32_t t = wc.tag[i];
        if (t != 0xffffffffu)
            atomicAdd(t < n ? first + t : second + (t - n), (unsigned long long)wc.hi[i] << 32 | wc.lo[i]);
    }
}

}  // namespace alb
