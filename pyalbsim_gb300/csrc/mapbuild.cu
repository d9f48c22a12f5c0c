// Photon-map index build: the GPU replacement of build_photon_map_data + PhotonMapIndex
// (alb_sim/photon_mapping/build_photon_map_data.py:8-62, photon_map_index.py:6-17).
//
// Records are sorted along a Hilbert curve (LSD radix sort of 24- or 32-bit keys on cubic cells),
// every 256 consecutive ones are cut into eight k-d leaves of 32 by a warp, and permuted into that
// order as two float4 streams. A leaf's bounding box is a leaf box; 32 consecutive boxes form the
// next level up, until 32 or fewer boxes remain. The gather walks this implicit 32-ary box tree
// warp-wide. Record sets whose box is far larger than what they fill (keys that do not tell them
// apart) take an exact left-balanced k-d order instead (median splits on each node's widest axis;
// streaming partition passes for the upper levels, one CTA per node of at most 4096 records for
// the rest). The same sort orders the gather queries.
#include <atomic>
#include <algorithm>
#include <cstdio>

#include "device_common.cuh"
#include "internal.h"

namespace alb {

// ------------------------------------------------------------------------------------------
// bounding box
// ------------------------------------------------------------------------------------------

ALB_DEVICE unsigned f2ord(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
ALB_HOST_DEVICE float ord2f(unsigned u) {
    unsigned b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    float f;
    memcpy(&f, &b, 4);
    return f;
}

// box[0..2] = ordered-min of x,y,z, box[3..5] = ordered-max; initialised to (~0, 0).
__global__ void k_bbox(const float4* __restrict__ a, uint64_t stride, uint64_t n, unsigned* box) {
    float lo[3] = {3.4e38f, 3.4e38f, 3.4e38f}, hi[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        float4 p = a[i * stride];
        float x = p.x, y = p.y, z = p.z;
        lo[0] = fminf(lo[0], x); hi[0] = fmaxf(hi[0], x);
        lo[1] = fminf(lo[1], y); hi[1] = fmaxf(hi[1], y);
        lo[2] = fminf(lo[2], z); hi[2] = fmaxf(hi[2], z);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    }
    // the block's warps meet in shared memory: one set of global atomics per block (they
    // all land on the same six words)
    __shared__ unsigned sb[6];
    if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            atomicMin(sb + k, f2ord(lo[k]));
            atomicMax(sb + 3 + k, f2ord(hi[k]));
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(box + threadIdx.x, sb[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(box + threadIdx.x, sb[threadIdx.x]);
}

// ------------------------------------------------------------------------------------------
// Hilbert keys on cubic cells (24 to 48 bits): the order of gather queries and of map records
//
// The gather's cost per query follows how far consecutive queries lie apart (search bounds are
// carried from one to the next, and neighbouring warps share leaves in L1 and L2), so the cells
// have the same size on every axis and the curve has no jumps: at the bench geometry (a query
// box of 330 x 20 x 330 m) the median step between consecutive queries is 0.43 k-th distances,
// against 0.46 on a Morton curve over the same cells and 0.95 on a Morton curve of 10 bits per
// axis, whose cells are 16 times flatter than they are wide.
// ------------------------------------------------------------------------------------------

// Key layout for a box: axes in order of extent (ax[0] the longest), cells of edge 1 / inv.
// 3 axes: the box is cut into cubes of 2^m cells per axis, m from the shortest extent; the
// cubes follow a 2-D Hilbert curve over the two longer axes (hi bits each), the cells of a cube
// a 3-D one. 2 axes: one 2-D curve of hi bits. 1 axis: the cell number (hi bits).
struct KeyGrid {
    float lo[3];
    float inv;
    int ax[3];
    int naxes, m, hi;
};

// Hilbert index of 2 or 3 coordinates of `bits` bits, from the top level down: the octant is
// mapped through the curve's entry corner e and axis d of the current cube, its Gray rank is the
// key's next digit, and e and d follow the curve into that octant (Hamilton, "Compact Hilbert
// indices", Dalhousie CS-2006-07). The curve's state is e + 8 d (e + 4 d in the plane); step3 and step2 take
// octant o and leave the digit and the next state. The keys take two levels (three in the plane) at a
// time from a table in shared memory: 1.12e8 keys of 48 bits level by level 3.2 ms, by table 1.1.
ALB_HOST_DEVICE constexpr uint32_t step3(uint32_t& state, uint32_t o) {
    uint32_t e = state & 7u, d = state >> 3;
    o ^= e;
    const uint32_t r = d == 2u ? 0u : d + 1u;
    o = ((o * 9u) >> r) & 7u;                            // rotated right by d + 1 of 3 bits
    const uint32_t w = (0x54672310u >> (4u * o)) & 7u;   // inverse Gray code: 0 1 3 2 7 6 4 5
    const uint32_t en = (0x56633000u >> (4u * w)) & 7u;  // entry corners: 0 0 0 3 3 6 6 5
    e ^= (((en * 9u) << r) >> 3) & 7u;                   // rotated left by d + 1
    d += ((0x01122110u >> (4u * w)) & 3u) + 1u;          // directions: 0 1 1 2 2 1 1 0
    state = e | (d >= 3u ? d - 3u : d) << 3;
    return w;
}
ALB_HOST_DEVICE constexpr uint32_t step2(uint32_t& state, uint32_t o) {
    uint32_t e = state & 3u, d = state >> 2;
    o ^= e;
    o = d ? o : (((o << 1) | (o >> 1)) & 3u);  // rotated by d + 1 of 2 bits
    const uint32_t w = o ^ (o >> 1);           // inverse Gray code: 0 1 3 2
    e ^= w == 3u ? 3u : 0u;                    // entry corners: 0 0 0 3
    d ^= (w == 0u || w == 3u) ? 1u : 0u;       // directions 0 1 1 0, plus 1, of 2
    state = e | d << 2;
    return w;
}

// [state][coordinate bits, the first coordinate's lowest] -> next state << 6 | six bits of key
struct HilbertTables {
    uint16_t t3[24 * 64];  // two bits of each of three coordinates
    uint16_t t2[8 * 64];   // three bits of each of two
};
constexpr HilbertTables hilbert_tables() {
    HilbertTables t{};
    for (uint32_t s = 0; s < 24; ++s)
        for (uint32_t i = 0; i < 64; ++i) {
            const uint32_t x = i & 3u, y = i >> 2 & 3u, z = i >> 4;
            uint32_t state = s;
            const uint32_t a = step3(state, x >> 1 | (y >> 1) << 1 | (z >> 1) << 2);
            const uint32_t b = step3(state, (x & 1u) | (y & 1u) << 1 | (z & 1u) << 2);
            t.t3[s * 64 + i] = (uint16_t)(state << 6 | a << 3 | b);
        }
    for (uint32_t s = 0; s < 8; ++s)
        for (uint32_t i = 0; i < 64; ++i) {
            const uint32_t x = i & 7u, y = i >> 3;
            uint32_t state = s, key = 0;
            for (int b = 2; b >= 0; --b) key = key << 2 | step2(state, (x >> b & 1u) | (y >> b & 1u) << 1);
            t.t2[s * 64 + i] = (uint16_t)(state << 6 | key);
        }
    return t;
}
__device__ const HilbertTables kHilbertTables = hilbert_tables();

template <class K>
ALB_DEVICE K hilbert_key3(const HilbertTables& t, uint32_t x, uint32_t y, uint32_t z, int bits) {
    K key = 0;
    uint32_t s = 0u;
    int b = bits;
    if (b & 1) {
        --b;
        key = step3(s, (x >> b & 1u) | (y >> b & 1u) << 1 | (z >> b & 1u) << 2);
    }
#pragma unroll 2
    while (b > 0) {
        b -= 2;
        const uint32_t v = t.t3[s * 64u + ((x >> b & 3u) | (y >> b & 3u) << 2 | (z >> b & 3u) << 4)];
        key = (key << 6) | (v & 63u);
        s = v >> 6;
    }
    return key;
}
template <class K>
ALB_DEVICE K hilbert_key2(const HilbertTables& t, uint32_t x, uint32_t y, int bits) {
    K key = 0;
    uint32_t s = 0u;
    int b = bits;
    for (int odd = bits % 3; odd > 0; --odd) {
        --b;
        key = (key << 2) | step2(s, (x >> b & 1u) | (y >> b & 1u) << 1);
    }
#pragma unroll 2
    while (b > 0) {
        b -= 3;
        const uint32_t v = t.t2[s * 64u + ((x >> b & 7u) | (y >> b & 7u) << 3)];
        key = (key << 6) | (v & 63u);
        s = v >> 6;
    }
    return key;
}

// `box` as left by k_bbox; total: key bits to spend (24, 32 or 48).
ALB_DEVICE KeyGrid make_key_grid(const unsigned* box, int total) {
    KeyGrid g;
    float e[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        g.lo[k] = ord2f(box[k]);
        e[k] = ord2f(box[3 + k]) - g.lo[k];
        if (!(e[k] > 0.f)) e[k] = 0.f;  // also NaN
    }
    int a0 = 0, a1 = 1, a2 = 2, t;
    if (e[a0] < e[a1]) { t = a0; a0 = a1; a1 = t; }
    if (e[a1] < e[a2]) { t = a1; a1 = a2; a2 = t; }
    if (e[a0] < e[a1]) { t = a0; a0 = a1; a1 = t; }
    g.ax[0] = a0; g.ax[1] = a1; g.ax[2] = a2;
    const float emax = fminf(e[a0], 1.0e30f);
    // an axis with (almost) no extent carries no key bits (planar surface / floor queries)
    g.naxes = !(emax > 0.f) ? 0 : (!(e[a1] > 1e-6f * emax) ? 1 : (!(e[a2] > 1e-6f * emax) ? 2 : 3));
    g.m = 0;
    int bits;  // bits of the longest axis
    if (g.naxes == 3) {
        int s = 0;  // floor(log2(longest / shortest)): the cube is that many doublings smaller
        while (s < 15 && e[a2] * (float)(2 << s) <= emax) ++s;
        // 2 hi + 3 m <= total, and a cell number is exact in a float32
        g.m = max((total - 2 * s) / 3, 1);
        g.hi = min(s, (total - 3 * g.m) / 2);
        g.m = min(g.m, 23 - g.hi);
        bits = g.m + g.hi;
    } else {
        g.hi = min(g.naxes == 2 ? total / 2 : total, 23);
        bits = g.hi;
    }
    g.inv = emax > 0.f ? (float)((1u << bits) - 1u) / emax : 0.f;
    return g;
}

template <class K>
ALB_DEVICE K cell_key(const KeyGrid& g, const HilbertTables& t, float x, float y, float z) {
    const float v[3] = {x, y, z};
    const float top = (float)((1u << (g.m + g.hi)) - 1u);
    uint32_t c[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = g.ax[i];
        const float w = a == 0 ? v[0] - g.lo[0] : (a == 1 ? v[1] - g.lo[1] : v[2] - g.lo[2]);
        c[i] = (uint32_t)fminf(fmaxf(w * g.inv, 0.f), top);  // NaN goes to cell 0
    }
    if (g.naxes == 1) return c[0];
    if (g.naxes == 2) {
        return hilbert_key2<K>(t, c[0], c[1], g.hi);
    }
    if (g.naxes == 0) return 0u;
    const uint32_t mask = (1u << g.m) - 1u;
    const K hi = hilbert_key2<K>(t, c[0] >> g.m, c[1] >> g.m, g.hi);
    return (hi << (3 * g.m)) | hilbert_key3<K>(t, c[0] & mask, c[1] & mask, min(c[2], mask), g.m);
}

// ------------------------------------------------------------------------------------------
// LSD radix sort of (u32 or u64 key, u32 value), 8-bit digits, stable. Blocks own contiguous ranges of
// whole tiles. A pass is three launches and waits for nothing else: per block a histogram of the
// digit (the first one comes with the keys), per digit a scan over the blocks, and a scatter in
// which a block keeps one running offset per digit. A tile is ranked by warps in order, rounds in
// order and lanes in order, put in digit order in shared memory and written out from there, so
// that a digit's records leave in runs (16 on average) instead of one by one.
// Bound by latency beside its DRAM traffic, 20 B per record and pass (key read for the histogram; key
// and value read and written): a tile waits for its loads, its ranking (votes and a shared counter per
// round) and six barriers. The next tile is therefore loaded while a ranked one is written out, in the
// registers that the ranking has left, which wants the 64 of two blocks per SM: map build of the large scene
// at 1e7 photons (2.8e8 records of 48 bits) 45.2 ms with three blocks and no loads ahead, 43.9 with them in
// 42 registers, 40.0 with two blocks; 9, 10 and 12 rounds 40.7, 41.5 and 41.4, 32 warps of 8 in one block
// 41.0, 8 warps of 16 in three 44.1.
// ------------------------------------------------------------------------------------------
constexpr int kRsBlocksPerSM = 2;
constexpr int kRsWarps = 16, kRsItems = 8, kRsThreads = kRsWarps * 32;
constexpr int kRsTile = kRsThreads * kRsItems;

struct SortPlan {
    uint32_t blocks;
    uint64_t per;  // records per block, a multiple of the tile
};

static SortPlan sort_plan(uint64_t n) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t tiles = (n + kRsTile - 1) / kRsTile;
    const uint64_t each = (tiles + kRsBlocksPerSM * sms - 1) / (kRsBlocksPerSM * sms);  // resident blocks
    return SortPlan{(uint32_t)((tiles + each - 1) / each), each * kRsTile};
}

constexpr int kRsHistThreads = 1024;
template <class K>
__global__ void __launch_bounds__(kRsHistThreads) k_rs_hist(const K* __restrict__ keys, uint64_t n, int shift,
                                                         uint64_t per, uint32_t* hist) {
    __shared__ uint32_t h[256];
    if (threadIdx.x < 256) h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t r0 = blockIdx.x * per, r1 = min(r0 + per, n);
    constexpr int V = 16 / sizeof(K);  // keys of one 16-byte load; r0 is a multiple of the tile: aligned
    for (uint64_t i = r0 + V * threadIdx.x; i < r1; i += V * kRsHistThreads) {
        if (i + V <= r1) {
            K v[V];
            *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(keys + i);
#pragma unroll
            for (int j = 0; j < V; ++j) atomicAdd(&h[(uint32_t)(v[j] >> shift) & 255u], 1u);
        } else {
            for (uint64_t j = i; j < r1; ++j) atomicAdd(&h[(uint32_t)(keys[j] >> shift) & 255u], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < 256) hist[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// One block per digit: exclusive scan of its counts over the sorting blocks; total[digit].
__global__ void __launch_bounds__(256) k_rs_scan(uint32_t* hist, uint32_t blocks, uint32_t* total) {
    __shared__ uint32_t wsum[8];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t* h = hist + (uint64_t)blockIdx.x * blocks;
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < blocks; b0 += 256) {
        const uint32_t i = b0 + threadIdx.x;
        const uint32_t v = i < blocks ? h[i] : 0u;
        uint32_t inc = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (l >= o) inc += t;
        }
        if (l == 31) wsum[w] = inc;
        __syncthreads();
        uint32_t before = carry, all = 0;
        for (int j = 0; j < 8; ++j) {
            before += j < w ? wsum[j] : 0u;
            all += wsum[j];
        }
        if (i < blocks) h[i] = before + inc - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// Lanes whose d (9 bits) is this lane's, by a vote per bit (Ashkiani et al., "GPU Multisplit", PPoPP 2016).
ALB_DEVICE unsigned same_digit(uint32_t d) {
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; ++b) {
        const bool on = d >> b & 1u;
        const unsigned v = __ballot_sync(0xffffffffu, on);
        peers &= on ? v : ~v;
    }
    return peers;
}

template <class K>
struct SortSmem {
    K key[kRsTile];
    uint32_t val[kRsTile];
    uint32_t wcnt[kRsWarps][256];
    uint32_t goff[256];   // next global position of the digit
    uint32_t shift[256];  // goff of the tile less the digit's place in it
    uint32_t wsum[8];
};

// FIRST: the values are the records' own numbers.
template <class K, bool FIRST>
__global__ void __launch_bounds__(kRsThreads, kRsBlocksPerSM) k_rs_scatter(const K* __restrict__ kin,
                                                               const uint32_t* __restrict__ vin,
                                                               K* __restrict__ kout, uint32_t* __restrict__ vout,
                                                               uint64_t n, int shift, uint64_t per,
                                                               const uint32_t* __restrict__ offs,
                                                               const uint32_t* __restrict__ total) {
    extern __shared__ __align__(16) unsigned char smraw[];
    SortSmem<K>& s = *reinterpret_cast<SortSmem<K>*>(smraw);
    const int t = threadIdx.x, w = t >> 5, l = t & 31;
    const unsigned lt = lanemask_lt();
    // exclusive scan of one value per thread of the first 256 threads
    auto scan256 = [&](uint32_t v) {
        uint32_t inc = v;
        if (t < 256) {
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
                if (l >= o) inc += u;
            }
            if (l == 31) s.wsum[w] = inc;
        }
        __syncthreads();
        uint32_t before = 0;
        if (t < 256)
            for (int j = 0; j < w; ++j) before += s.wsum[j];
        __syncthreads();
        return before + inc - v;
    };
    {
        const uint32_t base = scan256(t < 256 ? total[t] : 0u);
        if (t < 256) s.goff[t] = base + offs[(uint64_t)t * gridDim.x + blockIdx.x];
    }
    const uint64_t r0 = blockIdx.x * per, r1 = min(r0 + per, n);
    const uint32_t w0 = w * (kRsItems * 32) + l;
    K key[kRsItems];
    uint32_t val[kRsItems], rank[kRsItems];
    auto load = [&](uint64_t t0) {
#pragma unroll
        for (int j = 0; j < kRsItems; ++j) {
            const uint64_t i = t0 + w0 + j * 32;
            key[j] = i < r1 ? kin[i] : (K)0;
            if (!FIRST) val[j] = i < r1 ? vin[i] : 0u;
        }
    };
    load(r0);
    for (uint64_t t0 = r0; t0 < r1; t0 += kRsTile) {
        const uint32_t have = (uint32_t)min((uint64_t)kRsTile, r1 - t0);
        for (int i = t; i < kRsWarps * 256; i += kRsThreads) (&s.wcnt[0][0])[i] = 0u;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kRsItems; ++j) {
            const uint32_t i = w0 + j * 32;
            const bool valid = i < have;
            const uint32_t d = valid ? (uint32_t)(key[j] >> shift) & 255u : 256u;  // lanes past the end match one another
            const unsigned peers = same_digit(d);
            const uint32_t cur = valid ? s.wcnt[w][d] : 0u;
            __syncwarp();
            rank[j] = cur + __popc(peers & lt);
            if (valid && l == __ffs(peers) - 1) s.wcnt[w][d] = cur + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        uint32_t cnt = 0;
        if (t < 256) {
#pragma unroll
            for (int ww = 0; ww < kRsWarps; ++ww) {
                const uint32_t c = s.wcnt[ww][t];
                s.wcnt[ww][t] = cnt;
                cnt += c;
            }
        }
        const uint32_t place = scan256(cnt);
        if (t < 256) {
#pragma unroll
            for (int ww = 0; ww < kRsWarps; ++ww) s.wcnt[ww][t] += place;
            s.shift[t] = s.goff[t] - place;
            s.goff[t] += cnt;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kRsItems; ++j) {
            const uint32_t i = w0 + j * 32;
            if (i < have) {
                const uint32_t at = s.wcnt[w][(uint32_t)(key[j] >> shift) & 255u] + rank[j];
                s.key[at] = key[j];
                s.val[at] = FIRST ? (uint32_t)(t0 + i) : val[j];
            }
        }
        __syncthreads();
        load(t0 + kRsTile);  // the next tile comes in while this one is written out
#pragma unroll 4
        for (uint32_t i = t; i < have; i += kRsThreads) {
            const K k = s.key[i];
            const uint32_t dst = s.shift[(uint32_t)(k >> shift) & 255u] + i;
            kout[dst] = k;
            vout[dst] = s.val[i];
        }
        __syncthreads();
    }
}

// Keys of positions and their first digit's histogram, by sorting block.
template <class K>
__global__ void __launch_bounds__(kRsThreads) k_keys(const float4* __restrict__ a, uint64_t stride, uint64_t n,
                                                      uint64_t per, const unsigned* __restrict__ box, int total,
                                                      K* keys, uint32_t* hist) {
    __shared__ uint32_t h[256];
    __shared__ HilbertTables tables;
    if (threadIdx.x < 256) h[threadIdx.x] = 0;
    for (uint32_t i = threadIdx.x; i < 24 * 64; i += kRsThreads) tables.t3[i] = kHilbertTables.t3[i];
    for (uint32_t i = threadIdx.x; i < 8 * 64; i += kRsThreads) tables.t2[i] = kHilbertTables.t2[i];
    __syncthreads();
    const KeyGrid g = make_key_grid(box, total);
    const uint64_t r0 = blockIdx.x * per, r1 = min(r0 + per, n);
    for (uint64_t i0 = r0 + threadIdx.x; i0 < r1; i0 += 4 * kRsThreads) {
        float4 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)  // loads in flight before the first use
            if (i0 + j * kRsThreads < r1) p[j] = a[(i0 + j * kRsThreads) * stride];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i0 + j * kRsThreads < r1) {
                const K key = cell_key<K>(g, tables, p[j].x, p[j].y, p[j].z);
                keys[i0 + j * kRsThreads] = key;
                atomicAdd(&h[(uint32_t)key & 255u], 1u);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 256) hist[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// Record numbers of the positions a[0], a[stride], ... in Hilbert order of `bits`-bit keys into
// order[n]. k0, k1, other: scratch of n words, 16-byte aligned; returns the buffer that holds the
// sorted keys, or nullptr when a temporary could not be allocated (nothing is launched then).
template <class K>
static K* hilbert_sort(Workspace& ws, const float4* a, uint64_t stride, uint64_t n, const unsigned* box, int bits,
                       uint32_t* order, K* k0, K* k1, uint32_t* other, cudaStream_t st) {
    const SortPlan p = sort_plan(n);
    uint32_t* hist = ws.take_u32((uint64_t)p.blocks * 256 + 256);
    if (!hist) return nullptr;
    uint32_t* total = hist + (uint64_t)p.blocks * 256;
    static std::atomic<bool> attr_set[64];  // batched runs sort from several host threads
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        cudaFuncSetAttribute((k_rs_scatter<K, true>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortSmem<K>));
        cudaFuncSetAttribute((k_rs_scatter<K, false>), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortSmem<K>));
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    const int passes = bits / 8;
    // the passes alternate between the value buffers: the last one writes `order`
    uint32_t* vin = nullptr;
    uint32_t* vout = passes % 2 ? order : other;
    for (int i = 0; i < passes; ++i) {
        if (i == 0) k_keys<K><<<p.blocks, kRsThreads, 0, st>>>(a, stride, n, p.per, box, bits, k0, hist);
        else k_rs_hist<K><<<p.blocks, kRsHistThreads, 0, st>>>(k0, n, 8 * i, p.per, hist);
        k_rs_scan<<<256, 256, 0, st>>>(hist, p.blocks, total);
        if (i == 0)
            k_rs_scatter<K, true><<<p.blocks, kRsThreads, sizeof(SortSmem<K>), st>>>(k0, vin, k1, vout, n, 0, p.per, hist, total);
        else
            k_rs_scatter<K, false><<<p.blocks, kRsThreads, sizeof(SortSmem<K>), st>>>(k0, vin, k1, vout, n, 8 * i, p.per, hist, total);
        for (int j = 0; j < 3; ++j) note_launch();
        std::swap(k0, k1);
        vin = vout;
        vout = vin == order ? other : order;
    }
    return k0;
}

// ------------------------------------------------------------------------------------------
// k-d order: a left-balanced median-split k-d tree over 32-record leaves. A node holding
// c leaves gives its left child the largest power of two below c, so every aligned run of
// 32^j leaves is one k-d subtree and the implicit 32-ary box tree inherits k-d cells
// (tight, non-overlapping boxes) instead of Morton runs that straddle far-apart cells.
// Every split cuts the node's widest box axis at the 16-bit quantised coordinate that
// leaves exactly the left child's record count on its side.
// ------------------------------------------------------------------------------------------

ALB_DEVICE void kd_node(uint64_t leaf, uint64_t L, int depth, uint64_t& a, uint64_t& c) {
    a = 0;
    c = L;
    for (int i = 0; i < depth && c > 1; ++i) {
        uint64_t left = 1ull << (63 - __clzll((long long)(c - 1)));
        if (leaf - a < left) {
            c = left;
        } else {
            a += left;
            c -= left;
        }
    }
}

constexpr int kCellMax = 4096;  // records of one node ordered by one CTA in shared memory
constexpr int kCellThreads = 512;
constexpr uint32_t kDummy = 0xffffffffu;

static size_t cell_smem_bytes() {
    return (size_t)kCellMax * 8 + (size_t)kCellMax * 16 + (size_t)2 * 3 * (kCellMax / 32) * 4;
}

struct CellSmem {
    unsigned long long* key;  // kCellMax sort keys
    float *X, *Y, *Z;         // kCellMax coordinates
    uint32_t* ID;             // kCellMax record ids
    unsigned *blo, *bhi;      // 3 * (kCellMax / 32) ordered-int node boxes
};

ALB_DEVICE CellSmem cell_smem(unsigned char* raw) {
    CellSmem s;
    s.key = (unsigned long long*)raw;
    s.X = (float*)(s.key + kCellMax);
    s.Y = s.X + kCellMax;
    s.Z = s.Y + kCellMax;
    s.ID = (uint32_t*)(s.Z + kCellMax);
    s.blo = (unsigned*)(s.ID + kCellMax);
    s.bhi = s.blo + 3 * (kCellMax / 32);
    return s;
}

// Exact left-balanced k-d order of one node's records held in shared memory: entries
// [0, cnt) are records, [cnt, P) (P = cnt rounded up to 32) dummies with NaN positions.
// Reorders X/Y/Z/ID in place, level by level: node boxes -> key (node, 16-bit coordinate
// on the node's widest axis, slot) -> bitonic sort -> permute. Dummies sort last inside
// their node, so they stay in the last leaf. Called by every thread of the CTA.
ALB_DEVICE void cell_kd_sort(const CellSmem& s, unsigned cnt) {
    const unsigned P = (cnt + 31u) & ~31u;
    const unsigned Lc = P / 32;
    unsigned P2 = 32;
    while (P2 < P) P2 <<= 1;
    int depth = 0;
    while ((1u << depth) < Lc) ++depth;
    // In a full cell of a power-of-two leaf count every node of level d is an aligned block
    // of P >> d keys: sorting the blocks separately gives the same order as the full sort.
    const bool perfect = cnt == P && (Lc & (Lc - 1)) == 0;
    for (int d = 0; d < depth; ++d) {
        const unsigned S = perfect ? (P >> d) : P2;
        for (unsigned i = threadIdx.x; i < 3 * Lc; i += blockDim.x) {
            s.blo[i] = 0xffffffffu;
            s.bhi[i] = 0u;
        }
        __syncthreads();
        for (unsigned j = threadIdx.x; j < cnt; j += blockDim.x) {
            uint64_t na, nc;
            kd_node(j / 32, Lc, d, na, nc);
            if (nc > 1) {
                atomicMin(s.blo + 3 * na, f2ord(s.X[j])); atomicMax(s.bhi + 3 * na, f2ord(s.X[j]));
                atomicMin(s.blo + 3 * na + 1, f2ord(s.Y[j])); atomicMax(s.bhi + 3 * na + 1, f2ord(s.Y[j]));
                atomicMin(s.blo + 3 * na + 2, f2ord(s.Z[j])); atomicMax(s.bhi + 3 * na + 2, f2ord(s.Z[j]));
            }
        }
        __syncthreads();
        for (unsigned j = threadIdx.x; j < P2; j += blockDim.x) {
            unsigned long long k = ~0ull;
            if (j < P) {
                uint64_t na, nc;
                kd_node(j / 32, Lc, d, na, nc);
                uint64_t q = 0;
                if (j >= cnt) {
                    q = 0x1ffff;
                } else if (nc > 1) {
                    const unsigned* lo = s.blo + 3 * na;
                    const unsigned* hi = s.bhi + 3 * na;
                    float l0 = ord2f(lo[0]), l1 = ord2f(lo[1]), l2 = ord2f(lo[2]);
                    float e0 = ord2f(hi[0]) - l0, e1 = ord2f(hi[1]) - l1, e2 = ord2f(hi[2]) - l2;
                    float v, l, e;
                    if (e0 >= e1 && e0 >= e2) { v = s.X[j]; l = l0; e = e0; }
                    else if (e1 >= e2) { v = s.Y[j]; l = l1; e = e1; }
                    else { v = s.Z[j]; l = l2; e = e2; }
                    if (e > 0.f) q = (uint64_t)fminf(fmaxf((v - l) / e * 65535.f, 0.f), 65535.f);
                }
                k = (((na << 17) | q) << 13) | j;  // j < 8192 keeps equal keys in place
            }
            s.key[j] = k;
        }
        __syncthreads();
        // bitonic sort of every aligned block of S keys, ascending (the last merge of a block
        // runs ascending everywhere)
        for (unsigned kk = 2; kk <= S; kk <<= 1) {
            for (unsigned jj = kk >> 1; jj > 0; jj >>= 1) {
                for (unsigned i = threadIdx.x; i < P2; i += blockDim.x) {
                    unsigned p = i ^ jj;
                    if (p > i) {
                        unsigned long long x = s.key[i], y = s.key[p];
                        bool up = kk == S || (i & kk) == 0;
                        if ((x > y) == up) {
                            s.key[i] = y;
                            s.key[p] = x;
                        }
                    }
                }
                __syncthreads();
            }
        }
        constexpr int R = kCellMax / kCellThreads;  // each thread stages its slots in registers
        float rx[R], ry[R], rz[R];
        uint32_t rid[R];
#pragma unroll
        for (int t = 0; t < R; ++t) {
            unsigned j = threadIdx.x + t * kCellThreads;
            if (j < P) {
                unsigned src = (unsigned)(s.key[j] & 0x1fffull);
                rx[t] = s.X[src]; ry[t] = s.Y[src]; rz[t] = s.Z[src]; rid[t] = s.ID[src];
            }
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < R; ++t) {
            unsigned j = threadIdx.x + t * kCellThreads;
            if (j < P) {
                s.X[j] = rx[t]; s.Y[j] = ry[t]; s.Z[j] = rz[t]; s.ID[j] = rid[t];
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// Exact left-balanced k-d order by streaming partitions (the photon-map build).
// Global levels 0..D-1 (nodes larger than one CTA's cell) each take these passes over
// X = float4(x, y, z, record id) in position order (and Q, each record's 16-bit coordinate):
//   hist1: per node, 256-bin histogram of the top byte of a 16-bit coordinate quantised
//          on the node's widest axis (level 0 from X; every later level gets it from the
//          split above, which also writes the coordinates to Q);
//   hist2: per node, 256-bin histogram of the low byte inside the bucket that holds the
//          cut (the node's left child takes exactly its power-of-two leaf count), from Q;
//   split: every record goes left or right of that cut (ties at the 16-bit cut resolved
//          by an atomic ticket), with warp-aggregated cursors, into X2, its coordinate on
//          its child's axis into Q, and the children's first histogram on the way.
// The remaining levels (nodes of <= kCellMax records) run in one CTA per node in shared
// memory (k_local_kd_full for perfect cells, k_local_kd for the rest). The cut is placed at
// 16-bit resolution.
// ------------------------------------------------------------------------------------------

// (start leaf a, leaf count c, path bits) of the depth-d node holding `leaf`
ALB_DEVICE void kd_node_path(uint64_t leaf, uint64_t L, int depth, uint64_t& a, uint64_t& c, uint32_t& path,
                             int& reached) {
    a = 0;
    c = L;
    path = 0;
    reached = 0;
    while (reached < depth && c > 1) {
        if ((c & (c - 1)) == 0) {
            // a perfect subtree of c = 2^e leaves: the remaining path is the leading bits of
            // the leaf's offset in it
            const int e = 63 - __clzll((long long)c);
            const int take = min(depth - reached, e);
            const uint64_t top = (leaf - a) >> (e - take);
            path = (path << take) | (uint32_t)top;
            a += top << (e - take);
            c = 1ull << (e - take);
            reached += take;
            return;
        }
        uint64_t left = 1ull << (63 - __clzll((long long)(c - 1)));
        if (leaf - a < left) {
            c = left;
            path = path << 1;
        } else {
            a += left;
            c -= left;
            path = (path << 1) | 1u;
        }
        ++reached;
    }
}

// node of the depth-d path: start leaf a and leaf count c (c == 0 if the path ends early)
ALB_DEVICE void kd_node_of_path(uint32_t path, uint64_t L, int depth, uint64_t& a, uint64_t& c) {
    a = 0;
    c = L;
    for (int i = depth - 1; i >= 0; --i) {
        if (c <= 1) {
            c = 0;
            return;
        }
        uint64_t left = 1ull << (63 - __clzll((long long)(c - 1)));
        if ((path >> i) & 1u) {
            a += left;
            c -= left;
        } else {
            c = left;
        }
    }
}

// Per node of a level: the widest box axis (x = axis bits, -1 for an empty extent), its low
// end and 65535 / extent, so that a record's 16-bit coordinate is one multiply.
struct LevelNodes {
    const float4* par;
};

__global__ void k_kdl_params(const unsigned* __restrict__ lo, const unsigned* __restrict__ hi, uint32_t nodes,
                             float4* par) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nodes) return;
    const float l0 = ord2f(lo[3 * i]), l1 = ord2f(lo[3 * i + 1]), l2 = ord2f(lo[3 * i + 2]);
    const float e0 = ord2f(hi[3 * i]) - l0, e1 = ord2f(hi[3 * i + 1]) - l1, e2 = ord2f(hi[3 * i + 2]) - l2;
    int axis;
    float l, e;
    if (e0 >= e1 && e0 >= e2) { axis = 0; l = l0; e = e0; }
    else if (e1 >= e2) { axis = 1; l = l1; e = e1; }
    else { axis = 2; l = l2; e = e2; }
    if (!(e > 0.f)) axis = -1;
    par[i] = make_float4(__int_as_float(axis), l, axis >= 0 ? 65535.f / e : 0.f, 0.f);
}

ALB_DEVICE uint32_t kd_quant16(float4 p, LevelNodes nb, uint32_t path) {
    const float4 np = nb.par[path];
    const int axis = __float_as_int(np.x);
    if (axis < 0) return 0u;
    const float v = axis == 0 ? p.x : (axis == 1 ? p.y : p.z);
    return (uint32_t)fminf(fmaxf((v - np.y) * np.z, 0.f), 65535.f);
}

// warp-aggregated atomicAdd of 1 on cnt[key]; returns this lane's ticket
ALB_DEVICE unsigned agg_inc(unsigned* cnt, uint64_t key, unsigned active) {
    unsigned peers = __match_any_sync(active, key);
    int leader = __ffs(peers) - 1;
    unsigned rank = __popc(peers & lanemask_lt());
    unsigned base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(cnt, (unsigned)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + rank;
}

// Level passes run persistent blocks over contiguous record ranges (records of a node are
// contiguous, so a block meets few nodes at the upper levels, where global atomics would
// collide): per-node counters live in kSlots tagged shared-memory slots, records of nodes
// that find no slot go to global memory directly.
constexpr int kLvlThreads = 256;
constexpr int kSlots = 8;
constexpr int kHistItems = 4;
constexpr unsigned kNoTag = 0xffffffffu;

// claim the slot of `key` (path or child id); returns the slot or -1
ALB_DEVICE int slot_of(unsigned* tag, unsigned key) {
    const int sl = (int)(key & (kSlots - 1));
    unsigned t = tag[sl];
    if (t == kNoTag) {
        const unsigned old = atomicCAS(&tag[sl], kNoTag, key);
        t = (old == kNoTag) ? key : old;
    }
    return t == key ? sl : -1;
}

// Level 0's first pass: per node, 256-bin histogram of the top byte of the 16-bit
// coordinate, which goes to Q (later levels get both from the split of the level above).
__global__ void __launch_bounds__(kLvlThreads) k_kdl_hist1(const float4* __restrict__ X, uint16_t* Q, uint64_t n,
                                                           uint64_t L, int d, LevelNodes nb, unsigned* hist,
                                                           uint64_t per) {
    __shared__ unsigned tag[kSlots];
    __shared__ unsigned sh[kSlots * 256];
    for (int j = threadIdx.x; j < kSlots * 256; j += blockDim.x) sh[j] = 0u;
    if (threadIdx.x < kSlots) tag[threadIdx.x] = kNoTag;
    __syncthreads();
    const uint64_t r0 = blockIdx.x * per, r1 = min(r0 + per, n);
    // kHistItems records per thread and iteration, all loads issued before any is used:
    // the pass streams the records once, so loads in flight set its speed
    const uint64_t stride = (uint64_t)blockDim.x * kHistItems;
    for (uint64_t base0 = r0 + (threadIdx.x & ~31u); base0 < r1; base0 += stride) {
        float4 pv[kHistItems];
#pragma unroll
        for (int t = 0; t < kHistItems; ++t) {
            const uint64_t i = base0 + (uint64_t)t * blockDim.x + lane_id();
            if (i < r1) pv[t] = X[i];
        }
#pragma unroll
        for (int t = 0; t < kHistItems; ++t) {
            const uint64_t base = base0 + (uint64_t)t * blockDim.x;
            const uint64_t i = base + lane_id();
            bool act = false;
            uint32_t path = 0, h = 0;
            if (i < r1) {
                uint64_t a, c;
                int r;
                kd_node_path(i / 32, L, d, a, c, path, r);
                if (r == d && c > 1) {
                    const uint32_t q = kd_quant16(pv[t], nb, path);
                    Q[i] = (uint16_t)q;
                    act = true;
                    h = q >> 8;
                }
            }
            const unsigned am = __ballot_sync(0xffffffffu, act);
            if (am) {
                // a warp covers one 32-record leaf, so its records share one node: one slot
                // lookup per warp, then plain shared-memory atomics per record
                const int lead = __ffs(am) - 1;
                const uint32_t p0 = __shfl_sync(0xffffffffu, path, lead);
                if (__all_sync(0xffffffffu, !act || path == p0)) {
                    int sl = 0;
                    if ((int)lane_id() == lead) sl = slot_of(tag, p0);
                    sl = __shfl_sync(0xffffffffu, sl, lead);
                    if (act) {
                        if (sl >= 0) atomicAdd(&sh[sl * 256 + h], 1u);
                        else atomicAdd(hist + (uint64_t)path * 256 + h, 1u);
                    }
                } else if (act) {
                    const unsigned key = (path << 8) | h;
                    const unsigned peers = __match_any_sync(am, key);
                    if ((int)lane_id() == __ffs(peers) - 1) {
                        const int sl = slot_of(tag, path);
                        if (sl >= 0) atomicAdd(&sh[sl * 256 + h], (unsigned)__popc(peers));
                        else atomicAdd(hist + (uint64_t)path * 256 + h, (unsigned)__popc(peers));
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < kSlots * 256; j += blockDim.x) {
        const unsigned t = tag[j >> 8];
        if (t != kNoTag && sh[j]) atomicAdd(hist + (uint64_t)t * 256 + (j & 255), sh[j]);
    }
}

// PASS 2 from the coordinate stream: per node, 256-bin histogram of the low byte of the
// 16-bit coordinates inside the bucket that holds the cut. Each thread takes 8 consecutive
// records (one 16-byte load of Q), which lie in one 32-record leaf and so in one node: one
// node lookup and one slot claim per 8 records.
__global__ void __launch_bounds__(kLvlThreads) k_kdl_hist2q(const uint16_t* __restrict__ Q, uint64_t n, uint64_t L,
                                                            int d, const uint2* __restrict__ sel, unsigned* hist,
                                                            uint64_t per) {
    __shared__ unsigned tag[kSlots];
    __shared__ unsigned sh[kSlots * 256];
    for (int j = threadIdx.x; j < kSlots * 256; j += blockDim.x) sh[j] = 0u;
    if (threadIdx.x < kSlots) tag[threadIdx.x] = kNoTag;
    __syncthreads();
    const uint64_t r0 = blockIdx.x * per, r1 = min(r0 + per, n);  // per is a multiple of 1024
    for (uint64_t i0 = r0 + (uint64_t)threadIdx.x * 8; i0 < r1; i0 += (uint64_t)blockDim.x * 8) {
        uint32_t q[8];
        if (i0 + 8 <= r1) {
            const uint4 v = *reinterpret_cast<const uint4*>(Q + i0);  // i0 % 8 == 0: 16-byte aligned
            q[0] = v.x & 0xffffu; q[1] = v.x >> 16; q[2] = v.y & 0xffffu; q[3] = v.y >> 16;
            q[4] = v.z & 0xffffu; q[5] = v.z >> 16; q[6] = v.w & 0xffffu; q[7] = v.w >> 16;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) q[e] = i0 + e < r1 ? (uint32_t)Q[i0 + e] : 0u;
        }
        uint64_t a, c;
        uint32_t path;
        int r;
        kd_node_path(i0 / 32, L, d, a, c, path, r);
        if (r != d || c <= 1) continue;  // no split of this node at this level
        const unsigned bucket = sel[path].x;
        const int sl = slot_of(tag, path);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (i0 + e < r1 && (q[e] >> 8) == bucket) {
                if (sl >= 0) atomicAdd(&sh[sl * 256 + (q[e] & 255u)], 1u);
                else atomicAdd(hist + (uint64_t)path * 256 + (q[e] & 255u), 1u);
            }
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < kSlots * 256; j += blockDim.x) {
        const unsigned t = tag[j >> 8];
        if (t != kNoTag && sh[j]) atomicAdd(hist + (uint64_t)t * 256 + (j & 255), sh[j]);
    }
}

// one warp per node: locate the bucket of the cut; sel[node] = {bucket, need inside it}
__global__ void k_kdl_select1(const unsigned* __restrict__ hist1, uint64_t L, int d, uint32_t nodes, uint2* sel) {
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int l = lane_id();
    if (w >= nodes) return;
    uint64_t a, c;
    kd_node_of_path(w, L, d, a, c);
    if (c <= 1) {
        if (l == 0) sel[w] = make_uint2(0xffffffffu, 0u);
        return;
    }
    uint64_t left = 1ull << (63 - __clzll((long long)(c - 1)));
    unsigned need = (unsigned)(left * 32);
    const unsigned* h = hist1 + (uint64_t)w * 256;
    unsigned v[8], run = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[j] = h[l * 8 + j];
        run += v[j];
    }
    unsigned incl = run;
    for (int o = 1; o < 32; o <<= 1) {
        unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (l >= o) incl += t;
    }
    unsigned before = incl - run;
    int bucket = -1;
    unsigned below = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (bucket < 0 && before < need && before + v[j] >= need) {
            bucket = l * 8 + j;
            below = before;
        }
        before += v[j];
    }
    // the node holds need + (right child's records) > need records, so one lane finds it
    unsigned who = __ballot_sync(0xffffffffu, bucket >= 0);
    int src = who ? __ffs(who) - 1 : 0;
    bucket = __shfl_sync(0xffffffffu, bucket, src);
    below = __shfl_sync(0xffffffffu, below, src);
    if (l == 0) sel[w] = make_uint2((unsigned)bucket, need - below);
}

// one warp per node: the 16-bit cut value and how many records AT it go left
__global__ void k_kdl_select2(const unsigned* __restrict__ hist2, uint32_t nodes, const uint2* __restrict__ sel,
                              uint2* cut) {
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int l = lane_id();
    if (w >= nodes) return;
    uint2 s = sel[w];
    if (s.x >= 256u) {  // not an internal node of this level
        if (l == 0) cut[w] = make_uint2(0xffffffffu, 0u);
        return;
    }
    unsigned need = s.y;
    const unsigned* h = hist2 + (uint64_t)w * 256;
    unsigned v[8], run = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[j] = h[l * 8 + j];
        run += v[j];
    }
    unsigned incl = run;
    for (int o = 1; o < 32; o <<= 1) {
        unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (l >= o) incl += t;
    }
    unsigned before = incl - run;
    int sub = -1;
    unsigned below = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (sub < 0 && before < need && before + v[j] >= need) {
            sub = l * 8 + j;
            below = before;
        }
        before += v[j];
    }
    unsigned who = __ballot_sync(0xffffffffu, sub >= 0);
    int src = who ? __ffs(who) - 1 : 0;
    sub = __shfl_sync(0xffffffffu, sub, src);
    below = __shfl_sync(0xffffffffu, below, src);
    // records with q16 < cutv go left, records with q16 == cutv: the first `ties` go left
    if (l == 0) cut[w] = make_uint2((s.x << 8) | (unsigned)(sub < 0 ? 0 : sub), need - below);
}

// Every record goes left or right of its node's cut into X2. A tile of kSplitItems records
// per thread is read once; per tile, shared counters per (node slot, side) give each record
// its rank and one global atomic per (node, side) reserves the tile's range. The children's
// boxes (for the next level's axis choice) are reduced in shared memory over the block's
// whole range and flushed once.
constexpr int kSplitItems = 4;
constexpr uint32_t kNoQ = 0xffffffffu;

__global__ void __launch_bounds__(kLvlThreads, 4) k_kdl_split(const float4* __restrict__ X, float4* __restrict__ X2,
                                                           uint16_t* Q, uint64_t n, uint64_t L, int d, LevelNodes nb,
                                                           const uint2* __restrict__ cut, unsigned* cursors,
                                                           unsigned* ties, unsigned* err, uint64_t per,
                                                           LevelNodes nbn, unsigned* hist_next) {
    __shared__ unsigned ntag[kSlots];           // node slots of the current tile
    __shared__ unsigned ncnt[kSlots * 2];       // records per (slot, side) in the tile
    __shared__ unsigned nbase[kSlots * 2];      // their global start (cursor reservation)
    // next level's first histogram (top byte of the child's 16-bit coordinate), fused into
    // this pass: child slots for the block's whole range, global counters otherwise
    __shared__ unsigned htag[kSlots];
    __shared__ unsigned hsh[kSlots * 256];
    if (hist_next) {
        for (int j = threadIdx.x; j < kSlots * 256; j += blockDim.x) hsh[j] = 0u;
        if (threadIdx.x < kSlots) htag[threadIdx.x] = kNoTag;
    }
    __syncthreads();  // the slots are read by every thread, whatever the block's range holds
    const uint64_t r0 = blockIdx.x * per, r1 = min(r0 + per, n);
    const uint64_t tile = (uint64_t)kSplitItems * blockDim.x;
    // this thread's last node lookup: leaves [cn_a, cn_a + cn_c), its path, depth reached,
    // cut and parameters
    uint64_t cn_a = 0, cn_c = 0;
    uint32_t cn_path = 0;
    int cn_r = -1;
    uint2 cn_cut = make_uint2(0u, 0u);
    float4 cn_par = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint64_t t0 = r0; t0 < r1; t0 += tile) {
        if (threadIdx.x < kSlots) ntag[threadIdx.x] = kNoTag;
        if (threadIdx.x < kSlots * 2) ncnt[threadIdx.x] = 0u;
        __syncthreads();
        float4 p[kSplitItems];
        uint64_t dst0[kSplitItems];  // start of the record's child range
        uint64_t dend[kSplitItems];  // end of that range (bounds check)
        uint32_t path[kSplitItems], rank[kSplitItems];
        uint32_t qn[kSplitItems];    // the child's 16-bit coordinate, or kNoQ when not split again
        int code[kSplitItems];       // slot * 2 + side while the tile reservation is pending, else -1
#pragma unroll
        for (int t = 0; t < kSplitItems; ++t) {  // every load in flight before the first use
            const uint64_t i = t0 + (uint64_t)t * blockDim.x + threadIdx.x;
            if (i < r1) p[t] = X[i];
        }
#pragma unroll
        for (int t = 0; t < kSplitItems; ++t) {
            const uint64_t i = t0 + (uint64_t)t * blockDim.x + threadIdx.x;
            code[t] = -1;
            dst0[t] = 0;
            dend[t] = 0;
            path[t] = 0;
            rank[t] = 0;
            qn[t] = kNoQ;
            bool moves = false, counts_next = false;
            unsigned side = 0, hbin = 0;
            uint64_t a = 0, c = 0, left = 0;
            if (i < r1) {
                // the node of the previous item usually holds this one too (items are 8
                // leaves apart, split nodes at least 128 leaves wide): reuse its lookup
                const uint64_t leaf = i / 32;
                if (!(leaf >= cn_a && leaf - cn_a < cn_c)) {
                    kd_node_path(leaf, L, d, cn_a, cn_c, cn_path, cn_r);
                    if (cn_r == d && cn_c > 1) {
                        cn_cut = cut[cn_path];
                        cn_par = nb.par[cn_path];
                    }
                }
                a = cn_a;
                c = cn_c;
                path[t] = cn_path;
                if (cn_r == d && c > 1) {
                    moves = true;
                    left = 1ull << (63 - __clzll((long long)(c - 1)));
                    const uint2 ct = cn_cut;
                    const int axis = __float_as_int(cn_par.x);
                    const float v = axis == 0 ? p[t].x : (axis == 1 ? p[t].y : p[t].z);
                    const uint32_t q = axis < 0 ? 0u : (uint32_t)fminf(fmaxf((v - cn_par.y) * cn_par.z, 0.f), 65535.f);
                    if (q < ct.x) side = 0;
                    else if (q > ct.x) side = 1;
                    else side = (atomicAdd(ties + path[t], 1u) < ct.y) ? 0u : 1u;
                    dst0[t] = a * 32 + (side ? left * 32 : 0);
                    dend[t] = side ? min((a + c) * 32, n) : (a + left) * 32;
                    // the child node is split again at the next level if it has > 1 leaf
                    if (hist_next && (side ? c - left : left) > 1) {
                        counts_next = true;
                        qn[t] = kd_quant16(p[t], nbn, (path[t] << 1) | side);
                        hbin = qn[t] >> 8;
                    }
                } else {
                    X2[i] = p[t];  // already in place (a leaf of an earlier level)
                }
            }
            // per-warp aggregation of (path, side) for the tile counters
            const unsigned am = __ballot_sync(0xffffffffu, moves);
            // a warp covers one 32-record leaf, so its moving records share one node and the
            // peers of a record are the lanes on its side (match only as a fallback)
            const unsigned right = __ballot_sync(0xffffffffu, moves && side);
            const uint32_t p0 = __shfl_sync(0xffffffffu, path[t], am ? __ffs(am) - 1 : 0);
            const bool one_node = __all_sync(0xffffffffu, !moves || path[t] == p0);
            if (moves) {
                const unsigned key = (path[t] << 1) | side;
                const unsigned peers = one_node ? (side ? right : (am & ~right)) : __match_any_sync(am, key);
                const int leader = __ffs(peers) - 1;
                const unsigned lrank = __popc(peers & lanemask_lt());
                unsigned b = 0;
                int cd = -1;
                if ((int)lane_id() == leader) {
                    const int sl = slot_of(ntag, path[t]);
                    if (sl >= 0) {
                        cd = sl * 2 + (int)side;
                        b = atomicAdd(&ncnt[cd], (unsigned)__popc(peers));
                    } else {
                        b = atomicAdd(cursors + 2 * (uint64_t)path[t] + side, (unsigned)__popc(peers));
                    }
                }
                cd = __shfl_sync(peers, cd, leader);
                b = __shfl_sync(peers, b, leader);
                code[t] = cd;
                rank[t] = b + lrank;
                if (cd < 0) {  // global cursor: final position known now
                    const uint64_t dst = dst0[t] + rank[t];
                    if (dst < dend[t]) {
                        X2[dst] = p[t];
                        if (qn[t] != kNoQ) Q[dst] = (uint16_t)qn[t];
                    } else {
                        atomicOr(err, 1u);
                    }
                }
            }
            if (counts_next) {
                const unsigned child = (path[t] << 1) | side;
                const int hs = slot_of(htag, child);
                if (hs >= 0) atomicAdd(&hsh[hs * 256 + hbin], 1u);
                else atomicAdd(hist_next + (uint64_t)child * 256 + hbin, 1u);
            }
        }
        __syncthreads();
        if (threadIdx.x < kSlots * 2) {
            const unsigned tg = ntag[threadIdx.x >> 1];
            const unsigned cntv = ncnt[threadIdx.x];
            nbase[threadIdx.x] = (tg != kNoTag && cntv) ? atomicAdd(cursors + 2 * (uint64_t)tg + (threadIdx.x & 1), cntv) : 0u;
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < kSplitItems; ++t) {
            if (code[t] >= 0) {
                const uint64_t dst = dst0[t] + nbase[code[t]] + rank[t];
                if (dst < dend[t]) {
                    X2[dst] = p[t];
                    if (qn[t] != kNoQ) Q[dst] = (uint16_t)qn[t];
                } else {
                    atomicOr(err, 1u);
                }
            }
        }
        __syncthreads();
    }
    if (hist_next) {
        for (int j = threadIdx.x; j < kSlots * 256; j += blockDim.x) {
            const unsigned tg = htag[j >> 8];
            if (tg != kNoTag && hsh[j]) atomicAdd(hist_next + (uint64_t)tg * 256 + (j & 255), hsh[j]);
        }
    }
}

// Children's boxes of a level: the parent's box cut on its split axis at the cut value,
// left [lo, lo + (cut + 1) / scale], right [lo + cut / scale, hi] (they overlap by one
// quantisation step). Only the next level's axis and quantisation come from these boxes;
// any box that holds the records gives the same exact median split, and the gather's box
// tree is built from the final leaves.
__global__ void k_kdl_child_boxes(const unsigned* __restrict__ lo, const unsigned* __restrict__ hi,
                                  const float4* __restrict__ par, const uint2* __restrict__ cut, uint32_t nodes,
                                  unsigned* clo, unsigned* chi) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nodes) return;
    unsigned l[3], h[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        l[k] = lo[3 * i + k];
        h[k] = hi[3 * i + k];
    }
    unsigned ll[3] = {l[0], l[1], l[2]}, lh[3] = {h[0], h[1], h[2]};
    unsigned rl[3] = {l[0], l[1], l[2]}, rh[3] = {h[0], h[1], h[2]};
    const float4 np = par[i];
    const int axis = __float_as_int(np.x);
    if (axis >= 0 && axis < 3 && np.z > 0.f) {
        const float q = (float)cut[i].x;
        const unsigned split_hi = f2ord(np.y + (q + 1.f) / np.z);
        const unsigned split_lo = f2ord(np.y + q / np.z);
        lh[axis] = min(h[axis], max(l[axis], split_hi));
        rl[axis] = max(l[axis], min(h[axis], split_lo));
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        clo[3 * (2 * (uint64_t)i) + k] = ll[k];
        chi[3 * (2 * (uint64_t)i) + k] = lh[k];
        clo[3 * (2 * (uint64_t)i + 1) + k] = rl[k];
        chi[3 * (2 * (uint64_t)i + 1) + k] = rh[k];
    }
}

// One node of <= kCellMax records X[start + j] (id in .w) per CTA, reordered in place into
// its exact left-balanced k-d order (the CTA holds the whole node in shared memory).
__global__ void __launch_bounds__(kCellThreads) k_local_kd(float4* X, const unsigned* __restrict__ cstart,
                                                           const unsigned* __restrict__ ccount, unsigned* err) {
    extern __shared__ unsigned char smraw[];
    const CellSmem s = cell_smem(smraw);
    const unsigned cnt = ccount[blockIdx.x];
    const unsigned s0 = cstart[blockIdx.x];
    if (cnt == 0) return;
    if (cnt > (unsigned)kCellMax) {
        if (threadIdx.x == 0) atomicOr(err, 2u);
        return;
    }
    const unsigned P = (cnt + 31u) & ~31u;
    const float qnan = __int_as_float(0x7fc00000);
    for (unsigned j = threadIdx.x; j < P; j += blockDim.x) {
        if (j < cnt) {
            float4 p = X[s0 + j];
            s.X[j] = p.x; s.Y[j] = p.y; s.Z[j] = p.z; s.ID[j] = __float_as_uint(p.w);
        } else {
            s.X[j] = qnan; s.Y[j] = qnan; s.Z[j] = qnan; s.ID[j] = kDummy;
        }
    }
    __syncthreads();
    cell_kd_sort(s, cnt);
    for (unsigned j = threadIdx.x; j < cnt; j += blockDim.x)
        X[s0 + j] = make_float4(s.X[j], s.Y[j], s.Z[j], __uint_as_float(s.ID[j]));
}

// Full cells (perfect subtrees of 32, 64 or 128 whole leaves: 1024, 2048 or 4096 records,
// the bulk of every large map; which size a map's cells take depends on its leaf count): the
// same k-d order as k_local_kd, with the sort keys (16-bit coordinate : 13-bit slot) held in
// registers, 8 consecutive per thread. Levels of nodes of at least kPartitionMin records are
// split by a radix partition; below it a bitonic sort runs with strides under 8 inside a
// thread, 8..128 in warp shuffles and 256 or more through shared memory; node boxes come
// from segmented warp reductions.
// levels whose nodes hold at least this many records are split by a radix partition, the
// smaller ones by a bitonic sort inside a warp
constexpr unsigned kPartitionMin = 512;

template <int CELL>
struct FullCellSmem {
    float X[CELL], Y[CELL], Z[CELL];
    uint32_t ID[CELL];
    uint32_t sk[CELL];
    unsigned blo[3 * 64], bhi[3 * 64];
};

// Bitonic compare-exchange of a thread's 8 consecutive keys at a stride JJ < 8 (partners in
// the same thread; a compile-time stride keeps the keys in registers).
template <int JJ>
ALB_DEVICE void exchange_in_thread(uint32_t (&key)[8], int t, unsigned kk, unsigned S) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        if ((e & JJ) == 0) {
            const int f = e | JJ;
            const unsigned i = (unsigned)(t * 8 + e);
            const bool up = kk == S || (i & kk) == 0;
            const uint32_t a = key[e], b = key[f];
            if ((a > b) == up) {
                key[e] = b;
                key[f] = a;
            }
        }
    }
}

// One warp: the bin of the need-th (1-based) entry of a 256-bin histogram h; need becomes the
// entry's rank inside that bin.
ALB_DEVICE unsigned pick_bin256(const uint32_t* h, unsigned& need) {
    const int lane = threadIdx.x & 31;
    uint32_t c[8], run = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        c[i] = h[lane * 8 + i];
        run += c[i];
    }
    uint32_t inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    uint32_t before = inc - run;
    int bin = -1;
    uint32_t below = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (bin < 0 && before + c[i] >= need) {
            bin = lane * 8 + i;
            below = before;
        }
        before += c[i];
    }
    const unsigned who = __ballot_sync(0xffffffffu, bin >= 0);
    const int src = __ffs(who) - 1;
    bin = __shfl_sync(0xffffffffu, bin, src);
    below = __shfl_sync(0xffffffffu, below, src);
    need -= below;
    return (unsigned)bin;
}

// Exclusive prefix of v over the threads of this thread's node (an aligned block of tpn >= 64
// threads, whole warps), in thread order. wsum: 16 words of shared scratch.
ALB_DEVICE unsigned node_exclusive_scan(unsigned v, uint32_t* wsum, unsigned tpn) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    unsigned inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    const int w0 = (int)((t / tpn) * (tpn / 32));
    unsigned before = 0;
    for (int i = w0; i < w; ++i) before += wsum[i];
    __syncthreads();  // wsum is reused by the next scan
    return before + inc - v;
}

template <int CELL>
__global__ void __launch_bounds__(CELL / 8, 8192 / CELL) k_local_kd_full(float4* Xg, const unsigned* __restrict__ cstart) {
    constexpr int kFullThreads = CELL / 8;
    constexpr int kLevels = CELL == 4096 ? 7 : (CELL == 2048 ? 6 : 5);  // log2(CELL / 32)
    extern __shared__ unsigned char smraw[];
    FullCellSmem<CELL>& s = *reinterpret_cast<FullCellSmem<CELL>*>(smraw);
    const uint64_t s0 = cstart[blockIdx.x];
    const int t = threadIdx.x;
    const int lane = t & 31;
    for (int j = t; j < CELL; j += kFullThreads) {
        const float4 p = Xg[s0 + j];
        s.X[j] = p.x;
        s.Y[j] = p.y;
        s.Z[j] = p.z;
        s.ID[j] = __float_as_uint(p.w);
    }
    for (int d = 0; d < kLevels; ++d) {
        const unsigned S = (unsigned)CELL >> d;  // records per node at this level
        for (int i = t; i < 3 * 64; i += kFullThreads) {
            s.blo[i] = 0xffffffffu;
            s.bhi[i] = 0u;
        }
        __syncthreads();
        // node boxes: this thread's 8 records, then the node's lanes
        unsigned mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int j = t * 8 + e;
            const unsigned o[3] = {f2ord(s.X[j]), f2ord(s.Y[j]), f2ord(s.Z[j])};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                mn[k] = min(mn[k], o[k]);
                mx[k] = max(mx[k], o[k]);
            }
        }
        const int G = S >= 256 ? 32 : (int)(S >> 3);  // lanes per node within a warp
        for (int o = 1; o < G; o <<= 1) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                mn[k] = min(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
                mx[k] = max(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
            }
        }
        const unsigned node = (unsigned)(t * 8) / S;
        if ((lane & (G - 1)) == 0) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                atomicMin(&s.blo[3 * node + k], mn[k]);
                atomicMax(&s.bhi[3 * node + k], mx[k]);
            }
        }
        __syncthreads();
        // keys: 16-bit coordinate on the node's widest axis, then the slot
        const float l0 = ord2f(s.blo[3 * node]), l1 = ord2f(s.blo[3 * node + 1]), l2 = ord2f(s.blo[3 * node + 2]);
        const float e0 = ord2f(s.bhi[3 * node]) - l0, e1 = ord2f(s.bhi[3 * node + 1]) - l1,
                    e2 = ord2f(s.bhi[3 * node + 2]) - l2;
        const int axis = (e0 >= e1 && e0 >= e2) ? 0 : (e1 >= e2 ? 1 : 2);
        const float lo = axis == 0 ? l0 : (axis == 1 ? l1 : l2);
        const float ext = axis == 0 ? e0 : (axis == 1 ? e1 : e2);
        const float* V = axis == 0 ? s.X : (axis == 1 ? s.Y : s.Z);
        uint32_t key[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int j = t * 8 + e;
            uint32_t q = 0;
            if (ext > 0.f) q = (uint32_t)fminf(fmaxf((V[j] - lo) / ext * 65535.f, 0.f), 65535.f);
            key[e] = (q << 13) | (uint32_t)j;
        }
        if (S >= kPartitionMin) {
            // Radix partition: the node's first half takes the S/2 records of smallest
            // (coordinate, position) key, the same set a sort of the keys puts there, in
            // position order; the second half the others. Two 256-bin histogram passes find
            // the cut coordinate; records AT the cut go left in position order until the left
            // half is full.
            const unsigned nodes = (unsigned)CELL / S, tpn = S / 8, nstart = node * S;
            uint32_t* h1 = s.sk;              // nodes x 256 (nodes <= CELL / 512)
            uint32_t* h2 = s.sk + CELL / 2;   // nodes x 256
            uint32_t* sel = s.blo;        // per node: cut, records at the cut that go left
            uint32_t* wsum = s.bhi;       // scan scratch (the boxes are consumed)
            for (int i = t; i < (int)(nodes * 256); i += kFullThreads) {
                h1[i] = 0u;
                h2[i] = 0u;
            }
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 8; ++e) atomicAdd(&h1[node * 256 + (key[e] >> 21)], 1u);
            __syncthreads();
            const int w = t >> 5;
            if (w < (int)nodes) {
                unsigned need = S / 2;
                const unsigned b = pick_bin256(h1 + w * 256, need);
                if (lane == 0) {
                    sel[2 * w] = b;
                    sel[2 * w + 1] = need;
                }
            }
            __syncthreads();
            const unsigned hb = sel[2 * node];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if ((key[e] >> 21) == hb) atomicAdd(&h2[node * 256 + ((key[e] >> 13) & 255u)], 1u);
            __syncthreads();
            if (w < (int)nodes) {
                unsigned need = sel[2 * w + 1];
                const unsigned lb = pick_bin256(h2 + w * 256, need);
                __syncwarp();
                if (lane == 0) {
                    sel[2 * w] = (sel[2 * w] << 8) | lb;
                    sel[2 * w + 1] = need;
                }
            }
            __syncthreads();
            const unsigned cut = sel[2 * node], at_left = sel[2 * node + 1];
            unsigned nt = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) nt += (key[e] >> 13) == cut ? 1u : 0u;
            unsigned tr = node_exclusive_scan(nt, wsum, tpn);  // ties before this thread's
            unsigned lmask = 0u;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const unsigned qe = key[e] >> 13;
                bool left = qe < cut;
                if (qe == cut) left = tr++ < at_left;
                lmask |= (left ? 1u : 0u) << e;
            }
            unsigned lb4 = node_exclusive_scan((unsigned)__popc(lmask), wsum, tpn);  // lefts before
            float rx[8], ry[8], rz[8];
            uint32_t rid[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int j = t * 8 + e;
                rx[e] = s.X[j];
                ry[e] = s.Y[j];
                rz[e] = s.Z[j];
                rid[e] = s.ID[j];
            }
            __syncthreads();
            const unsigned pos0 = (unsigned)(t * 8) - nstart;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const bool left = (lmask >> e) & 1u;
                const unsigned dst = left ? nstart + lb4 : nstart + S / 2 + (pos0 + (unsigned)e - lb4);
                lb4 += left ? 1u : 0u;
                s.X[dst] = rx[e];
                s.Y[dst] = ry[e];
                s.Z[dst] = rz[e];
                s.ID[dst] = rid[e];
            }
            __syncthreads();
            continue;
        }
        // bitonic sort of every node's block of S keys, ascending
        for (unsigned kk = 2; kk <= S; kk <<= 1) {
            for (unsigned jj = kk >> 1; jj > 0; jj >>= 1) {
                if (jj >= 256) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) s.sk[t * 8 + e] = key[e];
                    __syncthreads();
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const unsigned i = (unsigned)(t * 8 + e);
                        const uint32_t o = s.sk[i ^ jj];
                        const bool lower = (i & jj) == 0, up = kk == S || (i & kk) == 0;
                        key[e] = (lower == up) ? min(key[e], o) : max(key[e], o);
                    }
                    __syncthreads();
                } else if (jj >= 8) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const unsigned i = (unsigned)(t * 8 + e);
                        const uint32_t o = __shfl_xor_sync(0xffffffffu, key[e], (int)(jj >> 3));
                        const bool lower = (i & jj) == 0, up = kk == S || (i & kk) == 0;
                        key[e] = (lower == up) ? min(key[e], o) : max(key[e], o);
                    }
                } else if (jj == 4) {
                    exchange_in_thread<4>(key, t, kk, S);
                } else if (jj == 2) {
                    exchange_in_thread<2>(key, t, kk, S);
                } else {
                    exchange_in_thread<1>(key, t, kk, S);
                }
            }
        }
        // reorder the records by the sorted slots
        float rx[8], ry[8], rz[8];
        uint32_t rid[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t src = key[e] & 0x1fffu;
            rx[e] = s.X[src];
            ry[e] = s.Y[src];
            rz[e] = s.Z[src];
            rid[e] = s.ID[src];
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int j = t * 8 + e;
            s.X[j] = rx[e];
            s.Y[j] = ry[e];
            s.Z[j] = rz[e];
            s.ID[j] = rid[e];
        }
        __syncthreads();
    }
    for (int j = t; j < CELL; j += kFullThreads)
        Xg[s0 + j] = make_float4(s.X[j], s.Y[j], s.Z[j], __uint_as_float(s.ID[j]));
}

// positions of the interleaved store (stride 2) with each record's index in the w lane
__global__ void k_pack_ids(const float4* __restrict__ a, uint64_t n, float4* X) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        float4 p = a[2 * i];
        X[i] = make_float4(p.x, p.y, p.z, __uint_as_float((uint32_t)i));
    }
}

// nodes of depth D (or leaves above it): perfect cells of 128, 64 or 32 whole leaves go to
// full[0], full[1] or full[2], the rest to (st, ct)
static void enumerate_cells(uint64_t a, uint64_t c, int depth, int D, uint64_t n, std::vector<unsigned> (&full)[3],
                            std::vector<unsigned>& st, std::vector<unsigned>& ct) {
    if (depth == D || c <= 1) {
        uint64_t s = a * 32, e = std::min<uint64_t>((a + c) * 32, n);
        const int fi = c == 128 ? 0 : (c == 64 ? 1 : (c == 32 ? 2 : -1));
        if (fi >= 0 && e - s == c * 32) {
            full[fi].push_back((unsigned)s);
        } else if (e > s) {
            st.push_back((unsigned)s);
            ct.push_back((unsigned)(e - s));
        }
        return;
    }
    uint64_t left = 1ull << (63 - __builtin_clzll((unsigned long long)(c - 1)));
    enumerate_cells(a, left, depth + 1, D, n, full, st, ct);
    enumerate_cells(a + left, c - left, depth + 1, D, n, full, st, ct);
}

// out[i] <- (position, record id) of the i-th record of `a` (the interleaved record store:
// record i at a[2 i]) in exact left-balanced k-d order.
// `out` (n float4) is one of the two ping-pong buffers, so the build needs one temporary of
// the same size besides it.
static int kd_order_fast(Workspace& ws, const float4* a, uint64_t n, const float blo[3], const float bhi[3],
                         float4* out, cudaStream_t st) {
    const uint64_t L = (n + 31) / 32;
    int depth_max = L > 1 ? 64 - __builtin_clzll((unsigned long long)(L - 1)) : 0;
    const int local_levels = 7;  // kCellMax / 32 = 128 leaves = 2^7
    const int D = std::max(0, depth_max - local_levels);
    size_t mark = ws.mark();
    float4* tmp = (float4*)ws.take_bytes(n * 16);
    unsigned* err = ws.take_u32(1);
    if (!tmp || !err) {
        ws.release(mark);
        return -1;
    }
    // D partition levels swap the buffers D times: start so that the result lands in `out`
    float4* X = (D % 2 == 0) ? out : tmp;
    float4* X2 = (D % 2 == 0) ? tmp : out;
    cudaMemsetAsync(err, 0, 4, st);
    unsigned blocks = (unsigned)std::min<uint64_t>((n + 255) / 256, 16384);
    k_pack_ids<<<blocks, 256, 0, st>>>(a, n, X);
    note_launch();
    if (D > 0) {
        const uint64_t maxnodes = 1ull << D;
        unsigned* hist1 = ws.take_u32(maxnodes * 256);
        unsigned* hist2 = ws.take_u32(maxnodes * 256);
        uint2* sel = (uint2*)ws.take_bytes(maxnodes * 8);
        uint2* cut = (uint2*)ws.take_bytes(maxnodes * 8);
        unsigned* cursors = ws.take_u32(maxnodes * 2);
        unsigned* ties = ws.take_u32(maxnodes);
        unsigned* lo = ws.take_u32(maxnodes * 6);  // current level boxes
        unsigned* hi = ws.take_u32(maxnodes * 6);
        unsigned* clo = ws.take_u32(maxnodes * 6);  // children boxes
        unsigned* chi = ws.take_u32(maxnodes * 6);
        float4* par = (float4*)ws.take_bytes(maxnodes * 16);
        float4* cpar = (float4*)ws.take_bytes(maxnodes * 16);  // children's parameters
        unsigned* hist1n = ws.take_u32(maxnodes * 256);       // children's first histogram
        // each record's 16-bit coordinate on its node's axis, in position order: written by
        // the level-0 histogram and by every split for the next level, read by the second
        // histogram instead of the whole record
        uint16_t* Q = (uint16_t*)ws.take_bytes(n * 2);
        if (!hist1 || !hist2 || !sel || !cut || !cursors || !ties || !lo || !hi || !clo || !chi || !par || !cpar ||
            !hist1n || !Q) {
            ws.release(mark);
            return -1;
        }
        // level 0 box: the records' bounding box
        unsigned h6[6];
        for (int k = 0; k < 3; ++k) {
            uint32_t u;
            memcpy(&u, &blo[k], 4);
            h6[k] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
            memcpy(&u, &bhi[k], 4);
            h6[3 + k] = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        }
        unsigned init_lo[3] = {h6[0], h6[1], h6[2]}, init_hi[3] = {h6[3], h6[4], h6[5]};
        cudaMemcpyAsync(lo, init_lo, 12, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(hi, init_hi, 12, cudaMemcpyHostToDevice, st);
        // persistent level blocks over contiguous ranges (a multiple of the split tile)
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const uint64_t lvl_blocks = std::max<uint64_t>(1, std::min<uint64_t>((n + 4095) / 4096, (uint64_t)sms * 8));
        uint64_t per = (n + lvl_blocks - 1) / lvl_blocks;
        per = (per + 1023) & ~1023ull;
        const unsigned lb = (unsigned)((n + per - 1) / per);
        // level 0: its parameters and first histogram; every later level gets both from
        // the previous level (children's boxes, and the histogram fused into the split pass)
        k_kdl_params<<<1, 256, 0, st>>>(lo, hi, 1u, par);
        note_launch();
        cudaMemsetAsync(hist1, 0, 256 * 4, st);
        k_kdl_hist1<<<lb, kLvlThreads, 0, st>>>(X, Q, n, L, 0, LevelNodes{par}, hist1, per);
        note_launch();
        for (int d = 0; d < D; ++d) {
            const uint32_t nodes = 1u << d;
            const bool more = d + 1 < D;
            cudaMemsetAsync(hist2, 0, (size_t)nodes * 256 * 4, st);
            cudaMemsetAsync(cursors, 0, (size_t)nodes * 8, st);
            cudaMemsetAsync(ties, 0, (size_t)nodes * 4, st);
            LevelNodes nb{par};
            k_kdl_select1<<<(nodes * 32 + 255) / 256, 256, 0, st>>>(hist1, L, d, nodes, sel);
            note_launch();
            k_kdl_hist2q<<<lb, kLvlThreads, 0, st>>>(Q, n, L, d, sel, hist2, per);
            note_launch();
            k_kdl_select2<<<(nodes * 32 + 255) / 256, 256, 0, st>>>(hist2, nodes, sel, cut);
            note_launch();
            if (more) {
                k_kdl_child_boxes<<<(nodes + 255) / 256, 256, 0, st>>>(lo, hi, par, cut, nodes, clo, chi);
                note_launch();
                k_kdl_params<<<(2 * nodes + 255) / 256, 256, 0, st>>>(clo, chi, 2 * nodes, cpar);
                note_launch();
                cudaMemsetAsync(hist1n, 0, (size_t)nodes * 2 * 256 * 4, st);
            }
            k_kdl_split<<<lb, kLvlThreads, 0, st>>>(X, X2, Q, n, L, d, nb, cut, cursors, ties, err, per,
                                                     LevelNodes{cpar}, more ? hist1n : nullptr);
            note_launch();
            std::swap(X, X2);
            std::swap(lo, clo);
            std::swap(hi, chi);
            std::swap(par, cpar);
            std::swap(hist1, hist1n);
        }
    }
    // local levels: one CTA per remaining node
    std::vector<unsigned> fs[3], cs, cc;
    enumerate_cells(0, L, 0, D, n, fs, cs, cc);
    unsigned* dfs[3];
    for (int f = 0; f < 3; ++f) dfs[f] = ws.take_u32(fs[f].size() + 1);
    unsigned* dcs = ws.take_u32(cs.size() + 1);
    unsigned* dcc = ws.take_u32(cc.size() + 1);
    if (!dfs[0] || !dfs[1] || !dfs[2] || !dcs || !dcc) {
        ws.release(mark);
        return -1;
    }
    for (int f = 0; f < 3; ++f)
        if (!fs[f].empty()) cudaMemcpyAsync(dfs[f], fs[f].data(), fs[f].size() * 4, cudaMemcpyHostToDevice, st);
    if (!cs.empty()) {
        cudaMemcpyAsync(dcs, cs.data(), cs.size() * 4, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(dcc, cc.data(), cc.size() * 4, cudaMemcpyHostToDevice, st);
    }
    static std::atomic<bool> attr_set[64];  // batched runs build from several host threads
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev].load(std::memory_order_acquire)) {
        cudaFuncSetAttribute(k_local_kd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cell_smem_bytes());
        cudaFuncSetAttribute(k_local_kd_full<4096>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(FullCellSmem<4096>));
        cudaFuncSetAttribute(k_local_kd_full<2048>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(FullCellSmem<2048>));
        cudaFuncSetAttribute(k_local_kd_full<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(FullCellSmem<1024>));
        attr_set[dev].store(true, std::memory_order_release);
    }
    if (!fs[0].empty()) {
        k_local_kd_full<4096><<<(unsigned)fs[0].size(), 512, sizeof(FullCellSmem<4096>), st>>>(X, dfs[0]);
        note_launch();
    }
    if (!fs[1].empty()) {
        k_local_kd_full<2048><<<(unsigned)fs[1].size(), 256, sizeof(FullCellSmem<2048>), st>>>(X, dfs[1]);
        note_launch();
    }
    if (!fs[2].empty()) {
        k_local_kd_full<1024><<<(unsigned)fs[2].size(), 128, sizeof(FullCellSmem<1024>), st>>>(X, dfs[2]);
        note_launch();
    }
    if (!cs.empty()) {
        k_local_kd<<<(unsigned)cs.size(), kCellThreads, cell_smem_bytes(), st>>>(X, dcs, dcc, err);
        note_launch();
    }
    unsigned herr = 0;
    cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);  // also keeps the host vectors alive for their copies
    ws.release(mark);
    return herr ? -1 : 0;
}

// ------------------------------------------------------------------------------------------
// permutation and box tree
// ------------------------------------------------------------------------------------------

// One warp per leaf: box of 32 consecutive sorted records.
__global__ void k_leaf_boxes(const float4* __restrict__ a, uint64_t n, float4* lo, float4* hi, uint64_t nleaf) {
    uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    int l = threadIdx.x & 31;
    if (warp >= nleaf) return;
    uint64_t i = warp * 32 + l;
    float x0 = 3.4e38f, y0 = 3.4e38f, z0 = 3.4e38f, x1 = -3.4e38f, y1 = -3.4e38f, z1 = -3.4e38f;
    if (i < n) {
        float4 p = a[i];
        x0 = x1 = p.x; y0 = y1 = p.y; z0 = z1 = p.z;
    }
    for (int o = 16; o > 0; o >>= 1) {
        x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        z0 = fminf(z0, __shfl_xor_sync(0xffffffffu, z0, o));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
        z1 = fmaxf(z1, __shfl_xor_sync(0xffffffffu, z1, o));
    }
    if (l == 0) {
        lo[warp] = make_float4(x0, y0, z0, 0.f);
        hi[warp] = make_float4(x1, y1, z1, 0.f);
    }
}

// One warp per parent: union of up to 32 child boxes.
__global__ void k_parent_boxes(const float4* __restrict__ clo, const float4* __restrict__ chi, uint64_t nchild,
                               float4* plo, float4* phi, uint64_t nparent) {
    uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    int l = threadIdx.x & 31;
    if (warp >= nparent) return;
    uint64_t i = warp * 32 + l;
    float x0 = 3.4e38f, y0 = 3.4e38f, z0 = 3.4e38f, x1 = -3.4e38f, y1 = -3.4e38f, z1 = -3.4e38f;
    if (i < nchild) {
        float4 a = clo[i], b = chi[i];
        x0 = a.x; y0 = a.y; z0 = a.z; x1 = b.x; y1 = b.y; z1 = b.z;
    }
    for (int o = 16; o > 0; o >>= 1) {
        x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        z0 = fminf(z0, __shfl_xor_sync(0xffffffffu, z0, o));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
        z1 = fmaxf(z1, __shfl_xor_sync(0xffffffffu, z1, o));
    }
    if (l == 0) {
        plo[warp] = make_float4(x0, y0, z0, 0.f);
        phi[warp] = make_float4(x1, y1, z1, 0.f);
    }
}

// ------------------------------------------------------------------------------------------
// host drivers
// ------------------------------------------------------------------------------------------

// Shape and storage of the box tree over m.n records.
static int shape_box_tree(Workspace& ws, MapIndex& m) {
    uint64_t cnt = (m.n + 31) / 32;
    int lev = 0;
    uint64_t off = 0;
    while (true) {
        m.lvl_off[lev] = off;
        m.lvl_cnt[lev] = cnt;
        off += cnt;
        ++lev;
        if (cnt <= 32 || lev >= kMaxLevels) break;
        cnt = (cnt + 31) / 32;
    }
    m.nlevels = lev;
    m.nboxes = off;
    m.box_lo = (float4*)ws.alloc_persistent(m.box_lo, m.box_cap, off);
    m.box_hi = (float4*)ws.alloc_persistent(m.box_hi, m.box_cap_hi, off);
    return m.box_lo && m.box_hi ? 0 : -1;
}

static void parent_boxes(MapIndex& m, cudaStream_t st) {
    for (int l = 1; l < m.nlevels; ++l) {
        uint64_t np = m.lvl_cnt[l];
        k_parent_boxes<<<(unsigned)((np * 32 + 255) / 256), 256, 0, st>>>(
            m.box_lo + m.lvl_off[l - 1], m.box_hi + m.lvl_off[l - 1], m.lvl_cnt[l - 1],
            m.box_lo + m.lvl_off[l], m.box_hi + m.lvl_off[l], np);
        note_launch();
    }
}

// Bounding box of a[0], a[stride], ... into the workspace's scratch words from `word` on (ordered ints,
// min then max), left on the device; nullptr when the scratch could not be allocated.
static unsigned* bbox_device(Workspace& ws, const float4* a, uint64_t n, cudaStream_t st, uint64_t stride, int word = 0) {
    unsigned* box = ws.scratch_box();
    if (!box) return nullptr;
    box += word;
    cudaMemsetAsync(box, 0xff, 12, st);
    cudaMemsetAsync(box + 3, 0, 12, st);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    unsigned blocks = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)sms * 8);
    if (blocks == 0) blocks = 1;
    k_bbox<<<blocks, 256, 0, st>>>(a, stride, n, box);
    note_launch();
    return box;
}

// a[i] holds (position, record id) in index order: gather every record field into index
// order, a last (in place: each thread reads its id before overwriting the entry).
__global__ void k_finalize(float4* a, float4* __restrict__ b, float4* __restrict__ fwi, float4* __restrict__ sfi,
                           uint32_t* __restrict__ id, float4* __restrict__ sco, RecordStore rec, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = __float_as_uint(a[i].w);
        b[i] = rec.b[2 * (uint64_t)r];  // the record's two halves share one 32-byte sector
        if (fwi) {
            fwi[i] = rec.fwi[r];
            sfi[i] = rec.sfi[r];
        }
        if (id) id[i] = rec.id[r];
        if (sco) sco[i] = rec.sco[r];
        a[i] = rec.a[2 * (uint64_t)r];
    }
}

void release_map_index(MapIndex& m, cudaStream_t st) {
    for (void* p : {(void*)m.a, (void*)m.b, (void*)m.fwi, (void*)m.sfi, (void*)m.id, (void*)m.sco}) dev_free(p, st);
    m.a = m.b = m.fwi = m.sfi = m.sco = nullptr;
    m.id = nullptr;
    m.a_cap = m.b_cap = m.fwi_cap = m.sfi_cap = m.id_cap = m.sco_cap = 0;
}

// ------------------------------------------------------------------------------------------
// Hilbert order finished by warps: every 256 records that are consecutive on the curve are split
// three times at the median of their box's widest axis, so that a leaf is one of eight k-d cells
// of its warp's records. Any order gives the same neighbours (the search is exact); the order
// decides how many leaves a search opens. A ball of 1.1 k-th distances meets 18.7 leaves of an
// exact k-d order, 22.3 of the plain Hilbert order, 20.9 of this one and 20.0 with 4096 records
// per cell (large scene, 7e6 records), while the k-d order takes 36 B of traffic per record on each
// of its 17 levels. Map build of the large scene at 1e7 photons (3.8e8 records): 132 -> 59 ms, at
// 1e6: 14.9 -> 5.2 ms, of 1e5 photons in 5 m of water (6e5 records): 2.8 -> 1.05 ms; the scatter
// gathers take 222 -> 234, 21.4 -> 22.9 and 0.47 -> 0.63 ms.
// ------------------------------------------------------------------------------------------
constexpr int kFinishWarps = 4;  // 40 KB of shared memory: five blocks per SM
constexpr int kRun = 256;  // records of one warp

struct FinishSmem {
    float4 b[kRun];  // by loading slot: the record's second half, energy and number
    float e[kRun];
    uint32_t id[kRun];
    float x[kRun], y[kRun], z[kRun];  // exchange between the levels
    uint32_t slot[kRun];
};

// One 32-byte record (both halves) by a single load, half the load instructions of two 16-byte ones. The time is
// DRAM's either way, 4.8 and 4.9 ms for 1.1e8 records: records are fetched at random, 262 B of traffic each.
ALB_DEVICE void load_record(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p));
}

struct FinishOut {
    float4 *a, *b, *fwi, *sfi, *sco;  // fwi, sfi, sco nullable
    uint32_t* id;                     // nullable
    float4 *box_lo, *box_hi;
};

// Destination of this lane's records [E0, E0 + R) of a node of 32 R records: the half with the
// smaller 16-bit coordinates on the widest axis first, records of one coordinate in slot order.
template <int E0, int R>
ALB_DEVICE void split_node(const float (&x)[8], const float (&y)[8], const float (&z)[8], uint32_t (&dst)[8]) {
    constexpr unsigned kAll = 0xffffffffu;
    unsigned mn[3] = {kAll, kAll, kAll}, mx[3] = {0u, 0u, 0u};
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const unsigned o[3] = {f2ord(x[E0 + r]), f2ord(y[E0 + r]), f2ord(z[E0 + r])};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            mn[k] = min(mn[k], o[k]);
            mx[k] = max(mx[k], o[k]);
        }
    }
    float lo[3], ex[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = ord2f(__reduce_min_sync(kAll, mn[k]));
        ex[k] = ord2f(__reduce_max_sync(kAll, mx[k])) - lo[k];
    }
    const int axis = (ex[0] >= ex[1] && ex[0] >= ex[2]) ? 0 : (ex[1] >= ex[2] ? 1 : 2);
    const float l0 = axis == 0 ? lo[0] : (axis == 1 ? lo[1] : lo[2]);
    const float e0 = axis == 0 ? ex[0] : (axis == 1 ? ex[1] : ex[2]);
    const float scale = e0 > 0.f ? 65535.f / e0 : 0.f;
    int q[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float v = axis == 0 ? x[E0 + r] : (axis == 1 ? y[E0 + r] : z[E0 + r]);
        q[r] = (int)fminf(fmaxf((v - l0) * scale, 0.f), 65535.f);  // NaN: 0
    }
    // the cut: counts at interpolated coordinates, every other step at the middle
    constexpr int kHalf = 16 * R;
    int a = -1, ca = 0, b = 65535, cb = 32 * R;
#pragma unroll 1
    for (int it = 0; it < 12 && ca < kHalf && b - a > 1; ++it) {
        int m = (it & 1) ? (a + b) >> 1 : a + (int)((float)(b - a) * ((float)(kHalf - ca) / (float)(cb - ca)));
        m = min(max(m, a + 1), b - 1);
        int c = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) c += q[r] <= m ? 1 : 0;
        c = __reduce_add_sync(kAll, c);
        if (c <= kHalf) {
            a = m;
            ca = c;
        } else {
            b = m;
            cb = c;
        }
    }
    // left: coordinates up to a, and the first records in (a, b] that fill the half
    const int need = kHalf - ca;
    const unsigned lt = lanemask_lt();
    int ties = 0, lefts = 0, rights = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool tie = q[r] > a && q[r] <= b;
        const unsigned bt = __ballot_sync(kAll, tie);
        const bool left = q[r] <= a || (tie && ties + __popc(bt & lt) < need);
        ties += __popc(bt);
        const unsigned bl = __ballot_sync(kAll, left);
        dst[E0 + r] = 32u * E0 + (left ? lefts + __popc(bl & lt) : kHalf + rights + __popc(~bl & lt));
        lefts += __popc(bl);
        rights += __popc(~bl);
    }
}

__global__ void __launch_bounds__(kFinishWarps * 32, 5) k_hilbert_finish(const uint32_t* __restrict__ order, RecordStore rec,
                                                                          uint64_t n, FinishOut out) {
    __shared__ FinishSmem smem[kFinishWarps];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    FinishSmem& s = smem[w];
    const uint64_t base = ((uint64_t)blockIdx.x * kFinishWarps + w) * kRun;
    if (base >= n) return;
    const int cnt = (int)min((uint64_t)kRun, n - base);
    float x[8], y[8], z[8];
    uint32_t slot[8];
    {
        uint32_t id[8];
        float4 b[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) id[i] = i * 32 + l < cnt ? order[base + i * 32 + l] : 0u;
        // every load in flight before the first use
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
            b[i] = p;
            if (i * 32 + l < cnt) load_record(rec.a + 2 * (uint64_t)id[i], p, b[i]);
            x[i] = p.x; y[i] = p.y; z[i] = p.z;
            s.e[i * 32 + l] = p.w;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            slot[i] = i * 32 + l;
            s.b[slot[i]] = b[i];
            s.id[slot[i]] = id[i];
        }
    }
    __syncwarp();
    if (cnt == kRun) {
        uint32_t dst[8];
#pragma unroll
        for (int lev = 0; lev < 3; ++lev) {
            if (lev == 0) {
                split_node<0, 8>(x, y, z, dst);
            } else if (lev == 1) {
                split_node<0, 4>(x, y, z, dst);
                split_node<4, 4>(x, y, z, dst);
            } else {
                split_node<0, 2>(x, y, z, dst);
                split_node<2, 2>(x, y, z, dst);
                split_node<4, 2>(x, y, z, dst);
                split_node<6, 2>(x, y, z, dst);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                s.x[dst[i]] = x[i]; s.y[dst[i]] = y[i]; s.z[dst[i]] = z[i];
                s.slot[dst[i]] = slot[i];
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int j = i * 32 + l;
                x[i] = s.x[j]; y[i] = s.y[j]; z[i] = s.z[j];
                slot[i] = s.slot[j];
            }
            __syncwarp();
        }
    }
    float4 blo = make_float4(0.f, 0.f, 0.f, 0.f), bhi = blo;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint64_t at = base + i * 32 + l;
        const bool in = i * 32 + l < cnt;
        if (in) {
            out.a[at] = make_float4(x[i], y[i], z[i], s.e[slot[i]]);
            out.b[at] = s.b[slot[i]];
            const uint32_t id = s.id[slot[i]];
            if (out.fwi) {
                out.fwi[at] = rec.fwi[id];
                out.sfi[at] = rec.sfi[id];
            }
            if (out.id) out.id[at] = rec.id[id];
            if (out.sco) out.sco[at] = rec.sco[id];
        }
        // the leaf's box (a NaN coordinate does not widen it, as in k_leaf_boxes)
        const float v[3] = {x[i], y[i], z[i]};
        float lo[3], hi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = ord2f(__reduce_min_sync(0xffffffffu, in ? f2ord(fminf(v[k], 3.4e38f)) : 0xffffffffu));
            hi[k] = ord2f(__reduce_max_sync(0xffffffffu, in ? f2ord(fmaxf(v[k], -3.4e38f)) : 0u));
        }
        if (l == i) {
            blo = make_float4(lo[0], lo[1], lo[2], 0.f);
            bhi = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
    }
    if (l < (cnt + 31) / 32) {
        out.box_lo[base / 32 + l] = blo;
        out.box_hi[base / 32 + l] = bhi;
    }
}

// How many runs of kRun consecutive records share one key: their leaves lie in no useful order.
template <class K>
__global__ void k_crowded(const K* __restrict__ keys, uint64_t n, unsigned* count) {
    const uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * kRun;
    const bool same = i + kRun <= n && keys[i] == keys[i + kRun - 1];
    const unsigned b = __ballot_sync(0xffffffffu, same);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(count, (unsigned)__popc(b));
}

// Index of one channel's n records: records permuted into Hilbert order with k-d leaves
// (k_hilbert_finish), or, where more than half of the records share their key's cell with over
// 256 others (a box far larger than what its records fill), into exact left-balanced k-d order; and
// the box tree over leaves of 32. The index's own position array holds the sort's scratch, so the
// peak is the record store, the index and four bytes per record.
// The last leaf's places beyond the records hold points too far for any search to admit (3.4e38 per axis):
// a search by leaves needs no test of its record numbers.
static void pad_leaf(const MapIndex& m, cudaStream_t st) {
    const uint64_t to = (m.n + 31) / 32 * 32;
    if (to > m.n) cudaMemsetAsync(m.a + m.n, 0x7f, (to - m.n) * sizeof(float4), st);
}

static int build_word(int slot) { return 16 + 8 * slot; }  // box in six words, crowded runs in the next

int start_map_index(Workspace& ws, const RecordStore& rec, uint64_t n, MapIndex& m, int slot, cudaStream_t st) {
    m.n = n;
    m.n_real = n;
    if (n == 0) {
        m.nlevels = 0;
        return 0;
    }
    if (n >= (1ull << 32)) return -1;  // record ids are 32-bit
    if (n + 64 > m.a_cap) release_map_index(m, st);  // else every array is reused in place
    const unsigned* box = bbox_device(ws, rec.a, n, st, 2, build_word(slot));
    m.a = (float4*)ws.alloc_persistent(m.a, m.a_cap, n + 64);
    if (!box || !m.a) return -1;
    const size_t mark = ws.mark();
    uint32_t* order = ws.take_u32(n);
    uint32_t* other = ws.take_u32(n);
    unsigned* crowded = ws.scratch_box() + build_word(slot) + 6;
    cudaMemsetAsync(crowded, 0, 4, st);
    // two 16-byte aligned key buffers in the position array (n + 64 float4). Key bits: 24 tell 2^16 records
    // apart even where they fill a thousandth of their box, 32 do for 2^26 (the large scene at 1e6
    // photons); beyond that the beam's core crowds its 8 cm cells (1e7 photons: the scatter gather
    // takes 410 ms on 32 bits)
    const uint64_t pad = (n + 63) & ~63ull;
    const unsigned crowd_blocks = (unsigned)((n / kRun + 256) / 256);
    bool sorted = order && other;
    if (sorted && n <= (1ull << 26)) {
        uint32_t* k0 = reinterpret_cast<uint32_t*>(m.a);
        const uint32_t* keys = hilbert_sort<uint32_t>(ws, rec.a, 2, n, box, n <= (1ull << 16) ? 24 : 32, order, k0,
                                                      k0 + pad, other, st);
        sorted = keys != nullptr;
        if (sorted) k_crowded<uint32_t><<<crowd_blocks, 256, 0, st>>>(keys, n, crowded);
    } else if (sorted) {
        uint64_t* k0 = reinterpret_cast<uint64_t*>(m.a);
        const uint64_t* keys = hilbert_sort<uint64_t>(ws, rec.a, 2, n, box, 48, order, k0, k0 + pad, other, st);
        sorted = keys != nullptr;
        if (sorted) k_crowded<uint64_t><<<crowd_blocks, 256, 0, st>>>(keys, n, crowded);
    }
    if (sorted) {
        note_launch();
        m.b = (float4*)ws.alloc_persistent(m.b, m.b_cap, n);
        if (rec.fwi) {
            m.fwi = (float4*)ws.alloc_persistent(m.fwi, m.fwi_cap, n);
            m.sfi = (float4*)ws.alloc_persistent(m.sfi, m.sfi_cap, n);
        }
        if (rec.id) m.id = (uint32_t*)ws.alloc_persistent_u32(m.id, m.id_cap, n);
        if (rec.sco) m.sco = (float4*)ws.alloc_persistent(m.sco, m.sco_cap, n);
    }
    if (!sorted || !m.b || (rec.fwi && (!m.fwi || !m.sfi)) || (rec.id && !m.id) || (rec.sco && !m.sco) ||
        shape_box_tree(ws, m) != 0) {
        ws.release(mark);
        return -1;
    }
    const FinishOut out{m.a, m.b, rec.fwi ? m.fwi : nullptr, rec.fwi ? m.sfi : nullptr, rec.sco ? m.sco : nullptr,
                        rec.id ? m.id : nullptr, m.box_lo, m.box_hi};
    const uint64_t warps = (n + kRun - 1) / kRun;
    k_hilbert_finish<<<(unsigned)((warps + kFinishWarps - 1) / kFinishWarps), kFinishWarps * 32, 0, st>>>(order, rec, n, out);
    note_launch();
    parent_boxes(m, st);
    pad_leaf(m, st);
    ws.release(mark);
    return 0;
}

int finish_map_index(Workspace& ws, const RecordStore& rec, MapIndex& m, int slot, cudaStream_t st) {
    const uint64_t n = m.n;
    if (n == 0) return 0;
    unsigned h[7];
    if (cudaMemcpyAsync(h, ws.scratch_box() + build_word(slot), sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return -1;
    if ((uint64_t)h[6] * kRun * 2 <= n) return 0;
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = ord2f(h[k]);
        hi[k] = ord2f(h[3 + k]);
    }
    if (kd_order_fast(ws, rec.a, n, lo, hi, m.a, st) != 0) return -1;
    // one record per thread: the gathers are random, so many loads in flight matter
    const unsigned blocks = (unsigned)((n + 255) / 256);
    k_finalize<<<blocks, 256, 0, st>>>(m.a, m.b, rec.fwi ? m.fwi : nullptr, rec.fwi ? m.sfi : nullptr,
                                       rec.id ? m.id : nullptr, rec.sco ? m.sco : nullptr, rec, n);
    note_launch();
    k_leaf_boxes<<<(unsigned)((m.lvl_cnt[0] * 32 + 255) / 256), 256, 0, st>>>(m.a, n, m.box_lo, m.box_hi, m.lvl_cnt[0]);
    note_launch();
    parent_boxes(m, st);
    pad_leaf(m, st);
    return 0;
}

// Points and queries of a standalone search: records whose w lane carries the point's number, and
// float32 query positions for the sort.
__global__ void k_pack_points(const float* __restrict__ pts, uint64_t m, float4* rec) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        rec[2 * i] = make_float4(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], __uint_as_float((uint32_t)i));
        rec[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__global__ void k_pack_queries(const double* __restrict__ qs, uint64_t n, float4* qa) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        qa[i] = make_float4((float)qs[3 * i], (float)qs[3 * i + 1], (float)qs[3 * i + 2], 0.f);
}
void pack_knn_points(const float* pts, uint64_t m, float4* rec, cudaStream_t st) {
    k_pack_points<<<(unsigned)std::min<uint64_t>((m + 255) / 256, 4096), 256, 0, st>>>(pts, m, rec);
    note_launch();
}
void pack_knn_queries(const double* qs, uint64_t n, float4* qa, cudaStream_t st) {
    k_pack_queries<<<(unsigned)std::min<uint64_t>((n + 255) / 256, 4096), 256, 0, st>>>(qs, n, qa);
    note_launch();
}

// Spatial order of gather queries (search bounds, cache locality): a Hilbert curve over their
// own bounding box. Over the map's box, queries far from a compact map (surface-reflection
// queries around the laser spot) would clamp to its edge and lose their order. Up to 2^18
// queries take 24-bit keys (three radix passes; still 64 cells per query), more take 32. The
// order only steers the search bounds, never the result. Nothing here waits for the device.
int sort_queries(Workspace& ws, const float4* qa, uint64_t n, uint32_t* perm, cudaStream_t st) {
    if (n == 0) return 0;
    const unsigned* box = bbox_device(ws, qa, n, st, 1);
    if (!box) return -1;
    size_t mark = ws.mark();
    uint32_t* k0 = ws.take_u32(n);
    uint32_t* k1 = ws.take_u32(n);
    uint32_t* other = ws.take_u32(n);
    const bool ok = k0 && k1 && other &&
                    hilbert_sort<uint32_t>(ws, qa, 1, n, box, n <= (1ull << 18) ? 24 : 32, perm, k0, k1, other, st);
    ws.release(mark);
    return ok ? 0 : -1;
}

}  // namespace alb
