// Photon-map gather: exact k-nearest-neighbour density estimation at every backward event
// and time-binned waveform accumulation. GPU form of Simulation.sample_photons
// (alb_sim/core/simulation.py:132-214) with scipy KDTree.query(x, k) as the neighbour
// search (alb_sim/photon_mapping/photon_map_index.py:17).
//
// One warp per query. The warp walks the 32-ary box tree depth first, nearest child
// first (children sorted by box distance with a warp bitonic sort), keeps candidates in a
// shared-memory buffer and shrinks it to the k best with a warp radix select whenever it
// fills. Distances are float32 for the search; the threshold carries a relative margin
// of 2^-18 so that every point whose float64 distance could rank at the k-th place
// survives, and the boundary band is resolved with float64 distances exactly as the
// reference's KDTree (float64 on float32-cast map positions) orders them.
//
// Planar maps: each warp takes contiguous chunks of the spatially sorted queries; from the second
// query of a chunk on, the search starts with the largest distance from the query to the previous
// query's k neighbours (k points lie within it, so it bounds the k-th distance; never looser
// than the triangle bound r_k(prev) + |q - prev|), inflated by 2^-14 so that every point of
// the float32 boundary band is still admitted. The scatter map's queries go in runs that share
// one walk of the tree (gather_group.cuh).
#include <algorithm>
#include <atomic>
#include <cfloat>

#include "device_common.cuh"
#include "internal.h"
#include "word_cache.cuh"

namespace alb {

constexpr int kGatherWarps = 8;   // 8-warp CTAs, 4 per SM: 32 warps hide the gather's latency
constexpr int kGatherBlocksPerSM = 4;
// At most this many consecutive sorted queries are handled by one warp: each chunk's first
// search runs without a bound, longer chunks balance worse (scatter map at 1e7 photons: 32 ->
// 546 ms, 64 -> 529 ms, 128 -> 524 ms; the planar maps' gathers lose 2-3% at 128). Fewer
// queries than fill the resident warps with such chunks take shorter ones (query_chunk).
constexpr int kQueryChunk = 64;
constexpr int kQueryChunkMin = 2;
constexpr int kStack = 32 * kMaxLevels;
constexpr int kCap = 288;         // candidate buffer (k <= kCap - 32)
constexpr int kSelectAt = 192;    // shrink the buffer once it holds more than this
constexpr int kBand = 32;         // near-tie entries resolved in float64
// Admission margin of the float32 screening distance (its error is below 2^-22 relative).
constexpr float kRelMargin = 9.5367431640625e-07f;  // 2^-20

// Candidates carry an error-free double-float squared distance, stored as its float32 high
// part cd and a 16-bit fraction cl of one ulp of cd (key48 = cd bits : cl + 2^15 orders
// them to ~2^-40 relative); only entries within one key unit of the k-th are resolved in
// float64.
struct WarpSmem {
    static constexpr int kCap = alb::kCap, kSelectAt = alb::kSelectAt, kTmp = 2 * kStack;
    uint32_t stk[kStack];
    float stk_d[kStack];
    float cd[kCap];
    uint32_t ci[kCap];
    int16_t cl[kCap];
    uint32_t hist[128];  // 256 radix bins, two 16-bit counters per word
    double bd[kBand];    // near-tie band: float64 distances
    uint32_t bi[kBand];  // map positions
    uint64_t bt[kBand];  // tie keys from the record's content (or 0)
    unsigned long long st[4];  // the warp's search counters: leaves, nodes, selects, queries
    // scratch words of the boundary band (the stack is free after the search)
    ALB_DEVICE uint32_t& tmp(int i) { return i < kStack ? stk[i] : reinterpret_cast<uint32_t*>(stk_d)[i - kStack]; }
};

// Lower bound of the squared distance from the float64 query (qx + lx, ...) to a box:
// the float32 per-axis gap is shrunk by its rounding bound and by the dropped low part,
// so that pruning never discards a box the float64 search would have to open.
ALB_DEVICE float box_gap(float lo, float hi, float q, float ql) {
    float g = fmaxf(fmaxf(lo - q, q - hi), 0.f);
    return fmaxf(g * (1.f - 2.384185791015625e-07f) - fabsf(ql), 0.f);
}
ALB_DEVICE float box_dist2(float qx, float qy, float qz, float lx, float ly, float lz, float4 lo, float4 hi) {
    float dx = box_gap(lo.x, hi.x, qx, lx);
    float dy = box_gap(lo.y, hi.y, qy, ly);
    float dz = box_gap(lo.z, hi.z, qz, lz);
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz)) * (1.f - 4.76837158203125e-07f);
}

// float32 distance of a map point to the query (hi + lo split of the float64 position)
ALB_DEVICE float point_dist2(float qx, float qy, float qz, float lx, float ly, float lz, float4 p) {
    float dx = (p.x - qx) - lx;
    float dy = (p.y - qy) - ly;
    float dz = (p.z - qz) - lz;
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

ALB_DEVICE double point_dist2_f64(double qx, double qy, double qz, float4 p) {
    double dx = (double)p.x - qx, dy = (double)p.y - qy, dz = (double)p.z - qz;
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Error-free transforms (Knuth two-sum); the _rn intrinsics keep the compiler from fusing
// the operations into FMAs, which would break the error terms.
ALB_DEVICE void two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Squared distance from the query (f + l per axis) to p as hi + lo with about 2^-44
// relative error: exact per-axis differences by two-sum, squares by FMA two-product.
ALB_DEVICE void point_dist2_df(float fx, float fy, float fz, float lx, float ly, float lz, float4 p, float& hi,
                               float& lo) {
    float sx, ex, sy, ey, sz, ez;
    two_sum(p.x, -fx, sx, ex);
    two_sum(p.y, -fy, sy, ey);
    two_sum(p.z, -fz, sz, ez);
    float hx, tx, hy, ty, hz, tz;
    two_sum(sx, __fsub_rn(ex, lx), hx, tx);
    two_sum(sy, __fsub_rn(ey, ly), hy, ty);
    two_sum(sz, __fsub_rn(ez, lz), hz, tz);
    const float px = __fmul_rn(hx, hx), py = __fmul_rn(hy, hy), pz = __fmul_rn(hz, hz);
    const float qx = fmaf(2.f * hx, tx, fmaf(hx, hx, -px));
    const float qy = fmaf(2.f * hy, ty, fmaf(hy, hy, -py));
    const float qz = fmaf(2.f * hz, tz, fmaf(hz, hz, -pz));
    float s1, e1, s2, e2;
    two_sum(px, py, s1, e1);
    two_sum(s1, pz, s2, e2);
    const float t = __fadd_rn(__fadd_rn(e1, e2), __fadd_rn(__fadd_rn(qx, qy), qz));
    hi = __fadd_rn(__fadd_rn(s2, t), 0.f);  // (+0 for an exact zero)
    lo = __fsub_rn(t, __fsub_rn(hi, s2));
}

// lo in units of 2^-16 ulp(hi), clamped to 16 bits
ALB_DEVICE int16_t frac16(float hi, float lo) {
    const int e = (int)((__float_as_uint(hi) >> 23) & 255u);
    if (e == 0) return 0;
    const int sh = min(166 - e, 127);  // 2^(16 + 23 - (e - 127))
    float q = lo * __uint_as_float((uint32_t)(sh + 127) << 23);
    q = fminf(fmaxf(rintf(q), -32767.f), 32767.f);
    return (int16_t)q;
}

template <class S>
ALB_DEVICE uint64_t cand_key(const S& s, int i) {
    return ((uint64_t)__float_as_uint(s.cd[i]) << 16) | (uint32_t)((int)s.cl[i] + 32768);
}

// float32(sqrt(x)) for a double x >= 0, correctly rounded (equal to casting the float64
// square root, as double rounding is harmless for sqrt from 53 to 24 bits): a float32
// estimate corrected against the squared float midpoints, which are exact in float64.
ALB_DEVICE float sqrt_to_f32(double x) {
    if (!(x > 0.0)) return 0.f;
    float s = sqrtf(__double2float_rn(x));
    const float up = __int_as_float(__float_as_int(s) + 1);
    const float dn = __int_as_float(__float_as_int(s) - 1);
    const double mh = 0.5 * ((double)s + (double)up), ml = 0.5 * ((double)s + (double)dn);
    const double mh2 = mh * mh, ml2 = ml * ml;
    if (x > mh2 || (x == mh2 && (__float_as_int(up) & 1) == 0)) s = up;
    else if (x < ml2 || (x == ml2 && (__float_as_int(dn) & 1) == 0)) s = dn;
    return s;
}

// Tie key of a map record: its time bits (high word; times are non-negative) and a 32-bit
// mix of its direction, time and energy bits (low word).
ALB_DEVICE uint64_t record_tie_key(float4 a, float4 b) {
    uint32_t h = 0x9e3779b9u;
    const uint32_t w[4] = {__float_as_uint(b.x), __float_as_uint(b.y), __float_as_uint(b.z), __float_as_uint(a.w)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h ^= w[i] * 0x85ebca6bu;
        h = (h << 13) | (h >> 19);
        h = h * 5u + 0xe6546b64u;
    }
    h ^= h >> 16;
    h *= 0x7feb352du;
    h ^= h >> 15;
    return ((uint64_t)__float_as_uint(b.w) << 32) | h;
}

// Warp bitonic sort of 32 (key, value) pairs, ascending by key. The stages are a loop, not
// an unrolled network: the gather is bound by instruction fetch, and the rolled form keeps
// its hot code smaller (measured 12% faster for the scatter-map gather).
ALB_DEVICE void warp_sort32(float& key, uint32_t& val) {
    const int l = lane_id();
#pragma unroll 1
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll 1
        for (int j = k >> 1; j > 0; j >>= 1) {
            float ok = __shfl_xor_sync(0xffffffffu, key, j);
            uint32_t ov = __shfl_xor_sync(0xffffffffu, val, j);
            bool up = ((l & k) == 0);
            bool lower = ((l & j) == 0);
            bool take_other = lower ? (up ? ok < key : ok > key) : (up ? ok > key : ok < key);
            if (take_other) {
                key = ok;
                val = ov;
            }
        }
    }
}

// Shared radix-select step: from the 256-bin histogram in s.hist (two 16-bit counters per
// word) pick the digit holding the need-th (1-based) entry; need becomes its rank inside.
template <class S>
ALB_DEVICE uint32_t radix_pick(const S& s, int& need) {
    const int l = lane_id();
    uint32_t h[8], run = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t w = s.hist[l * 4 + j];
        h[2 * j] = w & 0xffffu;
        h[2 * j + 1] = w >> 16;
        run += h[2 * j] + h[2 * j + 1];
    }
    uint32_t incl = run;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (l >= o) incl += t;
    }
    uint32_t before = incl - run;
    int digit = -1;
    uint32_t below = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (digit < 0 && before + h[j] >= (uint32_t)need) {
            digit = l * 8 + j;
            below = before;
        }
        before += h[j];
    }
    const unsigned who = __ballot_sync(0xffffffffu, digit >= 0);
    const int src = __ffs(who) - 1;
    digit = __shfl_sync(0xffffffffu, digit, src);
    below = __shfl_sync(0xffffffffu, below, src);
    need -= (int)below;
    return (uint32_t)digit;
}

// k-th smallest (1-based) float32 part cd[off .. off + cnt) (all >= 0): warp radix select.
template <class S>
ALB_DEVICE float warp_kth32(S& s, int off, int cnt, int k) {
    const int l = lane_id();
    uint32_t prefix = 0u, pmask = 0u;
    int need = k;
#pragma unroll 1
    for (int shift = 24; shift >= 0; shift -= 8) {
#pragma unroll 1
        for (int i = l; i < 128; i += 32) s.hist[i] = 0u;
        __syncwarp();
#pragma unroll 1
        for (int i = l; i < cnt; i += 32) {
            const uint32_t u = __float_as_uint(s.cd[off + i]);
            if ((u & pmask) == prefix) {
                const uint32_t d = (u >> shift) & 255u;
                atomicAdd(&s.hist[d >> 1], 1u << ((d & 1u) * 16u));
            }
        }
        __syncwarp();
        prefix |= radix_pick(s, need) << shift;
        pmask |= 255u << shift;
        __syncwarp();
    }
    return __uint_as_float(prefix);
}

// k-th smallest (1-based) float32 part cd[0 .. cnt), for candidates that mostly lie in
// [0, hi]: one pass of 256 linear bins over [0, hi] (bin = d * 256 / hi, truncated and
// clamped, which is monotone in d, so the bins keep the order), then an exact rank among the
// entries of the bin that holds the k-th (usually one to three). Falls back to the four-pass
// radix select when hi gives no spread or that bin holds more than 32 entries.
template <class S>
ALB_DEVICE float warp_kth32_lin(S& s, int cnt, int k, float hi) {
    const float scale = 256.f / hi;
    if (!(hi > 0.f) || !(scale < 1.0e30f)) return warp_kth32(s, 0, cnt, k);
    const int l = lane_id();
#pragma unroll 1
    for (int i = l; i < 128; i += 32) s.hist[i] = 0u;
    __syncwarp();
#pragma unroll 1
    for (int i = l; i < cnt; i += 32) {
        const uint32_t d = (uint32_t)min((int)(s.cd[i] * scale), 255);
        atomicAdd(&s.hist[d >> 1], 1u << ((d & 1u) * 16u));
    }
    __syncwarp();
    int need = k;
    const uint32_t B = radix_pick(s, need);  // need: rank inside bin B (1-based)
    __syncwarp();
    int m = 0;
#pragma unroll 1
    for (int base = 0; base < cnt; base += 32) {
        const int i = base + l;
        const float d = i < cnt ? s.cd[i] : 0.f;
        const bool in = i < cnt && (uint32_t)min((int)(d * scale), 255) == B;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int pos = m + __popc(b & lanemask_lt());
            if (pos < 32) s.hist[pos] = __float_as_uint(d);
        }
        m += __popc(b);
    }
    __syncwarp();
    if (m > 32) return warp_kth32(s, 0, cnt, k);
    const float v = l < m ? __uint_as_float(s.hist[l]) : FLT_MAX;
    int rank = 0;
#pragma unroll 1
    for (int j = 0; j < m; ++j) {
        const float o = __shfl_sync(0xffffffffu, v, j);
        rank += (o < v || (o == v && j < l)) ? 1 : 0;
    }
    const unsigned own = __ballot_sync(0xffffffffu, l < m && rank == need - 1);
    const float kth = __shfl_sync(0xffffffffu, v, __ffs(own) - 1);
    __syncwarp();
    return kth;
}

// k-th smallest (1-based) 48-bit candidate key by warp radix select over its top
// 8 * PASSES bits (PASSES = 4: the float32 part only; the lower bits return as 0).
template <int PASSES, class S>
ALB_DEVICE uint64_t warp_kth_key(S& s, int off, int cnt, int k) {
    const int l = lane_id();
    uint64_t prefix = 0ull, pmask = 0ull;
    int need = k;
#pragma unroll 1
    for (int pass = 0; pass < PASSES; ++pass) {
        const int shift = 40 - 8 * pass;
        for (int i = l; i < 128; i += 32) s.hist[i] = 0u;
        __syncwarp();
        for (int i = l; i < cnt; i += 32) {
            const uint64_t u = cand_key(s, off + i);
            if ((u & pmask) == prefix) {
                const uint32_t d = (uint32_t)(u >> shift) & 255u;
                atomicAdd(&s.hist[d >> 1], 1u << ((d & 1u) * 16u));
            }
        }
        __syncwarp();
        prefix |= ((uint64_t)radix_pick(s, need)) << shift;
        pmask |= 255ull << shift;
        __syncwarp();
    }
    return prefix;
}

// Keep the candidates whose float32 part is <= thr (order not preserved).
template <class S>
ALB_DEVICE int warp_compact(S& s, int cnt, float thr) {
    const int l = lane_id();
    int out = 0;
#pragma unroll 1
    for (int base = 0; base < cnt; base += 32) {
        int i = base + l;
        float d = i < cnt ? s.cd[i] : FLT_MAX;
        uint32_t id = i < cnt ? s.ci[i] : 0u;
        int16_t lo = i < cnt ? s.cl[i] : (int16_t)0;
        bool keep = i < cnt && d <= thr;
        unsigned b = __ballot_sync(0xffffffffu, keep);
        __syncwarp();
        if (keep) {
            int pos = out + __popc(b & lanemask_lt());
            s.cd[pos] = d;
            s.ci[pos] = id;
            s.cl[pos] = lo;
        }
        out += __popc(b);
        __syncwarp();
    }
    return out;
}


struct KnnResult {
    double rk2;    // float64 squared distance of the k-th neighbour
    float rkf;     // float32(sqrt(rk2)), correctly rounded
    int leaves;    // leaves opened (32 records each)
    int nodes;     // internal nodes expanded
    int selects;   // candidate-buffer reductions
    int fail;      // 0, or why the search has no answer (s.ci is then not valid):
                   // ALB_ERR_ITER_CAP (traversal guard), ALB_ERR_INVALID (fewer than k
                   // finite points admitted: a NaN or infinite query or map coordinates) or
                   // kCrowded (more near ties than its buffers hold)
};
// Searches whose near ties fill their buffers (coincident points, or a lattice of them) are left by the kernels
// below, marked, and answered by a launch of their own (k_gather_crowded, k_knn_crowded), which happens only where
// some are. Called from the searches' loops, the code that resolves any number of ties cost a whole run of the
// large scene 13% at 1e6 photons (34.6 -> 39.6 ms) and 16% at 1e7, by the registers that a call takes.
constexpr int kCrowded = 1;
ALB_DEVICE void leave_crowded(const QueryDev& q, uint32_t src, int channel) {
    if (lane_id() == 0) {
        atomicOr(reinterpret_cast<unsigned*>(&q.c[src].w), 1u << channel);
        atomicOr(q.crowded, 1u << channel);
    }
    __syncwarp();
}

// Positions of points: a map's records, or a packed array.
struct MapPoints {
    const float4* a;
    ALB_DEVICE float4 at(uint32_t r) const { return a[r]; }
};
struct PackedPoints {
    const float* p;
    ALB_DEVICE float4 at(uint32_t r) const { return make_float4(p[3 * r], p[3 * r + 1], p[3 * r + 2], 0.f); }
};

// float64 ranking of the band entries bi[0..nb) by (distance, tie key, map position); the
// `take` smallest go to ci[dst ..] in rank order. Returns the float64 squared distance of
// the take-th (0 if the band holds fewer).
template <class P, class S>
ALB_DEVICE double rank_band(P pts, S& s, int dst, int nb, int take, double qx, double qy,
                            double qz, const float4* tie_rec) {
    const int l = lane_id();
    double di = 0.0;
    uint64_t ti = 0ull;
    uint32_t ii = 0u;
    int rank = 0;
    if (l < nb) {
        ii = s.bi[l];
        const float4 a = pts.at(ii);
        di = point_dist2_f64(qx, qy, qz, a);
        ti = tie_rec ? record_tie_key(a, tie_rec[ii]) : 0ull;
        s.bd[l] = di;
        s.bt[l] = ti;
    }
    __syncwarp();
    if (l < nb) {
#pragma unroll 1
        for (int j = 0; j < nb; ++j) {
            const double dj = s.bd[j];
            const uint64_t tj = s.bt[j];
            rank += (dj < di || (dj == di && (tj < ti || (tj == ti && s.bi[j] < ii)))) ? 1 : 0;
        }
    }
    __syncwarp();
    if (l < nb && rank < take) s.ci[dst + rank] = ii;
    const unsigned owner = __ballot_sync(0xffffffffu, l < nb && rank == take - 1);
    const double rk2 = owner ? __shfl_sync(0xffffffffu, di, __ffs(owner) - 1) : 0.0;
    __syncwarp();
    return rk2;
}

// A point's place in the order of a search's answers: float64 squared distance (its bits: non-negative doubles
// order like them), tie key, map position.
struct Place {
    uint64_t d, t;
    uint32_t id;
    ALB_DEVICE bool before(const Place& o) const { return d < o.d || (d == o.d && (t < o.t || (t == o.t && id < o.id))); }
};

// Leaves of the entries [off, off + n) the first k in that order, whatever their ties, and returns the k-th's
// place. Every entry is ranked against every other one in registers: 288 entries take some 15 000
// instructions, but only searches with more entries at one distance than their buffers hold come here.
template <class P, class S>
__device__ __noinline__ Place keep_nearest(P pts, S& s, int off, int n, int k, double qx, double qy, double qz,
                                            const float4* tie_rec) {
    constexpr int R = S::kCap / 32;
    const int l = lane_id();
    Place e[R];
    int rank[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const bool on = i * 32 + l < n;
        e[i] = Place{~0ull, ~0ull, 0u};  // behind every entry
        rank[i] = 0;
        if (on) {
            e[i].id = s.ci[off + i * 32 + l];
            const float4 a = pts.at(e[i].id);
            e[i].d = (uint64_t)__double_as_longlong(point_dist2_f64(qx, qy, qz, a));
            e[i].t = tie_rec ? record_tie_key(a, tie_rec[e[i].id]) : 0ull;
        }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
#pragma unroll 1
        for (int src = 0; src < min(32, n - j * 32); ++src) {
            const Place o{__shfl_sync(0xffffffffu, e[j].d, src), __shfl_sync(0xffffffffu, e[j].t, src),
                          __shfl_sync(0xffffffffu, e[j].id, src)};
#pragma unroll
            for (int i = 0; i < R; ++i) rank[i] += o.before(e[i]) ? 1 : 0;
        }
    }
    int out = 0;
    Place last{0ull, 0ull, 0u};
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (i * 32 >= n) break;
        const int at = off + i * 32 + l;
        const bool keep = i * 32 + l < n && rank[i] < k;
        const float hi = keep ? s.cd[at] : 0.f;
        const int16_t lo = keep ? s.cl[at] : (int16_t)0;
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        __syncwarp();
        if (keep) {
            const int pos = off + out + __popc(b & lanemask_lt());
            s.cd[pos] = hi;
            s.ci[pos] = e[i].id;
            s.cl[pos] = lo;
        }
        out += __popc(b);
        const unsigned own = __ballot_sync(0xffffffffu, keep && rank[i] == k - 1);
        if (own) {
            const int src = __ffs(own) - 1;
            last = Place{__shfl_sync(0xffffffffu, e[i].d, src), __shfl_sync(0xffffffffu, e[i].t, src),
                         __shfl_sync(0xffffffffu, e[i].id, src)};
        }
        __syncwarp();
    }
    return last;
}

// The k_sub nearest among the entries [off, off + n) whose cd/cl hold refined keys: keys more
// than one unit below the k_sub-th are in, keys within one unit of it are ranked in float64.
// The chosen map positions end up in ci[off .. off + k_sub). A band of more than kBand entries is ranked with
// TIES (in scratch words: the search is done with its stack), and otherwise left: fail = kCrowded.
template <bool TIES, class P, class S>
ALB_DEVICE double select_refined(P pts, S& s, int off, int n, int k_sub, double qx, double qy,
                                 double qz, const float4* tie_rec, int& fail) {
    static_assert(S::kCap <= S::kTmp, "the band is a subset of the candidates");
    const int l = lane_id();
    const uint64_t K = warp_kth_key<6>(s, off, n, k_sub);
    int n_in = 0, n_band = 0;
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
        const bool valid = base + l < n;
        const int i = off + base + l;
        const uint64_t key = valid ? cand_key(s, i) : ~0ull;
        const uint32_t id = valid ? s.ci[i] : 0u;
        const bool in = valid && key + 1ull < K;
        const bool band = valid && !in && key <= K + 1ull;
        const unsigned bin = __ballot_sync(0xffffffffu, in);
        const unsigned bb = __ballot_sync(0xffffffffu, band);
        __syncwarp();
        if (in) s.ci[off + n_in + __popc(bin & lanemask_lt())] = id;
        if (band) {
            const int pos = n_band + __popc(bb & lanemask_lt());
            if (pos < kBand) s.bi[pos] = id;
            else if (TIES) s.tmp(pos) = id;
        }
        n_in += __popc(bin);
        n_band += __popc(bb);
        __syncwarp();
    }
    if (n_band > kBand) {
        if constexpr (TIES) {
            for (int j = l; j < n_band; j += 32) s.ci[off + n_in + j] = j < kBand ? s.bi[j] : s.tmp(j);
            __syncwarp();
            const Place kth = keep_nearest(pts, s, off + n_in, n_band, k_sub - n_in, qx, qy, qz, tie_rec);
            return __longlong_as_double((long long)kth.d);
        } else {
            fail = kCrowded;
            return 0.0;
        }
    }
    return rank_band(pts, s, off + n_in, n_band, k_sub - n_in, qx, qy, qz, tie_rec);
}

// Full k-NN search for one query. Returns false when the map has fewer than k records; the
// k nearest map positions are then in s.ci[0 .. k).
// bound: an upper bound of the squared k-th distance that already includes the band margin
// (FLT_MAX when none is known). A search that admits fewer than k points under it is repeated
// without one, so the answer is always the one a search from no bound gives.
// The query is (fx + lx, fy + ly, fz + lz) = (qx, qy, qz) exactly, |l*| <= half an ulp of f*.
// Points at exactly the same float64 distance rank by a key taken from their record content
// (time, then a hash of direction, time and energy; when tie_rec is given) and then by map
// position, so that the chosen neighbours do not depend on the order in which the map's
// records are stored (records equal in all of these contribute identically).
// REFINE: candidates carry double-float distances from admission on, so the buffer only ever
// holds entries within one float32 ulp of the k-th: needed where many points sit at nearly
// the same distance (queries far from a dense planar map). Without it candidates carry the
// float32 screening distance and only a crowded final band is refined.
// TIES: any number of near ties is resolved; without it a search whose buffers they fill ends with kCrowded.
// Once they have filled the buffers, a point is admitted only if it comes before the k-th best so far in the
// order of answers (one of coincident points needs no float64 distance for that): where all of a map's N records
// coincide, about k ln(N / k) of them are. Surface gather of 80 000 queries around a spot of 1e6 records 8 um wide:
// 2.5 s (23.8 s with every tied record admitted; 11.6 s when ties were dropped as they came).
template <bool REFINE, bool QSPLIT = false, bool TIES = false, class S>
ALB_DEVICE bool warp_knn(const MapDev& m, S& s, int k, double qx, double qy, double qz, float fx,
                         float fy, float fz, float lx, float ly, float lz, float bound, const float4* tie_rec,
                         KnnResult& res) {
    const int l = lane_id();
    if (m.n_real < (uint64_t)k) return false;
    float thr = bound;  // admission threshold (float32 squared distance, with margin)
    int cnt = 0;
    res.leaves = res.nodes = res.selects = res.fail = 0;
    // The carried bound first, then none (a caller's bound is a promise that k points lie within it; one that does
    // not hold costs a second search).
    float start = bound;
    Place last{~0ull, ~0ull, ~0u};  // (TIES) the k-th best so far, once the buffers have been full
    float4 at = make_float4(0.f, 0.f, 0.f, 0.f);
    bool full = false;
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (attempt == 1) {
            if (start == FLT_MAX) break;
            start = FLT_MAX;
        }
        thr = start;
        cnt = 0;
        int sp = 0;
        // roots
        {
            int top = m.nlevels - 1;
            uint64_t ntop = m.lvl_cnt[top];
            float d = FLT_MAX;
            uint32_t c = (uint32_t)l;
            if ((uint64_t)l < ntop) {
                d = box_dist2(fx, fy, fz, lx, ly, lz, m.box_lo[m.lvl_off[top] + l], m.box_hi[m.lvl_off[top] + l]);
                if (d > thr) d = FLT_MAX;
            }
            warp_sort32(d, c);
            unsigned b = __ballot_sync(0xffffffffu, d < FLT_MAX);
            int nv = __popc(b);
            if (l < nv) {
                s.stk[sp + nv - 1 - l] = ((uint32_t)top << 29) | c;
                s.stk_d[sp + nv - 1 - l] = d;
            }
            sp += nv;
            __syncwarp();
        }
        int guard = 0;
        // screen the 32 records of leaf `leaf` (p = this lane's record) against the threshold
        auto admit = [&](uint32_t leaf, float4 p) {
            ++res.leaves;
            const uint64_t r = (uint64_t)leaf * 32 + l;
            const bool real = r < m.n;  // the last leaf may be partial
            const float d = real ? point_dist2(fx, fy, fz, lx, ly, lz, p) : FLT_MAX;
            bool take = real && d <= thr;
            if (TIES && full && take) {
                Place o{last.d, 0ull, (uint32_t)r};
                if (p.x != at.x || p.y != at.y || p.z != at.z)
                    o.d = (uint64_t)__double_as_longlong(point_dist2_f64(qx, qy, qz, p));
                if (o.d == last.d && tie_rec) o.t = record_tie_key(p, tie_rec[r]);
                take = o.before(last);
            }
            const unsigned b = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int pos = cnt + __popc(b & lanemask_lt());
                s.ci[pos] = (uint32_t)r;
                if (REFINE) {
                    float hi, lo;
                    point_dist2_df(fx, fy, fz, lx, ly, lz, p, hi, lo);
                    s.cd[pos] = hi;
                    s.cl[pos] = frac16(hi, lo);
                } else {
                    s.cd[pos] = d;
                }
            }
            cnt += __popc(b);
            __syncwarp();
            if (TIES && full) {
                if (cnt > S::kCap - 32) {
                    ++res.selects;
                    last = keep_nearest(MapPoints{m.a}, s, 0, cnt, k, qx, qy, qz, tie_rec);
                    cnt = k;
                    at = m.a[last.id];
                    thr = fminf(thr, __double2float_ru(__longlong_as_double((long long)last.d)) * (1.0f + 2.0f * kRelMargin));
                }
            } else if (cnt >= k && (thr == FLT_MAX || cnt > S::kSelectAt)) {
                ++res.selects;
                // planar maps (REFINE) crowd their candidates into one linear bin: radix select
                const float kth = REFINE ? warp_kth32(s, 0, cnt, k) : warp_kth32_lin(s, cnt, k, thr);
                thr = fminf(thr, kth * (1.0f + 2.0f * kRelMargin));
                // REFINE: refined distances within one float32 ulp of the k-th can still
                // rank among the k nearest, nothing beyond can; otherwise the float32
                // screening margin decides
                cnt = warp_compact(s, cnt, REFINE ? __uint_as_float(__float_as_uint(kth) + 1u) : thr);
                if (cnt > S::kCap - 32) {  // more near ties than there is room for: the k best so far are enough
                    if (TIES) {
                        last = keep_nearest(MapPoints{m.a}, s, 0, cnt, k, qx, qy, qz, tie_rec);
                        cnt = k;
                        at = m.a[last.id];
                        full = true;
                    } else {
                        res.fail = kCrowded;
                        sp = 0;
                    }
                }
            }
        };
        auto load_leaf = [&](uint32_t leaf) {
            const uint64_t r = (uint64_t)leaf * 32 + l;
            return r < m.n ? m.a[r] : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        while (sp > 0) {
            if (++guard > (1 << 22)) {  // reported, never a silent partial answer
                res.fail = ALB_ERR_ITER_CAP;
                break;
            }
            uint32_t etop;
            {
                // the top 32 stack entries, one per lane (lane 0 = top)
                const int i = sp - 1 - l;
                uint32_t e = 0u;
                bool ok = false;
                if (i >= 0) {
                    e = s.stk[i];
                    ok = s.stk_d[i] <= thr;
                }
                const unsigned okm = __ballot_sync(0xffffffffu, ok);
                if (!okm) {  // 32 entries beyond the threshold
                    sp = sp > 32 ? sp - 32 : 0;
                    __syncwarp();
                    continue;
                }
                const int f = __ffs(okm) - 1;
                etop = __shfl_sync(0xffffffffu, e, f);
                sp -= f + 1;
                __syncwarp();
            }
            if ((etop >> 29) == 0) {
                // a leaf: admit its points within the threshold
                admit(etop, load_leaf(etop));
            } else {
                ++res.nodes;
                const int lev = (int)(etop >> 29);
                const uint32_t node = etop & 0x1fffffffu;
                uint64_t c = (uint64_t)node * 32 + l;
                float d = FLT_MAX;
                int cl = lev - 1;
                if (c < m.lvl_cnt[cl]) {
                    d = box_dist2(fx, fy, fz, lx, ly, lz, m.box_lo[m.lvl_off[cl] + c], m.box_hi[m.lvl_off[cl] + c]);
                    if (d > thr) d = FLT_MAX;
                }
                uint32_t cc = (uint32_t)c;
                const unsigned vm = __ballot_sync(0xffffffffu, d < FLT_MAX);
                int nv = __popc(vm);
                if (nv <= 16) {
                    // few children within the threshold: extract them nearest first
                    // (non-negative floats order like their bit patterns)
                    unsigned key = __float_as_uint(d);
                    for (int r = 0; r < nv; ++r) {
                        unsigned mn = __reduce_min_sync(0xffffffffu, key);
                        int src = __ffs(__ballot_sync(0xffffffffu, key == mn)) - 1;
                        if (l == src) {
                            s.stk[sp + nv - 1 - r] = ((uint32_t)cl << 29) | cc;
                            s.stk_d[sp + nv - 1 - r] = d;
                            key = 0xffffffffu;
                        }
                    }
                } else {
                    warp_sort32(d, cc);
                    if (l < nv) {
                        s.stk[sp + nv - 1 - l] = ((uint32_t)cl << 29) | cc;
                        s.stk_d[sp + nv - 1 - l] = d;
                    }
                }
                sp += nv;
                __syncwarp();
            }
        }
        if (res.fail || start == FLT_MAX || cnt >= k) break;
    }
    if (!res.fail && cnt < k) res.fail = ALB_ERR_INVALID;
    if (res.fail) return true;
    if (QSPLIT) {
        // the float64 query is exactly its float32 split (f + l): rebuilt here rather than
        // held in registers through the search
        qx = (double)fx + (double)lx;
        qy = (double)fy + (double)ly;
        qz = (double)fz + (double)lz;
    }
    double rk2;
    if (REFINE) {
        rk2 = select_refined<TIES>(MapPoints{m.a}, s, 0, cnt, k, qx, qy, qz, tie_rec, res.fail);
    } else {
        // float32 k-th; entries clearly below it are in, the band within the screening
        // margin around it is resolved exactly (refined keys when it is crowded)
        const float kth = warp_kth32(s, 0, cnt, k);
        const float blo = kth * (1.0f - 2.0f * kRelMargin), bhi = kth * (1.0f + 2.0f * kRelMargin);
        int n_in = 0, n_band = 0;
#pragma unroll 1
        for (int base = 0; base < cnt; base += 32) {
            const int i = base + l;
            const bool valid = i < cnt;
            const float d = valid ? s.cd[i] : FLT_MAX;
            const uint32_t id = valid ? s.ci[i] : 0u;
            const bool in = valid && d < blo;
            const bool band = valid && d >= blo && d <= bhi;
            const unsigned bin = __ballot_sync(0xffffffffu, in);
            const unsigned bb = __ballot_sync(0xffffffffu, band);
            __syncwarp();
            if (in) s.ci[n_in + __popc(bin & lanemask_lt())] = id;
            if (band) {
                const int pos = n_band + __popc(bb & lanemask_lt());
                if (pos < S::kTmp) s.tmp(pos) = id;
            }
            n_in += __popc(bin);
            n_band += __popc(bb);
            __syncwarp();
        }
        const int take = k - n_in;
        if (n_band <= kBand) {
            if (l < n_band) s.bi[l] = s.tmp(l);
            __syncwarp();
            rk2 = rank_band(MapPoints{m.a}, s, n_in, n_band, take, qx, qy, qz, tie_rec);
        } else {
#pragma unroll 1
            for (int j = l; j < n_band; j += 32) {
                const uint32_t id = s.tmp(j);
                float hi, lo;
                point_dist2_df(fx, fy, fz, lx, ly, lz, m.a[id], hi, lo);
                s.cd[n_in + j] = hi;
                s.cl[n_in + j] = frac16(hi, lo);
                s.ci[n_in + j] = id;
            }
            __syncwarp();
            rk2 = select_refined<TIES>(MapPoints{m.a}, s, n_in, n_band, take, qx, qy, qz, tie_rec, res.fail);
        }
    }
    res.rk2 = rk2;
    res.rkf = sqrt_to_f32(rk2);
    return true;
}

// The search of a query whose near ties fill a search's buffers (the map holds at least k records).
template <class S>
__device__ __noinline__ KnnResult crowded_knn(const MapDev& m, S& s, int k, double qx, double qy, double qz,
                                              const float4* tie_rec) {
    const float fx = (float)qx, fy = (float)qy, fz = (float)qz;
    KnnResult r;
    warp_knn<true, false, true>(m, s, k, qx, qy, qz, fx, fy, fz, (float)(qx - (double)fx), (float)(qy - (double)fy),
                                (float)(qz - (double)fz), FLT_MAX, tie_rec, r);
    return r;
}

}  // namespace alb
#include "gather_group.cuh"
namespace alb {

// ----------------------------------------------------------------------------------------
// per-neighbour weights (float32 restatement of the reference's energy multipliers)
// ----------------------------------------------------------------------------------------

// GGX Cook-Torrance, alb_sim/physics/reflection/microfacet_brdf.py:96-147, with
// wi = normalize(-d_map), wo = normalize(-d_query), n = +y.
ALB_DEVICE float ggx_weight(float a2, float f0, float wix, float wiy, float wiz, float wox, float woy, float woz) {
    float ni = rsqrtf(fmaf(wix, wix, fmaf(wiy, wiy, wiz * wiz)));
    wix *= ni; wiy *= ni; wiz *= ni;
    float n_wi = fminf(fmaxf(wiy, 0.f), 1.f);
    float n_wo = fminf(fmaxf(woy, 0.f), 1.f);
    if (!(n_wi > 0.f && n_wo > 0.f)) return 0.f;
    // Unnormalised half vector H = wi + wo. The reference's denominator
    // (a2 - 1) (n.h)^2 + 1 cancels near the specular peak; with h = H / |H| it equals
    // (Hx^2 + Hz^2 + a2 Hy^2) / |H|^2, a sum of non-negative terms that float32 keeps.
    float Hx = wix + wox, Hy = wiy + woy, Hz = wiz + woz;
    float t = fmaf(Hx, Hx, Hz * Hz);
    float H2 = fmaf(Hy, Hy, t);
    float den = 1.f, wi_h = 0.f;
    if (H2 > 0.f) {
        float inv = 1.f / H2;
        if (Hy > 0.f) den = fmaf(a2 * Hy, Hy, t) * inv;
        wi_h = fminf(fmaxf(fmaf(wix, Hx, fmaf(wiy, Hy, wiz * Hz)) * rsqrtf(H2), 0.f), 1.f);
    }
    float D = a2 / (3.14159265358979f * den * den + kEps32);
    float g1i = 2.f * n_wi / (n_wi + sqrtf(fmaf(1.f - a2, n_wi * n_wi, a2)));
    float g1o = 2.f * n_wo / (n_wo + sqrtf(fmaf(1.f - a2, n_wo * n_wo, a2)));
    float x = 1.f - wi_h;
    float x2 = x * x;
    float F = f0 + (1.f - f0) * (x2 * x2 * x);
    return (D * g1i * g1o * F) / (4.f * n_wi * n_wo + kEps32);
}

// Scatter weight: CDF mass of the angular bin of theta = acos(d_map . view),
// alb_sim/physics/scatter/energy.py:8-52 (view = normalize(-d_query)).
ALB_DEVICE int scatter_bin(const SceneDev& sc, int layer, float dx, float dy, float dz, float vx, float vy, float vz) {
    float n = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
    float c = fmaf(dx, vx, fmaf(dy, vy, dz * vz)) * n;
    c = fminf(fmaxf(c, -1.f), 1.f);
    float th = acosf(c);
    int i = (int)((th - kEps32) / sc.layer_binw[layer]);
    return min(max(i, 0), ALB_PHASE_DIVISIONS - 1);
}
ALB_DEVICE float scatter_weight(const SceneDev& sc, int layer, float dx, float dy, float dz, float vx, float vy, float vz) {
    return __ldg(sc.layer_weight[layer] + scatter_bin(sc, layer, dx, dy, dz, vx, vy, vz));
}

// Adjoint (extension): d ln(ggx_weight) / d(alpha^2), the same vectors as ggx_weight:
// 1/a2 - 2 Hy^2 / (|H|^2 den) * pi den^2 / (pi den^2 + eps) from the distribution term and
// -(1 - n^2) / (2 s (n + s)), s = sqrt((1 - a2) n^2 + a2), from each Smith G1 factor; the
// Fresnel term has no a2. Which products are rounded before their sum is written out, so that a result does not
// depend on what else the compiler finds around the call.
ALB_DEVICE float ggx_dlog_da2(float a2, float wix, float wiy, float wiz, float wox, float woy, float woz) {
    float ni = rsqrtf(fmaf(wix, wix, fmaf(wiy, wiy, wiz * wiz)));
    wix *= ni; wiy *= ni; wiz *= ni;
    float n_wi = fminf(fmaxf(wiy, 0.f), 1.f);
    float n_wo = fminf(fmaxf(woy, 0.f), 1.f);
    if (!(n_wi > 0.f && n_wo > 0.f)) return 0.f;
    float Hx = wix + wox, Hy = wiy + woy, Hz = wiz + woz;
    float t = fmaf(Hx, Hx, Hz * Hz);
    float H2 = fmaf(Hy, Hy, t);
    float d = 1.f / a2;
    if (H2 > 0.f && Hy > 0.f) {
        float den = fmaf(a2 * Hy, Hy, t) / H2;
        // D = a2 / (pi den^2 + eps): the epsilon takes the share eps / (pi den^2 + eps) of
        // the denominator (about 0.6% at the specular peak for a2 = 0.0025)
        float pd2 = __fmul_rn(__fmul_rn(3.14159265358979f, den), den);
        d = fmaf(-(2.f * (Hy * Hy / H2) / den), pd2 / __fadd_rn(pd2, kEps32), d);
    }
    float si = sqrtf(fmaf(1.f - a2, n_wi * n_wi, a2)), so = sqrtf(fmaf(1.f - a2, n_wo * n_wo, a2));
    d -= __fsub_rn(1.f, __fmul_rn(n_wi, n_wi)) / (2.f * si * (n_wi + si));
    d -= fmaf(-n_wo, n_wo, 1.f) / (2.f * so * (n_wo + so));
    return d;
}

// float32 -> 128-bit fixed point (64 fractional bits), integer ops only.
ALB_DEVICE Fix128 f32_to_fix(float v) {
    Fix128 r{0ull, 0ll};
    uint32_t b = __float_as_uint(v);
    uint32_t ex = (b >> 23) & 0xffu;
    if (ex == 0u || ex == 255u) return r;  // zero / subnormal / inf / nan contribute nothing
    uint64_t mant = (uint64_t)((b & 0x7fffffu) | 0x800000u);
    int sh = (int)ex - 150 + 64;  // value * 2^64 = mant * 2^sh
    uint64_t lo = 0ull, hi = 0ull;
    if (sh > 86) {
        lo = ~0ull;
        hi = 0x7fffffffffffffffull;
    } else if (sh >= 64) {
        hi = mant << (sh - 64);
    } else if (sh > 40) {
        lo = mant << sh;
        hi = mant >> (64 - sh);
    } else if (sh >= 0) {
        lo = mant << sh;
    } else if (sh > -24) {
        lo = mant >> (-sh);
    }
    if (b & 0x80000000u) {
        lo = ~lo + 1ull;
        hi = ~hi + (lo == 0ull ? 1ull : 0ull);
    }
    r.lo = lo;
    r.hi = (long long)hi;
    return r;
}

// One contribution to cell `i` of a 128-bit accumulator: one 64-bit add whose result nobody waits
// for. A float32 is 24 bits at a shift sh (value 2^64 = mant 2^sh); its class is sh / 4, and the
// class's word of the cell takes +- mant << (sh % 4), below 2^27, so 2^36 contributions fit
// (kClassMost, kept by the launches). k_merge_classes sums the words exactly into the
// accumulator and leaves them zero. A direct 128-bit add takes two atomics, the second on the
// first one's carry, and the warp waits for both: scatter gather of the large scene, 1e6 photons,
// 29.7 -> 24.8 ms. Bins in shared memory caught less than half of the scatter contributions
// (multiple scattering spreads a range of queries over ten thousand bins).
// 2^23 and more, and what is not finite, goes the direct way.
constexpr int kClasses = 16;
constexpr uint64_t kClassMost = 1ull << 36;
// c's class and what its word takes; -1: nothing (zero or subnormal), -2: the direct way.
ALB_DEVICE int class_of(float c, long long& v) {
    const uint32_t b = __float_as_uint(c) & 0x7fffffffu;
    if (b >= 0x4b000000u) return -2;
    if (b < 0x00800000u) return -1;
    uint32_t mant = (b & 0x7fffffu) | 0x800000u;
    int sh = (int)(b >> 23) - 86;
    if (sh < 0) {
        mant >>= min(-sh, 31);
        sh = 0;
    }
    v = (long long)(mant << (sh & 3));
    if (c < 0.f) v = -v;
    return sh >> 2;
}
template <class C>
ALB_DEVICE void class_add(C& cache, bool on, uint32_t base, unsigned long long* cls, uint32_t n, uint32_t i, float c,
                          unsigned long long* lo, unsigned long long* hi) {
    long long v;
    const int k = class_of(c, v);
    if (k >= 0) word_add(cache, on, cls, (uint64_t)(uint32_t)k * n + i, base, i + 37u * (uint32_t)k, v);
    else if (k == -2) fix_atomic_add(lo + i, hi + i, f32_to_fix(c));
}

// The same where the accumulator may have no class words (cls null: direct).
template <class C>
ALB_DEVICE void cell_add(C& cache, bool on, uint32_t base, unsigned long long* cls, uint32_t n, uint32_t i, float c,
                         unsigned long long* lo, unsigned long long* hi) {
    if (cls) class_add(cache, on, base, cls, n, i, c, lo, hi);
    else fix_atomic_add(lo + i, hi + i, f32_to_fix(c));
}

// The class words of n cells (blockIdx.y: one of several accumulators, cls_step and out_step words
// apart) into their 128-bit words; the class words are left zero.
__global__ void k_merge_classes(unsigned long long* cls, uint32_t n, unsigned long long* lo, unsigned long long* hi,
                                uint64_t cls_step, uint64_t out_step) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    cls += blockIdx.y * cls_step;
    unsigned long long w[kClasses];
    unsigned long long any = 0ull;
#pragma unroll
    for (int c = 0; c < kClasses; ++c) {
        w[c] = cls[(uint64_t)c * n + i];
        any |= w[c];
    }
    if (!any) return;
    Fix128 sum{0ull, 0ll};
#pragma unroll
    for (int c = 0; c < kClasses; ++c) {
        if (!w[c]) continue;
        cls[(uint64_t)c * n + i] = 0ull;
        fix_add(sum, Fix128{w[c] << (4 * c), (long long)w[c] >> (c ? 64 - 4 * c : 63)});
    }
    const uint64_t o = blockIdx.y * out_step + i;
    fix_atomic_add(lo + o, hi + o, sum);
}

// Per-CTA shared-memory cache of waveform bins: direct-mapped on the bin index, a slot is
// claimed once by CAS on its tag; hits are exact 128-bit integer adds in shared memory,
// misses go to global memory. Flushed once when the CTA finishes. The sum is integer, so
// the split between cache and global memory cannot change the result. The sum is held in 32-bit
// words, which shared memory adds natively: a float32 touches two of them, and a third on a carry (64-bit
// shared adds are compare-and-swap loops, and a query's neighbours mostly share a few bins: surface
// gather of 25 000 queries at a radius of 0.5 m 13.1 -> 4.3 ms, 250 000 k-nearest ones 2.46 -> 2.09).
constexpr int kBinCache = 256;
struct BinCache {
    int tag[kBinCache];
    uint32_t w[4][kBinCache];
};

ALB_DEVICE void bin_add(BinCache& bc, const Accum& acc, int channel, int bin, float c) {
    int slot = bin & (kBinCache - 1);
    int t = bc.tag[slot];
    if (t != bin && t == -1) {
        int old = atomicCAS(&bc.tag[slot], -1, bin);
        t = (old == -1) ? bin : old;
    }
    const uint32_t b = __float_as_uint(c);
    if (t == bin && b < 0x4f800000u) {  // 0 <= c < 2^32
        if (b < 0x00800000u) return;    // zero or subnormal
        uint32_t mant = (b & 0x7fffffu) | 0x800000u;
        int sh = (int)(b >> 23) - 86;  // c 2^64 = mant 2^sh
        if (sh < 0) {
            mant >>= min(-sh, 31);
            sh = 0;
        }
        const uint64_t v = (uint64_t)mant << (sh & 31);
        uint32_t* w = &bc.w[0][slot] + (sh >> 5) * kBinCache;
        const uint32_t lo = (uint32_t)v;
        const uint32_t old = atomicAdd(w, lo);
        uint32_t up = (uint32_t)(v >> 32) + (old + lo < old ? 1u : 0u);
        for (int i = (sh >> 5) + 1; up && i < 4; ++i) {
            w += kBinCache;
            up = atomicAdd(w, up) + up < up ? 1u : 0u;
        }
        return;
    }
    uint64_t o = (uint64_t)channel * acc.nbins + bin;
    fix_atomic_add(acc.wf_lo + o, acc.wf_hi + o, f32_to_fix(c));
}

// The CTA's cached bins into the global waveform (after a block barrier).
template <int CHANNEL>
ALB_DEVICE void bin_flush(const BinCache& bc, const Accum& acc) {
    for (int i = threadIdx.x; i < kBinCache; i += blockDim.x) {
        int t = bc.tag[i];
        if (t >= 0) {
            uint64_t o = (uint64_t)CHANNEL * acc.nbins + t;
            Fix128 f{(uint64_t)bc.w[1][i] << 32 | bc.w[0][i], (long long)((uint64_t)bc.w[3][i] << 32 | bc.w[2][i])};
            fix_atomic_add(acc.wf_lo + o, acc.wf_hi + o, f);
        }
    }
}

constexpr uint32_t kRoot = 0xffffffffu;
constexpr int kLeafBudget = 64;
struct RadiusWork {
    uint2* items;     // nullable
    uint32_t* count;  // items wanted (more than cap: the rest was searched in place)
    uint32_t cap;
    bool second;      // this launch takes the items
};

// Extension (no counterpart in the reference): every record within the fixed radius R of
// the query, visited in any order. Screening as in the k-NN search; points within the
// float32 error band of R are decided on their float64 distance. visit(record) runs on the
// lanes holding admitted records. start: the box to search (a stack entry), kRoot: the map.
// Queries at the beam's spot meet most of the map's leaves, others none: once a query has
// visited kLeafBudget leaves, the boxes of 32 leaves still to come become work items (src, box) of
// a second launch, where there is room for them. With a query left to one warp the heaviest of 25,000
// (3500 leaves) took the surface gather's 4.6 ms by itself; all four gathers 4.6 -> 0.56 ms (budgets of
// 32 and 128 leaves: 0.53, 0.60).
template <class F>
ALB_DEVICE void warp_radius_visit(const MapDev& m, WarpSmem& s, const RadiusWork& work, uint32_t src, uint32_t start, double qx, double qy, double qz, float fx, float fy,
                                  float fz, float lx, float ly, float lz, double R, F&& visit, KnnResult& res) {
    const int l = lane_id();
    const double R2 = R * R;
    const float thr = __double2float_ru(R2) * (1.0f + 2.0f * kRelMargin);
    const float lo_band = __double2float_rd(R2) * (1.0f - 2.0f * kRelMargin);
    res.leaves = res.nodes = res.selects = res.fail = 0;
    res.rk2 = R2;
    res.rkf = (float)R;
    if (m.nlevels <= 0) return;  // an empty map contributes nothing
    int sp = 0;
    if (start != kRoot) {
        if (l == 0) s.stk[0] = start;
        sp = 1;
        __syncwarp();
    } else {
        const int top = m.nlevels - 1;
        bool ok = false;
        if ((uint64_t)l < m.lvl_cnt[top])
            ok = box_dist2(fx, fy, fz, lx, ly, lz, m.box_lo[m.lvl_off[top] + l], m.box_hi[m.lvl_off[top] + l]) <= thr;
        const unsigned b = __ballot_sync(0xffffffffu, ok);
        if (ok) s.stk[sp + __popc(b & lanemask_lt())] = ((uint32_t)top << 29) | (uint32_t)l;
        sp += __popc(b);
        __syncwarp();
    }
    // every box is pushed at most once, so the box count bounds the loop
    const uint64_t boxes = m.lvl_off[m.nlevels - 1] + m.lvl_cnt[m.nlevels - 1];
    uint64_t guard = 0;
    while (sp > 0) {
        if (++guard > boxes) {
            res.fail = ALB_ERR_ITER_CAP;
            break;
        }
        --sp;
        const uint32_t e = s.stk[sp];
        __syncwarp();
        const int lev = (int)(e >> 29);
        const uint32_t node = e & 0x1fffffffu;
        if (lev == 1 && res.leaves >= kLeafBudget && work.items && !work.second) {
            uint32_t slot = 0u;
            if (l == 0) {
                // (not counted on once full: the counter must not wrap)
                slot = *(volatile uint32_t*)work.count;
                if (slot < work.cap) slot = atomicAdd(work.count, 1u);
                if (slot < work.cap) work.items[slot] = make_uint2(src, e);
            }
            if (__shfl_sync(0xffffffffu, slot, 0) < work.cap) continue;
        }
        if (lev == 0) {
            ++res.leaves;
            const uint64_t r = (uint64_t)node * 32 + l;
            bool in = false;
            if (r < m.n) {
                const float4 p = m.a[r];
                const float d = point_dist2(fx, fy, fz, lx, ly, lz, p);
                in = d < lo_band || (d <= thr && point_dist2_f64(qx, qy, qz, p) <= R2);
            }
            if (in) visit((uint32_t)r);
        } else {
            ++res.nodes;
            const int cl = lev - 1;
            const uint64_t c = (uint64_t)node * 32 + l;
            bool ok = false;
            if (c < m.lvl_cnt[cl])
                ok = box_dist2(fx, fy, fz, lx, ly, lz, m.box_lo[m.lvl_off[cl] + c], m.box_hi[m.lvl_off[cl] + c]) <= thr;
            const unsigned b = __ballot_sync(0xffffffffu, ok);
            if (ok) s.stk[sp + __popc(b & lanemask_lt())] = ((uint32_t)cl << 29) | (uint32_t)c;
            sp += __popc(b);
            __syncwarp();
        }
    }
}

// Adjoint (extension): one neighbour's c (s_query + s_record + d ln w / d theta) into the
// Jacobian for theta = a, b, g, albedo, roughness (128-bit fixed point by class words).
// Bins below which the number of every class word (the waveform's, then the Jacobian's or two heatmaps')
// fits 32 bits; a longer waveform's words are not cached.
constexpr int64_t kCachedBins = 1 << 25;

template <int CHANNEL, class C>
ALB_DEVICE void jac_add(const SceneDev& sc, const MapDev& m, const Accum& acc, C& cache, bool on, uint32_t base, int layer, int bin, uint32_t idx,
                        float c, float4 sq, float4 pb, float vx, float vy, float vz) {
    const float4 sp = m.sco ? m.sco[idx] : make_float4(0.f, 0.f, 0.f, 0.f);
    float d[kJacParams];
    d[0] = sq.x + sp.x;
    d[1] = sq.y + sp.y;
    d[2] = sq.z + sp.z;
    d[3] = sq.w + sp.w;
    d[4] = 0.f;
    if (CHANNEL == ALB_SCATTER && sc.layer_dlw_g[layer])
        d[2] += __ldg(sc.layer_dlw_g[layer] + scatter_bin(sc, layer, pb.x, pb.y, pb.z, vx, vy, vz));
    if (CHANNEL == ALB_BOTTOM_REFLECTION) d[3] += sc.inv_albedo;
    if (CHANNEL == ALB_SURFACE_REFLECTION) d[4] = sc.dla2_drough * ggx_dlog_da2(sc.ggx_a2, -pb.x, -pb.y, -pb.z, vx, vy, vz);
#pragma unroll
    for (int p = 0; p < kJacParams; ++p) {
        const uint64_t o = ((uint64_t)p * ALB_CHANNELS + CHANNEL) * acc.nbins + bin;
        long long v = 0;
        int k = -2;
        if (acc.jac_cls) k = class_of(c * d[p], v);
        if (k >= 0) {
            const uint32_t plane = (uint32_t)(p * kClasses + k);
            word_add(cache, on, acc.jac_cls, (uint64_t)plane * (uint32_t)acc.nbins + (uint32_t)bin, base,
                     (uint32_t)bin + 37u * plane + 13u, v);
        } else if (k == -2) {
            fix_atomic_add(acc.jac_lo + o, acc.jac_hi + o, f32_to_fix(c * d[p]));
        }
    }
}

// (long long)((x - c + ext) / bin) in float64, as numpy forms the heatmap cell, or -1 outside
// [0, bins). The float32 value v decides wherever it is farther from an integer than its own
// error: five roundings of terms up to |v| + 2 ext / bin <= 1024 cells, under 3.1e-4 (the host
// sets inv = 0 for more than 512 bins, which always takes the float64 path). A neighbour's four
// float64 divisions cost more issue time than the rest of its contribution: two FP64 lanes per SM.
ALB_DEVICE int heat_cell(float x, double c, double ext, double bin, float2 cf, float extf, float inv, int bins) {
    const float v = ((x - cf.x) - cf.y + extf) * inv;
    if (inv != 0.f && (v < -1.5f || v > (float)bins + 0.5f)) return -1;
    long long i;
    if (fabsf(v - rintf(v)) > 4.8828125e-04f) i = (long long)(int)v;
    else i = (long long)(((double)x - c + ext) / bin);
    return i >= 0 && i < bins ? (int)i : -1;
}

// accumulate_to_heatmap (alb_sim/math/accumulate_heatmap.py:6-61) for one neighbour
template <class C>
ALB_DEVICE void heat_add(const SceneDev& sc, const MapDev& m, const Accum& acc, C& cache, bool on, uint32_t base, uint32_t idx,
                         float c) {
    const float4 fw = m.fwi[idx], sf = m.sfi[idx];
    const uint32_t cells = (uint32_t)(sc.hm_bins * sc.hm_bins);
    if (fw.x == fw.x) {
        const int xi = heat_cell(fw.x, sc.wc[0], sc.hm_wext, sc.hm_wbin, sc.hm_wc32[0], sc.hm_wext32, sc.hm_winv, sc.hm_bins);
        const int zi = heat_cell(fw.z, sc.wc[2], sc.hm_wext, sc.hm_wbin, sc.hm_wc32[1], sc.hm_wext32, sc.hm_winv, sc.hm_bins);
        if (xi >= 0 && zi >= 0) cell_add(cache, on, base, acc.heat_cls, cells, (uint32_t)(xi * sc.hm_bins + zi), c, acc.hw_lo, acc.hw_hi);
    }
    if (sf.x == sf.x) {
        const int xi = heat_cell(sf.x, sc.fc[0], sc.hm_fext, sc.hm_fbin, sc.hm_fc32[0], sc.hm_fext32, sc.hm_finv, sc.hm_bins);
        const int zi = heat_cell(sf.z, sc.fc[2], sc.hm_fext, sc.hm_fbin, sc.hm_fc32[1], sc.hm_fext32, sc.hm_finv, sc.hm_bins);
        if (xi >= 0 && zi >= 0)
            cell_add(cache, on, base + kClasses * cells, acc.heat_cls ? acc.heat_cls + (uint64_t)kClasses * cells : nullptr,
                     cells, (uint32_t)(xi * sc.hm_bins + zi), c, acc.hf_lo, acc.hf_hi);
    }
}

// MODE: kModeKnn (the reference's estimator without heatmaps, the hot path),
// kModeKnnAdjoint (k-NN with the Jacobian, and heatmaps when set), kModeRadius (fixed
// radius; Jacobian and heatmaps when their accumulators are set), kModeKnnHeat (k-NN with
// the sampled heatmaps, the reference's default). Separate instantiations keep code a run
// never executes out of its instruction stream: the kernel is bound by instruction issue
// and fetch.
constexpr int kModeKnn = 0, kModeKnnAdjoint = 1, kModeRadius = 2, kModeKnnHeat = 3;

// One query's k neighbours s.ci[0 .. k) of a planar map into the waveform (and Jacobian,
// heatmaps): Es, qb the query's energy, direction and time; rk the k-th distance.
template <int CHANNEL, int MODE, class J>
ALB_DEVICE void accumulate(const SceneDev& sc, const MapDev& m, const QueryDev& q, const Accum& acc, BinCache& bc, J& jc, int* err,
                           const WarpSmem& s, int k, uint64_t src, float Es, float4 qb, float rk) {
    const int l = lane_id();
    const float ts = qb.w;
    const float norm = 1.0f / (3.14159265358979f * rk * rk);
    // query-constant pieces
    float vinv = rsqrtf(fmaf(qb.x, qb.x, fmaf(qb.y, qb.y, qb.z * qb.z)));
    float vx = -qb.x * vinv, vy = -qb.y * vinv, vz = -qb.z * vinv;  // normalize(-d_query)
    float wconst = 0.f;
    if (CHANNEL == ALB_BOTTOM_REFLECTION) wconst = sc.floor_lambert * fmaxf(0.f, -qb.y);
    if (CHANNEL == ALB_SURFACE_TRANSMISSION_UP) wconst = sc.surface_lambert;
    float4 sq = make_float4(0.f, 0.f, 0.f, 0.f);
    if (MODE == kModeKnnAdjoint && q.s) sq = q.s[src];
    const bool jac_on = acc.nbins < kCachedBins;
    // the next neighbour's record is loaded while this one is weighted
    uint32_t idx_n = l < k ? s.ci[l] : 0u;
    float4 pb_n = make_float4(0.f, 0.f, 0.f, 0.f);
    float e_n = 0.f;
    if (l < k) {
        pb_n = m.b[idx_n];
        e_n = m.a[idx_n].w;
    }
#pragma unroll 1
    for (int j = l; j < k; j += 32) {
        const uint32_t idx = idx_n;
        const float4 pb = pb_n;
        const float Ep = e_n;
        if (j + 32 < k) {
            idx_n = s.ci[j + 32];
            pb_n = m.b[idx_n];
            e_n = m.a[idx_n].w;
        }
        float w;
        if (CHANNEL == ALB_BOTTOM_REFLECTION || CHANNEL == ALB_SURFACE_TRANSMISSION_UP) w = wconst;
        else w = ggx_weight(sc.ggx_a2, (float)sc.f0, -pb.x, -pb.y, -pb.z, vx, vy, vz);
        const float c = ((Es * Ep) * norm) * w;
        const int bin = (int)((ts + pb.w) / (float)sc.mult) - (int)sc.gate_lo;
        if (bin >= 0 && bin < acc.nbins) {
            bin_add(bc, acc, CHANNEL, bin, c);
            if (MODE == kModeKnnAdjoint && acc.jac_lo)
                jac_add<CHANNEL>(sc, m, acc, jc, jac_on, 0u, 0, bin, idx, c, sq, pb, vx, vy, vz);
        } else if (!sc.gated) {
            atomicCAS(err, 0, ALB_ERR_CAPACITY);
        }
    }
    if (MODE != kModeKnn && acc.hw_lo && m.fwi) {
        // accumulate_to_heatmap, alb_sim/math/accumulate_heatmap.py:6-61 (a separate,
        // non-unrolled pass: heatmaps are off in production runs)
#pragma unroll 1
        for (int j = l; j < k; j += 32) {
            const uint32_t idx = s.ci[j];
            const float4 pb = m.b[idx];
            float w;
            if (CHANNEL == ALB_BOTTOM_REFLECTION || CHANNEL == ALB_SURFACE_TRANSMISSION_UP) w = wconst;
            else w = ggx_weight(sc.ggx_a2, (float)sc.f0, -pb.x, -pb.y, -pb.z, vx, vy, vz);
            {
                NoCache none;
                heat_add(sc, m, acc, none, false, 0u, idx, ((Es * m.a[idx].w) * norm) * w);
            }
        }
    }
}

template <int CHANNEL, int MODE>
__global__ void __launch_bounds__(kGatherWarps * 32, kGatherBlocksPerSM) k_gather(SceneDev sc, MapDev m, QueryDev q, Accum acc, int k,
                                                              int* err, uint32_t kChunk, RadiusWork work) {
    __shared__ WarpSmem smem[kGatherWarps];
    __shared__ BinCache bc;
    __shared__ std::conditional_t<MODE == kModeKnnAdjoint, WordCache<512>, NoCache> jc;  // of acc.jac_cls
    cache_clear(jc);
    for (int i = threadIdx.x; i < kBinCache; i += blockDim.x) {
        bc.tag[i] = -1;
        for (int j = 0; j < 4; ++j) bc.w[j][i] = 0u;
    }
    __syncthreads();
    const int w = threadIdx.x >> 5, l = lane_id();
    WarpSmem& s = smem[w];
    const uint64_t warps = (uint64_t)gridDim.x * kGatherWarps;
    const bool second = MODE == kModeRadius && work.second;
    const uint64_t queries = second ? min(*work.count, work.cap) : q.n;  // or work items, one per chunk
    const uint64_t chunks = (queries + kChunk - 1) / kChunk;
    bool failed = false;
    // search counters accumulate in the warp's shared memory, not in registers held through
    // every search
    if (l < 4) s.st[l] = 0ull;
    __syncwarp();
    for (uint64_t ch = (uint64_t)blockIdx.x * kGatherWarps + w; ch < chunks && !failed; ch += warps) {
        const uint64_t q_end = min((ch + 1) * kChunk, queries);
        bool have_prev = false;  // s.ci[0 .. k) holds the previous query's neighbours
        for (uint64_t qi = ch * kChunk; qi < q_end; ++qi) {
            const uint2 item = second ? work.items[qi] : make_uint2(0u, kRoot);
            uint64_t src = second ? item.x : q.perm ? q.perm[qi] : qi;
            const float4 qa = q.a[src], qc = q.c[src];
            if (MODE == kModeRadius) {
                const float4 qb = q.b[src];
                const double qx = (double)qa.x + (double)qc.x, qy = (double)qa.y + (double)qc.y,
                             qz = (double)qa.z + (double)qc.z;
                // extension: every record within the fixed radius contributes at once
                KnnResult r;
                const float Es = qa.w, ts = qb.w;
                const float R = (float)sc.radius;
                const float norm = (CHANNEL == ALB_SCATTER) ? 1.0f / ((4.0f / 3.0f) * 3.14159265358979f * R * R * R)
                                                            : 1.0f / (3.14159265358979f * R * R);
                const float vinv = rsqrtf(fmaf(qb.x, qb.x, fmaf(qb.y, qb.y, qb.z * qb.z)));
                const float vx = -qb.x * vinv, vy = -qb.y * vinv, vz = -qb.z * vinv;
                float wconst = 0.f;
                if (CHANNEL == ALB_BOTTOM_REFLECTION) wconst = sc.floor_lambert * fmaxf(0.f, -qb.y);
                if (CHANNEL == ALB_SURFACE_TRANSMISSION_UP) wconst = sc.surface_lambert;
                const int layer = (CHANNEL == ALB_SCATTER) ? layer_of(sc, qy) : 0;
                const float4 sq = q.s ? q.s[src] : make_float4(0.f, 0.f, 0.f, 0.f);
                warp_radius_visit(m, s, work, (uint32_t)src, item.y, qx, qy, qz, qa.x, qa.y, qa.z, qc.x, qc.y, qc.z, sc.radius,
                    [&](uint32_t idx) {
                        const float4 pb = m.b[idx];
                        float w;
                        if (CHANNEL == ALB_BOTTOM_REFLECTION || CHANNEL == ALB_SURFACE_TRANSMISSION_UP) w = wconst;
                        else if (CHANNEL == ALB_SCATTER) w = scatter_weight(sc, layer, pb.x, pb.y, pb.z, vx, vy, vz);
                        else w = ggx_weight(sc.ggx_a2, (float)sc.f0, -pb.x, -pb.y, -pb.z, vx, vy, vz);
                        const float c = ((Es * m.a[idx].w) * norm) * w;
                        const int bin = (int)((ts + pb.w) / (float)sc.mult) - (int)sc.gate_lo;
                        if (bin >= 0 && bin < acc.nbins) {
                            bin_add(bc, acc, CHANNEL, bin, c);
                            if (acc.jac_lo) jac_add<CHANNEL>(sc, m, acc, jc, false, 0u, layer, bin, idx, c, sq, pb, vx, vy, vz);
                        } else if (!sc.gated) {
                            atomicCAS(err, 0, ALB_ERR_CAPACITY);
                        }
                        if (acc.hw_lo && m.fwi) heat_add(sc, m, acc, jc, false, 0u, idx, c);
                    },
                    r);
                if (r.fail) {
                    if (l == 0) atomicCAS(err, 0, r.fail);
                    failed = true;
                    break;
                }
                if (l == 0) {
                    s.st[0] += r.leaves;
                    s.st[1] += r.nodes;
                    s.st[3] += second ? 0 : 1;
                }
                if (q.rk_out && l == 0) q.rk_out[src] = sc.radius;
                __syncwarp();
                continue;
            }
            // k points lie within the farthest of the previous query's neighbours
            float bound = FLT_MAX;
            if (have_prev) {
                // the float32 screening error (below 2^-21) is far inside the 2^-14 inflation
                unsigned mx = 0u;
                float4 pn = l < k ? m.a[s.ci[l]] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1  // rolled: the kernel is bound by instruction fetch, and these loops run 4 times
                for (int j = l; j < k; j += 32) {
                    const float4 p = pn;
                    if (j + 32 < k) pn = m.a[s.ci[j + 32]];  // in flight during this neighbour
                    const float d = point_dist2(qa.x, qa.y, qa.z, qc.x, qc.y, qc.z, p);
                    mx = max(mx, __float_as_uint(d));  // non-negative floats order like their bits
                }
                const float t = __uint_as_float(__reduce_max_sync(0xffffffffu, mx)) * (1.f + 1.f / 16384.f);
                if (t < 1.0e37f) bound = t;
            }
            KnnResult r;
            if (!warp_knn<true, true>(m, s, k, 0.0, 0.0, 0.0, qa.x, qa.y, qa.z, qc.x, qc.y, qc.z, bound, m.b, r)) {
                if (l == 0) atomicCAS(err, 0, ALB_ERR_TOO_FEW);
                failed = true;
                break;
            }
            if (r.fail) {
                if (r.fail == kCrowded) {
                    leave_crowded(q, (uint32_t)src, CHANNEL);
                    have_prev = false;
                    if (l == 0) s.st[3] += 1;
                    continue;
                }
                // no valid neighbour set: report it and stop this warp's work
                if (l == 0) atomicCAS(err, 0, r.fail);
                failed = true;
                break;
            }
            // the query's direction and time are needed from here on
            const float4 qb = q.b[src];
            have_prev = true;
            if (q.rk_out && l == 0) q.rk_out[src] = sqrt(r.rk2);
            if (l == 0) {
                s.st[0] += r.leaves;
                s.st[1] += r.nodes;
                s.st[2] += r.selects;
                s.st[3] += 1;
            }
            accumulate<CHANNEL, MODE>(sc, m, q, acc, bc, jc, err, s, k, src, qa.w, qb, r.rkf);
            __syncwarp();
        }
    }
    if (l == 0) {
        if (q.stats && (s.st[3] || s.st[0])) {
            atomicAdd(q.stats + 0, s.st[0]);
            atomicAdd(q.stats + 1, s.st[1]);
            atomicAdd(q.stats + 2, s.st[2]);
            atomicAdd(q.stats + 3, s.st[3]);
        }
    }
    __syncthreads();
    bin_flush<CHANNEL>(bc, acc);
    cache_flush(jc, nullptr, 0u, acc.jac_cls);
}

// One query's k neighbours s.cp[0 .. k) into the waveform's class words (and Jacobian, heatmaps);
// qy the query's float64 depth, rk the k-th distance.
template <int CHANNEL, int MODE, class S, class J>
ALB_DEVICE void accumulate_run(const SceneDev& sc, const MapDev& m, const QueryDev& q, const Accum& acc, J& cache, bool on,
                               int* err, const S& s, int k, uint32_t src, float Es, float4 qb,
                               double qy, float rk) {
    constexpr bool volume = CHANNEL == ALB_SCATTER;
    const int l = lane_id();
    const float norm = volume ? 1.0f / ((4.0f / 3.0f) * 3.14159265358979f * rk * rk * rk)
                              : 1.0f / (3.14159265358979f * rk * rk);
    const float vinv = rsqrtf(fmaf(qb.x, qb.x, fmaf(qb.y, qb.y, qb.z * qb.z)));
    const float vx = -qb.x * vinv, vy = -qb.y * vinv, vz = -qb.z * vinv;  // normalize(-d_query)
    // WaterModel.scatter_energy picks the layer of the query depth (water.py:418-447)
    const int layer = volume && sc.n_layers > 1 ? layer_of(sc, qy) : 0;
    const float* wtab = sc.layer_weight[layer];
    const float binw = sc.layer_binw[layer], binw_inv = sc.layer_binw_inv[layer];
    float w = 0.f;
    if (CHANNEL == ALB_BOTTOM_REFLECTION) w = sc.floor_lambert * fmaxf(0.f, -qb.y);
    if (CHANNEL == ALB_SURFACE_TRANSMISSION_UP) w = sc.surface_lambert;
    const int gate = (int)sc.gate_lo;
    const uint32_t nbins = (uint32_t)acc.nbins;
    unsigned long long* cls = acc.cls;
    unsigned long long* wf_lo = acc.wf_lo + (uint64_t)CHANNEL * acc.nbins;
    unsigned long long* wf_hi = acc.wf_hi + (uint64_t)CHANNEL * acc.nbins;
    float4 sq = make_float4(0.f, 0.f, 0.f, 0.f);
    if (MODE == kModeKnnAdjoint && q.s) sq = q.s[src];
    // the next neighbour's record is loaded while this one is weighted
    float4 pb_n = make_float4(0.f, 0.f, 0.f, 0.f);
    if (l < k) pb_n = m.b[s.cp[l].x];
#pragma unroll 1
    for (int j = l; j < k; j += 32) {
        const float4 pb = pb_n;
        const uint2 cp = s.cp[j];
        if (j + 32 < k) pb_n = m.b[s.cp[j + 32].x];
        if (volume) {
            // scatter_bin with its division by a constant
            const float n = rsqrtf(fmaf(pb.x, pb.x, fmaf(pb.y, pb.y, pb.z * pb.z)));
            const float ca = fminf(fmaxf(fmaf(pb.x, vx, fmaf(pb.y, vy, pb.z * vz)) * n, -1.f), 1.f);
            const int a = min(max((int)div_by(acosf(ca) - kEps32, binw, binw_inv), 0), ALB_PHASE_DIVISIONS - 1);
            w = __ldg(wtab + a);
        }
        if (CHANNEL == ALB_SURFACE_REFLECTION) w = ggx_weight(sc.ggx_a2, (float)sc.f0, -pb.x, -pb.y, -pb.z, vx, vy, vz);
        const float c = ((Es * __uint_as_float(cp.y)) * norm) * w;
        const int bin = (int)div_by(qb.w + pb.w, sc.mult32, sc.mult32_inv) - gate;
        if ((uint32_t)bin < nbins) {
            class_add(cache, on, 0u, cls, nbins, (uint32_t)bin, c, wf_lo, wf_hi);
            if (MODE == kModeKnnAdjoint && acc.jac_lo)
                jac_add<CHANNEL>(sc, m, acc, cache, on, kClasses * nbins, layer, bin, cp.x, c, sq, pb, vx, vy, vz);
        } else if (!sc.gated) {
            atomicCAS(err, 0, ALB_ERR_CAPACITY);
        }
        if (MODE != kModeKnn && acc.hw_lo && m.fwi) {
            if constexpr (MODE == kModeKnnHeat) {
                heat_add(sc, m, acc, cache, on, kClasses * nbins, cp.x, c);
            } else {
                NoCache none;
                heat_add(sc, m, acc, none, false, 0u, cp.x, c);
            }
        }
    }
}

// s.ci to s.cp, which overlay each other: the last 32 first.
template <class S>
ALB_DEVICE void pack_neighbours(const MapDev& m, S& s, int k) {
    for (int j = (k - 1) / 32 * 32 + lane_id(); j >= 0; j -= 32) {
        uint2 c = make_uint2(0u, 0u);
        if (j < k) {
            c.x = s.ci[j];
            c.y = __float_as_uint(m.a[c.x].w);
        }
        __syncwarp();
        if (j < k) s.cp[j] = c;
        __syncwarp();
    }
}

// The search of one query alone, out of line: the grouped kernel takes it for the first query of
// a CTA, runs whose list does not fit, guesses that fail and near ties, 1-3% of the queries,
// and its code and registers stay out of the hot loop. The k neighbours are left
// in s.cp. bound < 0: it holds k points to take one from. For planes with double-float distances, as in k_gather: around a
// dense spot more records lie within float32's margin of a far query's k-th distance than the buffer holds (the same
// times with and without on the large scene). A crowded query is left here, with k of its candidates and an infinite
// k-th distance: what the caller then adds for it is zero. A branch for it in the caller's loop cost the adjoint's
// scatter gather 6% (12.6 -> 13.4 ms).
template <int CHANNEL, class S>
__device__ __noinline__ bool cold_knn(const MapDev& m, S& s, int k, float fx, float fy, float fz, float lx, float ly,
                                      float lz, float bound, KnnResult& res, const QueryDev& q, uint32_t src) {
    if (bound < 0.f) {
        // k points lie within the farthest of them; the float32 screening error (below 2^-21) is far
        // inside the 2^-14 inflation
        unsigned mx = 0u;
#pragma unroll 1
        for (int j = lane_id(); j < k; j += 32)
            mx = max(mx, __float_as_uint(point_dist2(fx, fy, fz, lx, ly, lz, m.a[s.cp[j].x])));
        const float t = __uint_as_float(__reduce_max_sync(0xffffffffu, mx)) * (1.f + 1.f / 16384.f);
        bound = t < 1.0e37f ? t : FLT_MAX;
    }
    if (!warp_knn<CHANNEL != ALB_SCATTER, true>(m, s, k, 0.0, 0.0, 0.0, fx, fy, fz, lx, ly, lz, bound, m.b, res)) return false;
    if (res.fail == kCrowded) {
        leave_crowded(q, src, CHANNEL);
        res.fail = 0;
        res.rk2 = -1.0;
        res.rkf = __int_as_float(0x7f800000);
    }
    if (!res.fail) pack_neighbours(m, s, k);
    return true;
}

// Queries far from a planar map (a receiver's footprint wider than the beam's spot) have all their
// neighbours at its near edge, and the ball of a guess holds most of the map: where a query's leaf list
// does not fit, the next ones are searched alone at once, twice as many after each list in a row that does
// not fit, up to this many.
constexpr int kAlone = 64;

// Gather of the k nearest by runs of neighbouring queries (gather_group.cuh). One CTA per SM.
// The sorted queries are cut into segments that CTAs take in turn: the first half of them in
// a few per CTA, half of the rest in as many, and so on (ScatterPlan), since the work of a
// range varies with the density of the map around it: with one range per SM the slowest of 152 SMs
// issued 19% more than the mean, 27.5 against 22.9 ms at 1e6 photons of the large scene. A segment is
// 16 to 64 chunks; the CTA's warps fetch chunks in turn. Two segments per CTA and level below 2^24 queries,
// four above: scatter gather of 6.2e5 queries (default scene) 3.7 and 3.9 ms, 1.7e6 (a scene of the
// sweep) 5.0 and 5.3, 8.7e6 22.1 and 22.3, 8.7e7 229 and 225.
struct ScatterPlan {
    uint64_t first, n;  // the launch's range of the sorted queries
    uint32_t pieces;    // segments per level
    int levels;         // level L holds half of what the levels before it left, the last one the rest
    int chunk_bits;     // a segment is 2^chunk_bits chunks
    bool cached;        // class words go through the CTA's cache, where it has one
    uint32_t* ticket;   // segments taken, zero at the launch
};
constexpr uint64_t kManyQueries = 1ull << 24;
constexpr int kSegBits = 6;  // 64 chunks in a segment, fewer for few queries
constexpr int kSegRing = 64;  // segments of a CTA whose numbers are kept

ALB_DEVICE void segment_range(const ScatterPlan& p, uint32_t g, uint64_t& s0, uint64_t& s1) {
    const uint32_t lev = g / p.pieces, j = g % p.pieces;
    const uint64_t left = p.n >> lev;
    const uint64_t m = (int)lev == p.levels - 1 ? left : left - (p.n >> (lev + 1));
    const uint64_t base = p.first + (p.n - left);
    s0 = base + m * j / p.pieces;
    s1 = base + m * (j + 1) / p.pieces;
}

// SLOTS: slots of the cache of class words, 0: none. LOW: queries have low parts (else lo_zero).
template <int CHANNEL, int MODE, int CAP, int WARPS, int SLOTS, bool LOW>
__global__ void __launch_bounds__(WARPS * 32, 1)
    k_gather_runs(const __grid_constant__ SceneDev sc, const __grid_constant__ MapDev m,
                     const __grid_constant__ QueryDev q, const __grid_constant__ Accum acc, int k, int* err,
                     const __grid_constant__ ScatterPlan plan) {
    extern __shared__ __align__(16) unsigned char group_raw[];
    using S = GroupSmem<CAP>;
    using G = std::conditional_t<CHANNEL == ALB_SCATTER, VolumeRuns, PlaneRuns>;
    S* smem = reinterpret_cast<S*>(group_raw);
    __shared__ uint32_t next;  // the CTA's next chunk
    __shared__ float last2;    // squared k-th distance of some query just answered (a chunk's first guess)
    // (the CTA's segment number << 32) | its global number; a segment's number is fetched by the
    // warp that takes the first chunk of the one before it
    __shared__ unsigned long long ring[kSegRing];
    // class words: the waveform's, then the Jacobian's or the heatmaps'
    using Cache = std::conditional_t<SLOTS != 0, WordCache<SLOTS>, NoCache>;
    __shared__ Cache cache;
    cache_clear(cache);
    if (threadIdx.x < kSegRing) ring[threadIdx.x] = ~0ull;
    __syncthreads();
    if (threadIdx.x == 0) {
        next = 0u;
        last2 = -1.f;
        ring[0] = atomicAdd(plan.ticket, 1u);
    }
    __syncthreads();
    const int w = threadIdx.x >> 5, l = lane_id();
    S& s = smem[w];
    const uint32_t segments = plan.pieces * (uint32_t)plan.levels, chunks = 1u << plan.chunk_bits;
    const float side_rk = G::side((float)k);
    bool failed = false;
    if (l < 4) s.st[l] = 0ull;
    if (l == 0) {
        s.alone = 0;
        s.streak = 1;
    }
    __syncwarp();
    while (!failed) {
        uint32_t t = 0u, g = 0u;
        if (l == 0) {
            t = atomicAdd(&next, 1u);
            const uint32_t seg = t >> plan.chunk_bits;
            volatile unsigned long long* v = ring;
            if ((t & (chunks - 1u)) == 0u) v[(seg + 1) % kSegRing] = (unsigned long long)(seg + 1) << 32 | atomicAdd(plan.ticket, 1u);
            // published a segment (16 to 64 chunks) ago; the bound only guards against a lost slot
            unsigned long long e = v[seg % kSegRing];
            for (int wait = 0; (uint32_t)(e >> 32) != seg && wait < (1 << 20); ++wait) e = v[seg % kSegRing];
            if ((uint32_t)(e >> 32) != seg) atomicCAS(err, 0, ALB_ERR_ITER_CAP);
            g = (uint32_t)(e >> 32) == seg ? (uint32_t)e : 0xffffffffu;
        }
        t = __shfl_sync(0xffffffffu, t, 0) & (chunks - 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= segments) break;
        uint64_t s0, s1;
        segment_range(plan, g, s0, s1);
        const uint64_t c0 = s0 + ((s1 - s0) * t >> plan.chunk_bits), q_end = s0 + ((s1 - s0) * (t + 1) >> plan.chunk_bits);
        if (c0 == q_end) continue;
        QueryRun run{0, 0, 0, 0.f};
        uint64_t r_base = 0;  // first query of the run the lanes hold
        uint32_t gsrc = 0u;   // this lane's query of the run: index and position
        float gx = 0.f, gy = 0.f, gz = 0.f;
        // squared k-th distance of the previous query; a chunk starts from the CTA's latest
        float prev2 = *reinterpret_cast<volatile float*>(&last2);
        for (uint64_t qi = c0; qi < q_end; ++qi) {
            // the guess, the whole list, then lists of 1.25 times the radius for this query
            float thr = prev2 * G::kGuess2;
            bool fresh = qi >= r_base + run.take || !(thr <= run.T2);
            float fx, fy, fz, lx = 0.f, ly = 0.f, lz = 0.f, kth = 0.f, rk, d2;
            uint32_t src, kid = 0u;
            int got = 0, leaves = 0;
#pragma unroll 1
            for (int tries = 0;; ++tries) {
                bool listed = prev2 > 0.f;
                if (fresh) {
                    const int avail = (int)min(q_end - qi, (uint64_t)32);
                    r_base = qi;
                    float la = 0.f;
                    if (l < avail) {
                        gsrc = q.perm ? q.perm[qi + l] : (uint32_t)(qi + l);
                        const float4 a = q.a[gsrc];
                        gx = a.x; gy = a.y; gz = a.z;
                        if (LOW && !q.lo_zero) {
                            const float4 c = q.c[gsrc];
                            la = fmaxf(fabsf(c.x), fmaxf(fabsf(c.y), fabsf(c.z)));
                        }
                    }
                    run.take = 1;
                    run.nodes = 0;
                    if (CHANNEL != ALB_SCATTER && s.alone > 0) {
                        listed = false;
                        __syncwarp();
                        if (l == 0) --s.alone;
                    } else if (listed) {
                        listed = build_run<G>(m, s, avail, gx, gy, gz, la, prev2, side_rk * sqrtf(prev2), run);
                        if (CHANNEL != ALB_SCATTER && l == 0) {
                            s.alone = listed ? 0 : s.streak;
                            s.streak = listed ? 1 : min(2 * s.streak, kAlone);
                        }
                    }
                    if (l == 0) s.st[1] += run.nodes;
                }
                const int at = (int)(qi - r_base);
                src = __shfl_sync(0xffffffffu, gsrc, at);
                fx = __shfl_sync(0xffffffffu, gx, at);
                fy = __shfl_sync(0xffffffffu, gy, at);
                fz = __shfl_sync(0xffffffffu, gz, at);
                if (LOW && !q.lo_zero) {
                    const float4 c = q.c[src];
                    lx = c.x; ly = c.y; lz = c.z;
                }
                if (!listed) break;
                got = run_search<G>(m, s, k, run.n, fx, fy, fz, lx, ly, lz, thr, kth, kid, leaves);
                if (got != 0 || tries == 6) break;
                if (l == 0 && q.retries) atomicAdd(q.retries, 1ull);
                fresh = !(thr < run.T2);
                if (fresh) prev2 = run.T2;
                thr = fresh ? prev2 * G::kList2 : run.T2;
            }
            if (got == 1) {
                rk = dist_f32(fx, fy, fz, lx, ly, lz, m.a[kid], d2);
                if (q.rk_out && l == 0)
                    q.rk_out[src] = sqrt(point_dist2_f64((double)fx + (double)lx, (double)fy + (double)ly,
                                                         (double)fz + (double)lz, m.a[kid]));
                if (l == 0) {
                    s.st[0] += leaves;
                    s.st[2] += 1;
                    s.st[3] += 1;
                }
            } else {
                // a proven k-th distance bounds the search, or, while s.cp still holds them, the previous
                // query's neighbours; the run's boxes share its scratch
                const float bound = got < 0 && kth > 0.f ? kth * (1.f + 1.f / 16384.f)
                                    : leaves == 0 && s.st[3] ? -1.f : FLT_MAX;
                run.take = 0;
                KnnResult r;
                const bool enough = cold_knn<CHANNEL>(m, s, k, fx, fy, fz, lx, ly, lz, bound, r, q, src);
                if (!enough || r.fail) {  // no valid neighbour set: report it and stop this warp's work
                    if (l == 0) atomicCAS(err, 0, enough ? r.fail : ALB_ERR_TOO_FEW);
                    failed = true;
                    break;
                }
                rk = r.rkf;
                d2 = (float)r.rk2;
                if (q.rk_out && l == 0) q.rk_out[src] = sqrt(r.rk2);
                if (l == 0) {
                    s.st[0] += r.leaves;
                    s.st[1] += r.nodes;
                    s.st[2] += r.selects;
                    s.st[3] += 1;
                }
            }
            prev2 = d2;
            const float4 qb = q.b[src];
            accumulate_run<CHANNEL, MODE>(sc, m, q, acc, cache, plan.cached, err, s, k, src, q.a[src].w, qb, (double)fy + (double)ly, rk);
            __syncwarp();
        }
        if (l == 0) last2 = prev2;
    }
    if (l == 0) {
        if (q.stats && s.st[3]) {
            atomicAdd(q.stats + 0, s.st[0]);
            atomicAdd(q.stats + 1, s.st[1]);
            atomicAdd(q.stats + 2, s.st[2]);
            atomicAdd(q.stats + 3, s.st[3]);
        }
    }
    if constexpr (SLOTS != 0) {
        __syncthreads();
        cache_flush(cache, acc.cls, kClasses * (uint32_t)acc.nbins,
                    MODE == kModeKnnAdjoint ? acc.jac_cls : acc.heat_cls);
    }
}

// The queries that this channel's gather left (kCrowded): the k nearest under any number of ties, and their sums.
// A warp looks at 32 queries' marks at a time. One mode: what it sums is decided by the accumulators it is given.
constexpr int kCrowdedWarps = 4;
template <int CHANNEL>
__global__ void __launch_bounds__(kCrowdedWarps * 32) k_gather_crowded(const __grid_constant__ SceneDev sc, const __grid_constant__ MapDev m,
                                                                       const __grid_constant__ QueryDev q,
                                                                       const __grid_constant__ Accum acc, int k, int* err,
                                                                       uint64_t first, uint64_t end) {
    __shared__ GroupSmem<448> smem[kCrowdedWarps];
    const int w = threadIdx.x >> 5, l = lane_id();
    GroupSmem<448>& s = smem[w];
    NoCache none;
    if (l < 4) s.st[l] = 0ull;
    __syncwarp();
    const uint64_t step = 32ull * gridDim.x * kCrowdedWarps;
    for (uint64_t base = first + 32ull * ((uint64_t)blockIdx.x * kCrowdedWarps + w); base < end; base += step) {
        const bool left = base + l < end && (__float_as_uint(q.c[base + l].w) >> CHANNEL & 1u);
        for (unsigned todo = __ballot_sync(0xffffffffu, left); todo; todo &= todo - 1u) {
            const uint32_t src = (uint32_t)(base + __ffs(todo) - 1);
            const float4 qa = q.a[src], qc = q.c[src];
            const double qx = (double)qa.x + (double)qc.x, qy = (double)qa.y + (double)qc.y, qz = (double)qa.z + (double)qc.z;
            const KnnResult r = crowded_knn(m, s, k, qx, qy, qz, m.b);
            if (r.fail) {
                if (l == 0) atomicCAS(err, 0, r.fail);
                continue;
            }
            pack_neighbours(m, s, k);
            if (q.rk_out && l == 0) q.rk_out[src] = sqrt(r.rk2);
            if (l == 0) {
                s.st[0] += r.leaves;
                s.st[1] += r.nodes;
                s.st[2] += r.selects;
                s.st[3] += 1;
            }
            accumulate_run<CHANNEL, kModeKnnAdjoint>(sc, m, q, acc, none, false, err, s, k, src, qa.w, q.b[src], qy, r.rkf);
            __syncwarp();
        }
    }
    // (the gathers counted these queries when they left them)
    if (l < 3 && q.stats && s.st[3]) atomicAdd(q.stats + l, s.st[l]);
    if (l == 0 && s.st[3]) atomicAdd(q.n_crowded, s.st[3]);
}

// One query's k neighbours s.ci[0 .. k) in order of (float64 distance, index), as out_idx / out_dist
// rows of k. Every distance is formed once and ranked as its bit pattern against the others in
// shared memory (non-negative doubles order like integers): comparing k x k freshly formed
// distances took 4400 FP64 instructions per query at k = 100, at two FP64 lanes per SM and cycle.
// tag: the index to report for a position (nullptr: the position itself).
template <class P>
ALB_DEVICE void write_sorted(const P& pts, WarpSmem& s, int k, double qx, double qy, double qz, const float4* tag,
                             int32_t* out_idx, double* out_dist) {
    const int l = lane_id();
    static_assert(sizeof(s.stk) + sizeof(s.stk_d) >= 256 * sizeof(uint64_t), "the bit patterns lie in the stack");
    uint64_t* bits = reinterpret_cast<uint64_t*>(s.stk);
    for (int j = l; j < k; j += 32)
        bits[j] = (uint64_t)__double_as_longlong(point_dist2_f64(qx, qy, qz, pts.at(s.ci[j])));
    __syncwarp();
    int sum = 0;
    for (int j0 = 0; j0 < k; j0 += 128) {
        uint64_t own[4];
        int rank[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 4; ++i) own[i] = j0 + i * 32 + l < k ? bits[j0 + i * 32 + l] : 0ull;
#pragma unroll 2
        for (int t = 0; t < k; ++t) {
            const uint64_t o = bits[t];
#pragma unroll
            for (int i = 0; i < 4; ++i) rank[i] += o < own[i] ? 1 : 0;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = j0 + i * 32 + l;
            if (j < k) {
                sum += rank[i];
                s.cd[j] = __int_as_float(rank[i]);
            }
        }
    }
    __syncwarp();
    // equal distances leave the ranks short of 0 .. k - 1: rank those by index too
    if (__reduce_add_sync(0xffffffffu, sum) != k * (k - 1) / 2) {
        for (int j = l; j < k; j += 32) {
            int extra = 0;
            for (int t = 0; t < k; ++t) extra += bits[t] == bits[j] && s.ci[t] < s.ci[j] ? 1 : 0;
            s.cd[j] = __int_as_float(__float_as_int(s.cd[j]) + extra);
        }
    }
    for (int j = l; j < k; j += 32) {
        const uint32_t idx = s.ci[j];
        const int rank = __float_as_int(s.cd[j]);
        out_idx[rank] = tag ? (int32_t)__float_as_uint(tag[idx].w) : (int32_t)idx;
        out_dist[rank] = sqrt(__longlong_as_double((long long)bits[j]));
    }
    __syncwarp();
}

// A query without an answer gets index -1 and distance NaN in all its k slots, so no slot is left
// holding whatever the caller's buffer held before.
ALB_DEVICE void write_failed(int k, int32_t* out_idx, double* out_dist) {
    for (int j = lane_id(); j < k; j += 32) {
        out_idx[j] = -1;
        out_dist[j] = __longlong_as_double(0x7ff8000000000000ll);
    }
    __syncwarp();
}

constexpr int32_t kLeft = -2;  // a crowded query's first index, until its answer replaces it

// Standalone KDTree.query(x, k): sorted indices (the w lanes of the map's records) and float64
// distances. Queries go in `perm` order, `chunk` consecutive ones per warp, each bounded by the
// farthest of its predecessor's neighbours.
__global__ void __launch_bounds__(kGatherWarps * 32, kGatherBlocksPerSM)
    k_knn(MapDev m, const double* __restrict__ qs, const uint32_t* __restrict__ perm, uint64_t nq, uint32_t chunk, int k,
          int32_t* out_idx, double* out_dist, int* err, uint32_t* crowded) {
    __shared__ WarpSmem smem[kGatherWarps];
    const int w = threadIdx.x >> 5, l = lane_id();
    WarpSmem& s = smem[w];
    const uint64_t warps = (uint64_t)gridDim.x * kGatherWarps;
    const uint64_t chunks = (nq + chunk - 1) / chunk;
    for (uint64_t ch = (uint64_t)blockIdx.x * kGatherWarps + w; ch < chunks; ch += warps) {
        const uint64_t q_end = min((ch + 1) * chunk, nq);
        bool have_prev = false;
        for (uint64_t i = ch * chunk; i < q_end; ++i) {
            const uint64_t qi = perm[i];
            const double qx = qs[3 * qi], qy = qs[3 * qi + 1], qz = qs[3 * qi + 2];
            const float fx = (float)qx, fy = (float)qy, fz = (float)qz;
            const float lx = (float)(qx - (double)fx), ly = (float)(qy - (double)fy), lz = (float)(qz - (double)fz);
            float bound = FLT_MAX;
            if (have_prev) {
                unsigned mx = 0u;
                for (int j = l; j < k; j += 32)
                    mx = max(mx, __float_as_uint(point_dist2(fx, fy, fz, lx, ly, lz, m.a[s.ci[j]])));
                const float t = __uint_as_float(__reduce_max_sync(0xffffffffu, mx)) * (1.f + 1.f / 16384.f);
                if (t < 1.0e37f) bound = t;
            }
            KnnResult r;
            int why = 0;
            if (!warp_knn<true>(m, s, k, qx, qy, qz, fx, fy, fz, lx, ly, lz, bound, nullptr, r)) why = ALB_ERR_TOO_FEW;
            else if (r.fail) why = r.fail;
            have_prev = !why;
            if (why == kCrowded) {
                if (l == 0) {
                    out_idx[qi * k] = kLeft;
                    atomicOr(crowded, 1u);
                }
                __syncwarp();
                continue;
            }
            if (why) {
                if (l == 0) atomicCAS(err, 0, why);
                write_failed(k, out_idx + qi * k, out_dist + qi * k);
                continue;
            }
            write_sorted(MapPoints{m.a}, s, k, qx, qy, qz, m.a, out_idx + qi * k, out_dist + qi * k);
        }
    }
}

// The queries that k_knn left.
__global__ void __launch_bounds__(kCrowdedWarps * 32) k_knn_crowded(const __grid_constant__ MapDev m, const double* __restrict__ qs,
                                                                    uint64_t nq, int k, int32_t* out_idx, double* out_dist,
                                                                    int* err) {
    __shared__ WarpSmem smem[kCrowdedWarps];
    const int w = threadIdx.x >> 5, l = lane_id();
    WarpSmem& s = smem[w];
    const uint64_t step = 32ull * gridDim.x * kCrowdedWarps;
    for (uint64_t base = 32ull * ((uint64_t)blockIdx.x * kCrowdedWarps + w); base < nq; base += step) {
        const bool left = base + l < nq && out_idx[(base + l) * k] == kLeft;
        for (unsigned todo = __ballot_sync(0xffffffffu, left); todo; todo &= todo - 1u) {
            const uint64_t qi = base + __ffs(todo) - 1;
            const double qx = qs[3 * qi], qy = qs[3 * qi + 1], qz = qs[3 * qi + 2];
            const int fail = crowded_knn(m, s, k, qx, qy, qz, nullptr).fail;
            if (fail) {
                if (l == 0) atomicCAS(err, 0, fail);
                write_failed(k, out_idx + qi * k, out_dist + qi * k);
                continue;
            }
            write_sorted(MapPoints{m.a}, s, k, qx, qy, qz, m.a, out_idx + qi * k, out_dist + qi * k);
        }
    }
}

// The k nearest of at most a few thousand points float[3 m] by screening all of them, one warp per
// query: no index, no scratch memory, one launch. At 4096 points the 128 screening steps cost what
// a walk over a tree does, and the tree's one-CTA build cost 0.8 ms on top.
constexpr int kBruteWarps = 4;

// One query (TIES as in warp_knn): 0, or ALB_ERR_INVALID (fewer than k points admitted) or kCrowded.
template <bool TIES>
ALB_DEVICE int brute_knn(PackedPoints pp, uint32_t m, WarpSmem& s, int k, double qx, double qy, double qz) {
    const int l = lane_id();
    const float fx = (float)qx, fy = (float)qy, fz = (float)qz;
    const float lx = (float)(qx - (double)fx), ly = (float)(qy - (double)fy), lz = (float)(qz - (double)fz);
    float thr = FLT_MAX;
    int cnt = 0;
    constexpr int kAhead = 4;  // steps whose points are loaded together
    for (uint32_t r0 = 0; r0 < m; r0 += 32 * kAhead) {
        float4 p[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const uint32_t r = r0 + i * 32 + l;
            p[i] = r < m ? pp.at(r) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const uint32_t r = r0 + i * 32 + l;
            const float d = point_dist2(fx, fy, fz, lx, ly, lz, p[i]);
            const bool take = r < m && d <= thr;
            const unsigned b = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int pos = cnt + __popc(b & lanemask_lt());
                float hi, lo;
                point_dist2_df(fx, fy, fz, lx, ly, lz, p[i], hi, lo);
                s.ci[pos] = r;
                s.cd[pos] = hi;
                s.cl[pos] = frac16(hi, lo);
            }
            cnt += __popc(b);
            __syncwarp();
            if (cnt >= k && (thr == FLT_MAX || cnt > kCap - 32)) {
                // refined distances within one float32 ulp of the k-th can still rank
                const float kth = warp_kth32(s, 0, cnt, k);
                thr = fminf(thr, kth * (1.0f + 2.0f * kRelMargin));
                cnt = warp_compact(s, cnt, __uint_as_float(__float_as_uint(kth) + 1u));
                if (cnt > kCap - 32) {  // more near ties than there is room for: the k best so far are enough
                    if (!TIES) return kCrowded;
                    keep_nearest(pp, s, 0, cnt, k, qx, qy, qz, nullptr);
                    cnt = k;
                }
            }
        }
    }
    if (cnt < k) return ALB_ERR_INVALID;
    // select_refined ranks the near ties on their float64 distances
    int fail = 0;
    select_refined<TIES>(pp, s, 0, cnt, k, qx, qy, qz, nullptr, fail);
    return fail;
}

__device__ __noinline__ int crowded_brute(PackedPoints pp, uint32_t m, WarpSmem& s, int k, double qx, double qy, double qz) {
    return brute_knn<true>(pp, m, s, k, qx, qy, qz);
}

__global__ void __launch_bounds__(kBruteWarps * 32, 8) k_knn_brute(const float* __restrict__ pts, uint32_t m,
                                                                   const double* __restrict__ qs, uint64_t nq, int k,
                                                                   int32_t* out_idx, double* out_dist) {
    __shared__ WarpSmem smem[kBruteWarps];
    WarpSmem& s = smem[threadIdx.x >> 5];
    const PackedPoints pp{pts};
    const uint64_t q0 = (uint64_t)blockIdx.x * kBruteWarps + (threadIdx.x >> 5), step = (uint64_t)gridDim.x * kBruteWarps;
    bool crowded = false;
    for (uint64_t qi = q0; qi < nq; qi += step) {
        const double qx = qs[3 * qi], qy = qs[3 * qi + 1], qz = qs[3 * qi + 2];
        const int fail = brute_knn<false>(pp, m, s, k, qx, qy, qz);
        if (!fail) {
            write_sorted(pp, s, k, qx, qy, qz, nullptr, out_idx + qi * k, out_dist + qi * k);
        } else {
            crowded = crowded || fail == kCrowded;
            write_failed(k, out_idx + qi * k, out_dist + qi * k);
            if (fail == kCrowded && lane_id() == 0) out_idx[qi * k] = kLeft;
            __syncwarp();
        }
    }
    if (!crowded) return;
    // the caller's stream may be under capture, so these queries have no launch of their own
    for (uint64_t qi = q0; qi < nq; qi += step) {
        int32_t first = 0;
        if (lane_id() == 0) first = out_idx[qi * k];
        if (__shfl_sync(0xffffffffu, first, 0) != kLeft) continue;
        const double qx = qs[3 * qi], qy = qs[3 * qi + 1], qz = qs[3 * qi + 2];
        if (crowded_brute(pp, m, s, k, qx, qy, qz)) write_failed(k, out_idx + qi * k, out_dist + qi * k);
        else write_sorted(pp, s, k, qx, qy, qz, nullptr, out_idx + qi * k, out_dist + qi * k);
    }
}

// The same for many queries of few neighbours: one query per lane, a block's points in shared memory, two passes over
// them. The first finds the k-th smallest screening distance, the second ranks every point within its margin
// by (float64 distance, index), any number of ties included. Bound by issue: a dozen instructions for a point
// and 32 queries in each pass, and the insertions, which lanes make one at a time.
constexpr int kLaneThreads = 128, kLanePoints = 1024;
template <int K>
__global__ void __launch_bounds__(kLaneThreads) k_knn_lanes(const float* __restrict__ pts, uint32_t m, const double* __restrict__ qs,
                                                            uint64_t nq, int k, int32_t* out_idx, double* out_dist) {
    __shared__ float4 tile[kLanePoints];
    const uint64_t qi = blockIdx.x * (uint64_t)kLaneThreads + threadIdx.x;
    const bool on = qi < nq;
    const double qx = on ? qs[3 * qi] : 0.0, qy = on ? qs[3 * qi + 1] : 0.0, qz = on ? qs[3 * qi + 2] : 0.0;
    const float fx = (float)qx, fy = (float)qy, fz = (float)qz;
    const float lx = (float)(qx - (double)fx), ly = (float)(qy - (double)fy), lz = (float)(qz - (double)fz);
    // visit(number, position) for every point, by all threads
    auto each_point = [&](auto&& visit) {
        for (uint32_t r0 = 0; r0 < m; r0 += kLanePoints) {
            const uint32_t n = min(m - r0, (uint32_t)kLanePoints);
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < n; i += kLaneThreads) tile[i] = PackedPoints{pts}.at(r0 + i);
            __syncthreads();
#pragma unroll 4
            for (uint32_t i = 0; i < n; ++i) visit(r0 + i, tile[i]);
        }
    };
    float v[K];
#pragma unroll
    for (int j = 0; j < K; ++j) v[j] = FLT_MAX;
    each_point([&](uint32_t, float4 p) {
        const float d = point_dist2(fx, fy, fz, lx, ly, lz, p);
        if (K == 1) {
            v[0] = fminf(v[0], d);  // (a NaN is passed over)
        } else if (d < v[K - 1]) {
            v[K - 1] = d;
#pragma unroll
            for (int j = K - 1; j > 0; --j) {
                const float a = fminf(v[j - 1], v[j]), b = fmaxf(v[j - 1], v[j]);
                v[j - 1] = a;
                v[j] = b;
            }
        }
    });
    float kth = FLT_MAX;
#pragma unroll
    for (int j = 0; j < K; ++j) kth = j == k - 1 ? v[j] : kth;
    const bool found = kth < FLT_MAX;
    const float thr = found ? kth * (1.0f + 2.0f * kRelMargin) : -1.f;
    uint64_t e[K];
    uint32_t id[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        e[j] = ~0ull;
        id[j] = 0u;
    }
    each_point([&](uint32_t r, float4 p) {
        if (!(point_dist2(fx, fy, fz, lx, ly, lz, p) <= thr)) return;
        uint64_t d = (uint64_t)__double_as_longlong(point_dist2_f64(qx, qy, qz, p));
        uint32_t i = r;
        // points come in order of their numbers: behind its equals, the ones after it one place on
        bool in = false;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            in = in || d < e[j];
            if (in) {
                const uint64_t t = e[j];
                const uint32_t u = id[j];
                e[j] = d;
                id[j] = i;
                d = t;
                i = u;
            }
        }
    });
    if (!on) return;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        if (j < k) {
            out_idx[qi * k + j] = found ? (int32_t)id[j] : -1;
            out_dist[qi * k + j] = found ? sqrt(__longlong_as_double((long long)e[j])) : __longlong_as_double(0x7ff8000000000000ll);
        }
    }
}

static int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

static unsigned gather_blocks(uint64_t nq) {
    uint64_t want = (nq + kGatherWarps - 1) / kGatherWarps;
    uint64_t cap = (uint64_t)sm_count() * 16;
    return (unsigned)(want < cap ? (want ? want : 1) : cap);
}

// Consecutive queries per warp: as many as the resident warps need to take every query in one
// wave, within [kQueryChunkMin, kQueryChunk]. With 64 whatever the count,
// 25 000 queries ran on 391 of the 4864 resident warps and took as long as 250 000 (bottom
// gather 1.67 ms; with chunks of 6, 0.24 ms); 5000 queries take 0.07 ms at a floor of 2, 0.12
// at 4, 0.21 at 8. The fixed-radius gather carries nothing from query to query and its visits
// differ by four orders of magnitude between neighbouring queries: one query at a time (surface
// gather of 25 000 queries at 0.5 m: 22.3 -> 13.1 ms).
static uint32_t query_chunk(uint64_t nq, bool radius) {
    if (radius) return 1;
    const uint64_t warps = (uint64_t)sm_count() * kGatherBlocksPerSM * kGatherWarps;
    const uint64_t fit = (nq + warps - 1) / warps;
    return (uint32_t)std::min<uint64_t>(kQueryChunk, std::max<uint64_t>(fit, kQueryChunkMin));
}

// The class words that a gather of `channel` filled (waveform: gathers by runs and of crowded queries only).
static void merge_classes(const SceneDev& sc, const Accum& acc, int channel, bool waveform, cudaStream_t st) {
    const uint32_t nb = (uint32_t)acc.nbins;
    const unsigned blocks = (nb + 255u) / 256u;
    if (waveform) {
        k_merge_classes<<<blocks, 256, 0, st>>>(acc.cls, nb, acc.wf_lo + (uint64_t)channel * nb,
                                                acc.wf_hi + (uint64_t)channel * nb, 0, 0);
        note_launch();
    }
    if (acc.jac_lo && acc.jac_cls) {
        k_merge_classes<<<dim3(blocks, kJacParams), 256, 0, st>>>(acc.jac_cls, nb, acc.jac_lo + (uint64_t)channel * nb,
                                                                  acc.jac_hi + (uint64_t)channel * nb,
                                                                  (uint64_t)kClasses * nb, (uint64_t)ALB_CHANNELS * nb);
        note_launch();
    }
    if (acc.hw_lo && acc.heat_cls) {
        // the two maps' words lie 2 cells apart: hw_lo, hw_hi, hf_lo, hf_hi
        const uint32_t cells = (uint32_t)(sc.hm_bins * sc.hm_bins);
        k_merge_classes<<<dim3((cells + 255u) / 256u, 2), 256, 0, st>>>(acc.heat_cls, cells, acc.hw_lo, acc.hw_hi,
                                                                        (uint64_t)kClasses * cells, (uint64_t)2 * cells);
        note_launch();
    }
}

template <int CHANNEL, int MODE, int CAP, int WARPS, int SLOTS, bool LOW = true>
static void launch_runs(const SceneDev& sc, const MapDev& map, const QueryDev& q, const Accum& acc, int k, int* err,
                           cudaStream_t st) {
    constexpr int bytes = WARPS * (int)sizeof(GroupSmem<CAP>);
    static_assert(bytes + 12 * SLOTS + 8 * kSegRing + 32 <= 232448, "one CTA's shared memory");
    auto kernel = k_gather_runs<CHANNEL, MODE, CAP, WARPS, SLOTS, LOW>;
    static std::atomic<bool> attr_set[64];  // per device; batched runs launch from several host threads
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    // a class word holds kClassMost contributions: more queries go in slices
    const uint64_t most = kClassMost / (uint64_t)k;
    for (uint64_t first = 0; first < q.n; first += most) {
        ScatterPlan plan{first, std::min<uint64_t>(most, q.n - first), 0u, 1, kSegBits, acc.nbins < kCachedBins, q.ticket};
        const uint64_t blocks = std::min<uint64_t>(sm_count(), plan.n);
        using G = std::conditional_t<CHANNEL == ALB_SCATTER, VolumeRuns, PlaneRuns>;
        plan.pieces = (uint32_t)((plan.n < kManyQueries ? 2 : 4) * blocks);
        // fewer chunks, or more levels, until a segment's chunks hold kChunk queries
        while (plan.chunk_bits > 4 && plan.n < (uint64_t)plan.pieces * G::kChunk << plan.chunk_bits) --plan.chunk_bits;
        while (plan.levels < 16 && (plan.n >> plan.levels) >= (uint64_t)plan.pieces * G::kChunk << plan.chunk_bits) ++plan.levels;
        cudaMemsetAsync(q.ticket, 0, sizeof(uint32_t), st);
        kernel<<<(unsigned)blocks, WARPS * 32, bytes, st>>>(sc, map, q, acc, k, err, plan);
        note_launch();
        merge_classes(sc, acc, CHANNEL, true, st);
    }
}

// Whether a planar channel's gather goes by runs (gather_group.cuh): from 2^16 queries, 13 for each
// resident warp, with 224 candidates enough for k. The bottom gather of the large scene at 1e6 photons
// (3e5 queries): 2.8 -> 0.89 ms, transmission 2.0 -> 0.65, at 1e7 photons 21.6 -> 5.4 and 19.0 -> 4.5; 28 000 queries
// take the same time either way (default scene: bottom 0.43 and 0.37 ms, transmission 0.31 and 0.32), and
// the one-query kernel leaves room on the SMs for the gathers beside it. The surface gather stays with
// k_gather: most of its queries lie far from the beam's spot, each has its neighbours at the same
// edge of it, and the neighbours' few bins are hot words in L2 (8.0 ms by runs, 2.1 with the bins cached).
constexpr uint64_t kPlanarRunsMin = 1u << 16;
static constexpr bool runs_channel(int channel) { return channel != ALB_SURFACE_REFLECTION; }
static bool planar_runs(int channel, uint64_t nq, int k) {
    return runs_channel(channel) && nq >= kPlanarRunsMin && k <= 128;
}

// Bins up to which the scatter gather caches the waveform's class words: 126 bins (a 40 ns record at
// 3 GHz, 3.1e5 queries) 4.7 -> 2.7 ms; 2858 bins are the same either way, 84,056 bins 22.7 -> 23.7.
constexpr int64_t kFewBins = 1024;
template <int CHANNEL, int MODE>
static void launch_channel(const MapDev& map, const QueryDev& q, const SceneDev& sc, const Accum& acc, int* err,
                           uint64_t nq, int k, cudaStream_t st) {
    if constexpr (MODE != kModeRadius && runs_channel(CHANNEL)) {
        if (CHANNEL == ALB_SCATTER || planar_runs(CHANNEL, nq, k)) {
            // candidates of a first guess: 1.33 k, twice that where the map thickens
            constexpr int slots = MODE == kModeKnnHeat || CHANNEL != ALB_SCATTER ? 1024 : 0;
            if constexpr (CHANNEL == ALB_SCATTER) {
                if (k > 128) {
                    launch_runs<CHANNEL, MODE, 448, 22, slots>(sc, map, q, acc, k, err, st);
                    return;
                }
                if constexpr (MODE == kModeKnn) {
                    if (acc.nbins <= kFewBins) {
                        launch_runs<CHANNEL, MODE, 224, 32, 1024>(sc, map, q, acc, k, err, st);
                        return;
                    }
                }
                if (q.lo_zero) launch_runs<CHANNEL, MODE, 224, 32, slots, false>(sc, map, q, acc, k, err, st);
                else launch_runs<CHANNEL, MODE, 224, 32, slots>(sc, map, q, acc, k, err, st);
            } else {
                launch_runs<CHANNEL, MODE, 224, 32, slots>(sc, map, q, acc, k, err, st);
            }
            return;
        }
    }
    if constexpr (CHANNEL != ALB_SCATTER || MODE == kModeRadius) {
        const uint32_t chunk = query_chunk(nq, MODE == kModeRadius);
        const unsigned blocks = gather_blocks((nq + chunk - 1) / chunk);
        RadiusWork work{};
        if (MODE == kModeRadius && q.work) {
            work = RadiusWork{(uint2*)(q.work + 2), q.work, kRadiusItems, false};
            cudaMemsetAsync(q.work, 0, 4, st);
        }
        k_gather<CHANNEL, MODE><<<blocks, kGatherWarps * 32, 0, st>>>(sc, map, q, acc, k, err, chunk, work);
        note_launch();
        if (work.items) {
            work.second = true;
            k_gather<CHANNEL, MODE><<<sm_count() * kGatherBlocksPerSM, kGatherWarps * 32, 0, st>>>(sc, map, q, acc, k, err, 1, work);
            note_launch();
        }
        if (MODE != kModeKnn) merge_classes(sc, acc, CHANNEL, false, st);
    }
}

template <int MODE>
static void launch_gather_mode(const MapDev& map, const QueryDev& q, int channel, const SceneDev& sc, const Accum& acc,
                               int* err, uint64_t nq, int k, cudaStream_t st) {
    switch (channel) {
        case ALB_BOTTOM_REFLECTION: launch_channel<ALB_BOTTOM_REFLECTION, MODE>(map, q, sc, acc, err, nq, k, st); break;
        case ALB_SCATTER: launch_channel<ALB_SCATTER, MODE>(map, q, sc, acc, err, nq, k, st); break;
        case ALB_SURFACE_REFLECTION: launch_channel<ALB_SURFACE_REFLECTION, MODE>(map, q, sc, acc, err, nq, k, st); break;
        default: launch_channel<ALB_SURFACE_TRANSMISSION_UP, MODE>(map, q, sc, acc, err, nq, k, st); break;
    }
}

void launch_gather(const SceneDev& sc, const MapDev& map, const QueryDev& q, int channel, const Accum& accum,
                   int* err, int* launches, cudaStream_t st) {
    if (q.n == 0) return;
    int k = sc.k;
    Accum acc = accum;
    acc.cls += (uint64_t)channel * acc.cls_step;
    // contributions of the launch at most (a fixed radius admits any number of the map's records);
    // the gathers by runs keep below kClassMost by slices
    const uint64_t per = sc.radius > 0.0 ? std::max<uint64_t>(map.n, 1) : (uint64_t)k;
    if (q.n > kClassMost / per && (sc.radius > 0.0 || (channel != ALB_SCATTER && !planar_runs(channel, q.n, k)))) acc.jac_cls = acc.heat_cls = nullptr;
    if (sc.radius > 0.0) launch_gather_mode<kModeRadius>(map, q, channel, sc, acc, err, q.n, k, st);
    else if (acc.jac_lo) launch_gather_mode<kModeKnnAdjoint>(map, q, channel, sc, acc, err, q.n, k, st);
    else if (acc.hw_lo && map.fwi) launch_gather_mode<kModeKnnHeat>(map, q, channel, sc, acc, err, q.n, k, st);
    else launch_gather_mode<kModeKnn>(map, q, channel, sc, acc, err, q.n, k, st);
    if (launches) ++*launches;
}

// Blocks of the launches over marks: 32 queries to a warp's step, one wave at most.
static unsigned crowded_blocks(uint64_t nq) {
    const uint64_t want = (nq + 32 * kCrowdedWarps - 1) / (32 * kCrowdedWarps);
    return (unsigned)std::min<uint64_t>(want, (uint64_t)sm_count() * 4);
}

template <int CHANNEL>
static void launch_crowded_channel(const SceneDev& sc, const MapDev& map, const QueryDev& q, const Accum& acc, int* err,
                                   cudaStream_t st) {
    const uint64_t most = kClassMost / (uint64_t)sc.k;
    for (uint64_t first = 0; first < q.n; first += most) {
        const uint64_t end = std::min<uint64_t>(q.n, first + most);
        k_gather_crowded<CHANNEL><<<crowded_blocks(end - first), kCrowdedWarps * 32, 0, st>>>(sc, map, q, acc, sc.k, err, first, end);
        note_launch();
        merge_classes(sc, acc, CHANNEL, true, st);
    }
}

void launch_gather_crowded(const SceneDev& sc, const MapDev& map, const QueryDev& q, int channel, const Accum& accum,
                           int* err, cudaStream_t st) {
    Accum acc = accum;
    acc.cls += (uint64_t)channel * acc.cls_step;
    switch (channel) {
        case ALB_BOTTOM_REFLECTION: launch_crowded_channel<ALB_BOTTOM_REFLECTION>(sc, map, q, acc, err, st); break;
        case ALB_SCATTER: launch_crowded_channel<ALB_SCATTER>(sc, map, q, acc, err, st); break;
        case ALB_SURFACE_REFLECTION: launch_crowded_channel<ALB_SURFACE_REFLECTION>(sc, map, q, acc, err, st); break;
        default: launch_crowded_channel<ALB_SURFACE_TRANSMISSION_UP>(sc, map, q, acc, err, st); break;
    }
}

void launch_knn(const MapDev& map, const double* queries, const uint32_t* perm, uint64_t nq, int k, int32_t* out_idx,
                double* out_dist, int* err, uint32_t* crowded, cudaStream_t st) {
    if (nq == 0) return;
    const uint32_t chunk = query_chunk(nq, false);
    k_knn<<<gather_blocks((nq + chunk - 1) / chunk), kGatherWarps * 32, 0, st>>>(map, queries, perm, nq, chunk, k, out_idx,
                                                                                  out_dist, err, crowded);
    note_launch();
}

void launch_knn_crowded(const MapDev& map, const double* queries, uint64_t nq, int k, int32_t* out_idx, double* out_dist,
                        int* err, cudaStream_t st) {
    k_knn_crowded<<<crowded_blocks(nq), kCrowdedWarps * 32, 0, st>>>(map, queries, nq, k, out_idx, out_dist, err);
    note_launch();
}

// Whether a query goes to a lane (k_knn_lanes) or to a warp (k_knn_brute): from 2^14 queries of up to 4 neighbours and
// 2^16 of up to 16. 4096 points, 1e6 queries, k = 1, 4, 16: 16.5, 19.0, 20.3 ms by warps, 3.1, 4.4, 10.2 by lanes (a
// walk of a tree 4.3, 6.5, 15.9); 2^14 queries, k = 4, 16: 0.34 and 0.35 by warps, 0.29 and 0.58 by lanes; 24
// neighbours take 22.6 by warps and 31.7 by lanes.
static bool lane_queries(uint64_t nq, int k) { return nq >= (k <= 4 ? 1u << 14 : 1u << 16) && k <= 16; }

template <int K>
static void launch_knn_lanes(const float* pts, uint32_t m, const double* queries, uint64_t nq, int k, int32_t* out_idx,
                             double* out_dist, cudaStream_t st) {
    k_knn_lanes<K><<<(unsigned)((nq + kLaneThreads - 1) / kLaneThreads), kLaneThreads, 0, st>>>(pts, m, queries, nq, k, out_idx, out_dist);
    note_launch();
}

void launch_knn_brute(const float* pts, uint32_t m, const double* queries, uint64_t nq, int k, int32_t* out_idx,
                      double* out_dist, cudaStream_t st) {
    if (lane_queries(nq, k)) {
        if (k == 1) launch_knn_lanes<1>(pts, m, queries, nq, k, out_idx, out_dist, st);
        else if (k <= 4) launch_knn_lanes<4>(pts, m, queries, nq, k, out_idx, out_dist, st);
        else if (k <= 8) launch_knn_lanes<8>(pts, m, queries, nq, k, out_idx, out_dist, st);
        else launch_knn_lanes<16>(pts, m, queries, nq, k, out_idx, out_dist, st);
        return;
    }
    const unsigned blocks = (unsigned)std::min<uint64_t>((nq + kBruteWarps - 1) / kBruteWarps, (uint64_t)sm_count() * 16);
    k_knn_brute<<<blocks, kBruteWarps * 32, 0, st>>>(pts, m, queries, nq, k, out_idx, out_dist);
    note_launch();
}

// 128-bit fixed-point words as floating point numbers (fix_to_double).
template <class T>
__global__ void k_fix_to_float(const unsigned long long* __restrict__ lo, const unsigned long long* __restrict__ hi, int64_t n,
                               T* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = (T)fix_to_double(lo[i], (long long)hi[i]);
}
void launch_fix_to_float(const unsigned long long* lo, const unsigned long long* hi, int64_t n, float* out, cudaStream_t st) {
    k_fix_to_float<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(lo, hi, n, out);
    note_launch();
}
void launch_fix_to_float(const unsigned long long* lo, const unsigned long long* hi, int64_t n, double* out, cudaStream_t st) {
    k_fix_to_float<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(lo, hi, n, out);
    note_launch();
}

}  // namespace alb
