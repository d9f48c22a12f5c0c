// Grouped k-NN search of the scatter map and of large planar gathers (included by gather.cu).
//
// A warp takes a run of consecutive sorted queries whose common box is small against their k-th
// distance, walks the box tree once for all of them, and keeps the leaves it meets with their
// boxes in shared memory. Each query then tests the listed boxes lane-parallel (two or three
// rounds) and screens only the leaves its own ball meets. The walk from the root, which the
// one-query search pays for every query, is shared by the run.
//
// A query's first threshold is a guess from its predecessor's k-th distance, (1.1 r)^2, and its
// answer is taken only when it proves itself complete: at least k candidates, and the k-th with
// its band margin within the guess, so that every point that can rank among the k nearest was
// below the admission threshold and every leaf holding one was screened. Consecutive k-th
// distances differ by less than 10% for 97.7% of the queries in Hilbert order; the others are
// searched again under the list's own radius (1.25 r), and alone if that fails too.
//
// What bounds it: instruction issue and L2 latency. One-query search in the same query order, per
// query of the large scene at 1e6 photons (8.7e6 queries): 7.8 tree nodes walked, 4600 warp
// instructions, 51.0 ms; in runs: 0.07 nodes, 2650 warp instructions, 31.7 ms (1e7 photons:
// 492 -> 318 ms). With the accumulation by class words and the map in Hilbert order 23.0 ms (231);
// leaves padded to 32 records, position and energy of a candidate in one access, boxes by centre and half
// width, and no low parts where the queries have none: 22.2 ms (225), of which the search is three
// quarters.
#pragma once

namespace alb {

constexpr int kGroupLeaves = 128;  // capacity of the leaf list
// Leaves a run is sized for (estimated from its box): longer runs share one walk among more
// queries, but every query tests the whole list (large scene, 1e6 photons: 36 -> 31.7 ms, 48 ->
// 29.2, 64 -> 27.9, 80 -> 27.6).
constexpr float kGroupTarget = 80.f;

// What depends on how records fill space. kGuess2, kList2: squared widening of the previous query's k-th
// distance, what a query first admits within and what the run's leaf list covers (the second
// attempt). side: edge of a leaf over the k-th distance, 32 records against k in the ball.
// est: leaves that a ball of radius T around a box of the given extents meets, the ball as the
// cube (square) of its volume. kGrow: count ~ (squared distance)^kGrow. kChunk: queries that a chunk of
// the last level holds at least (planar gathers of 3e5 and 2.5e5 queries: 8 -> 16 0.95 -> 0.78 and 0.65 ->
// 0.53 ms; the scatter gather of 4e6 adjoint queries 14.1 -> 14.6).
struct VolumeRuns {
    static constexpr float kGuess2 = 1.21f, kList2 = 1.5625f, kGrow = 1.5f;
    static constexpr uint64_t kChunk = 8;
    static ALB_DEVICE float side(float k) { return cbrtf(134.04f / k); }
    static ALB_DEVICE float est(float dx, float dy, float dz, float side, float T) {
        const float w = side + 1.61f * T;
        return (dx + w) * (dy + w) * (dz + w) / (side * side * side);
    }
};
// A horizontal plane. (Guesses of 1.15 and 1.3 measured the same to 4%.)
struct PlaneRuns {
    static constexpr float kGuess2 = 1.21f, kList2 = 1.5625f, kGrow = 1.f;
    static constexpr uint64_t kChunk = 16;
    static ALB_DEVICE float side(float k) { return sqrtf(100.53f / k); }
    static ALB_DEVICE float est(float dx, float, float dz, float side, float T) {
        const float w = side + 1.77f * T;
        return (dx + w) * (dz + w) / (side * side);
    }
};
constexpr int kGroupStack = 192;  // 31 open boxes per level below the root level's 32, 6 levels

template <int CAP>
struct GroupSmem {
    static constexpr int kCap = CAP, kSelectAt = CAP - 32, kTmp = 2 * kGroupStack + 128;
    float cd[CAP];     // candidates: squared float32 distance
    union {
        uint2 cp[CAP];  // map position and energy (grouped search: one access for both)
        struct {
            uint32_t ci[CAP];  // map position
            int16_t cl[CAP];   // distance fraction (one-query search)
        };
    };
    uint32_t leaf[kGroupLeaves];  // the run's leaves
    uint32_t hit[kGroupLeaves];   // those the current query's ball meets
    union {
        float box[6][kGroupLeaves];  // the run's leaf boxes: centre x, y, z, half width x, y, z
        struct {                     // scratch of the one-query search
            uint32_t stk[kGroupStack];
            float stk_d[kGroupStack];
            uint32_t hist[128];
            double bd[kBand];
            uint32_t bi[kBand];
            uint64_t bt[kBand];
        };
    };
    unsigned long long st[4];
    int alone, streak;  // queries still to be searched alone, and the next such stretch
    // scratch words of the boundary band, once the one-query search has left its stack
    ALB_DEVICE uint32_t& tmp(int i) {
        if (i < kGroupStack) return stk[i];
        if (i < 2 * kGroupStack) return reinterpret_cast<uint32_t*>(stk_d)[i - kGroupStack];
        return hist[i - 2 * kGroupStack];
    }
};

// A run of queries: its box and the leaf list.
struct QueryRun {
    int take;   // queries covered
    int n;      // leaves listed
    int nodes;  // boxes expanded for the list
    float T2;   // the list holds every leaf within this squared distance of the run's box
};

ALB_DEVICE float run_gap(float lo, float hi, float qlo, float qhi, float ql) {
    float g = fmaxf(fmaxf(lo - qhi, qlo - hi), 0.f);
    return fmaxf(g * (1.f - 2.384185791015625e-07f) - ql, 0.f);
}

// Half width of a box around its centre as a float, rounded up, with the largest low part of the run's
// queries; and a query's gap to the box from both, three operations, never above the true one: |q - c|
// is off by 2^-24 of itself and the last rounding by 2^-24 of the gap, both below the 2^-22 taken off.
// (NaN, where a box reaches infinity, counts as no gap.)
ALB_DEVICE float half_width(float lo, float hi, float low) {
    const float c = 0.5f * (lo + hi);
    return __fadd_ru(fmaxf(__fsub_ru(hi, c), __fsub_ru(c, lo)), low);
}
ALB_DEVICE float centre_gap(float q, float c, float h) {
    return fmaxf(fmaf(fabsf(q - c), 1.f - 2.384185791015625e-07f, -h), 0.f);
}

// Builds the run starting at the first of `avail` queries whose positions the lanes hold (lane i
// the i-th; la = the largest low part of its coordinates). Every float operation of run_gap is
// monotone in the query, so a listed leaf's lower bound is never above any covered query's own.
template <class G, class S>
ALB_DEVICE bool build_run(const MapDev& m, S& s, int avail, float x, float y, float z, float la, float r2, float side,
                          QueryRun& run) {
    const int l = lane_id();
    const bool have = l < avail;
    float x0 = have ? x : 3.0e38f, y0 = have ? y : 3.0e38f, z0 = have ? z : 3.0e38f;
    float x1 = have ? x : -3.0e38f, y1 = have ? y : -3.0e38f, z1 = have ? z : -3.0e38f;
    la = have ? la : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float a0 = __shfl_up_sync(0xffffffffu, x0, o), b0 = __shfl_up_sync(0xffffffffu, y0, o),
                    c0 = __shfl_up_sync(0xffffffffu, z0, o), a1 = __shfl_up_sync(0xffffffffu, x1, o),
                    b1 = __shfl_up_sync(0xffffffffu, y1, o), c1 = __shfl_up_sync(0xffffffffu, z1, o),
                    lb = __shfl_up_sync(0xffffffffu, la, o);
        if (l >= o) {
            x0 = fminf(x0, a0); y0 = fminf(y0, b0); z0 = fminf(z0, c0);
            x1 = fmaxf(x1, a1); y1 = fmaxf(y1, b1); z1 = fmaxf(z1, c1);
            la = fmaxf(la, lb);
        }
    }
    run.T2 = r2 * G::kList2;
    const float est = G::est(x1 - x0, y1 - y0, z1 - z0, side, sqrtf(run.T2));
    run.take = max(__popc(__ballot_sync(0xffffffffu, have && est <= kGroupTarget)), 1);
    uint32_t* stk = reinterpret_cast<uint32_t*>(s.cd);  // the candidates are free here
    static_assert(S::kCap >= kGroupStack, "the walk's stack lies in the candidate buffer");
    while (true) {
        const int t = run.take - 1;
        const float bx0 = __shfl_sync(0xffffffffu, x0, t), by0 = __shfl_sync(0xffffffffu, y0, t),
                    bz0 = __shfl_sync(0xffffffffu, z0, t), bx1 = __shfl_sync(0xffffffffu, x1, t),
                    by1 = __shfl_sync(0xffffffffu, y1, t), bz1 = __shfl_sync(0xffffffffu, z1, t),
                    bl = __shfl_sync(0xffffffffu, la, t);
        int n = 0, sp = 0;
        int cl = m.nlevels - 1;
        uint32_t c0 = 0u;
        bool full = false;
        __syncwarp();
        // every box is expanded at most once, and the list's bound ends the walk of a wide run
        for (int guard = 0; guard < (1 << 16); ++guard) {
            const uint32_t c = c0 + l;
            ++run.nodes;
            bool in = (uint64_t)c < m.lvl_cnt[cl];
            float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
            if (in) {
                lo = m.box_lo[m.lvl_off[cl] + c];
                hi = m.box_hi[m.lvl_off[cl] + c];
                const float dx = run_gap(lo.x, hi.x, bx0, bx1, bl), dy = run_gap(lo.y, hi.y, by0, by1, bl),
                            dz = run_gap(lo.z, hi.z, bz0, bz1, bl);
                in = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) * (1.f - 4.76837158203125e-07f) <= run.T2;
            }
            const unsigned b = __ballot_sync(0xffffffffu, in);
            const int pos = __popc(b & lanemask_lt());
            if (cl == 0) {
                if (n + __popc(b) > kGroupLeaves) {
                    full = true;
                    break;
                }
                if (in) {
                    const int e = n + pos;
                    s.leaf[e] = c;
                    s.box[0][e] = 0.5f * (lo.x + hi.x);
                    s.box[1][e] = 0.5f * (lo.y + hi.y);
                    s.box[2][e] = 0.5f * (lo.z + hi.z);
                    s.box[3][e] = half_width(lo.x, hi.x, bl);
                    s.box[4][e] = half_width(lo.y, hi.y, bl);
                    s.box[5][e] = half_width(lo.z, hi.z, bl);
                }
                n += __popc(b);
            } else {
                if (in) stk[sp + pos] = ((uint32_t)cl << 29) | c;
                sp += __popc(b);
            }
            __syncwarp();
            if (sp == 0) break;
            const uint32_t e = stk[--sp];
            __syncwarp();
            cl = (int)(e >> 29) - 1;
            c0 = (e & 0x1fffffffu) * 32u;
            if (guard == (1 << 16) - 1) full = true;
        }
        if (!full) {
            run.n = n;
            return true;
        }
        if (run.take == 1) return false;
        run.take >>= 1;
    }
}

// The k-th smallest of the candidates cd[0 .. cnt), k <= cnt, none above hi: a value x with exactly
// k candidates <= x is searched by secant steps on the count (which grows like x^1.5 in a
// volume), every count one pass over registers and one warp reduction. Returns false when equal
// distances straddle the k-th place (no such x). v: this lane's candidates (FLT_MAX beyond cnt).
template <int R>
ALB_DEVICE int count_le(const float (&v)[R], float x) {
    int c = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) c += v[j] <= x ? 1 : 0;
    return __reduce_add_sync(0xffffffffu, c);
}
template <class G, int R>
ALB_DEVICE bool find_cut(const float (&v)[R], int cnt, int k, float hi, float& x) {
    if (cnt == k) {
        x = hi;
        return true;
    }
    float a = 0.f, b = hi;  // count(a) < k (count(0) = k is the degenerate case below), count(b) > k
    int ca = 0, cb = cnt;
    x = hi * __powf((float)k / (float)cnt, 1.f / G::kGrow);
#pragma unroll 1
    for (int it = 0; it < 20; ++it) {
        if (!(x > a && x < b)) x = 0.5f * (a + b);
        const int c = count_le(v, x);
        if (c == k) return true;
        if (c < k) {
            a = x;
            ca = c;
        } else {
            b = x;
            cb = c;
        }
        // interpolate within the bracket, aiming between the k-th and the next
        x = a + (b - a) * (((float)(k - ca) + 0.5f) / ((float)(cb - ca) + 1.f));
    }
    return false;
}

// One query against the run's list under the threshold thr (squared, with the band margin).
// 1: s.cp[0 .. k) holds the k nearest, kth their largest float32 distance, kid its map
// position; 0: the threshold does not prove an answer; -1: a near tie at the k-th place (kth is
// then a proven bound when > 0), or too many candidates at one distance.
template <class G, class S>
ALB_DEVICE int run_search(const MapDev& m, S& s, int k, int nlist, float fx, float fy, float fz, float lx, float ly,
                          float lz, float thr, float& kth, uint32_t& kid, int& leaves) {
    constexpr int R = S::kCap / 32;
    const int l = lane_id();
    const float guess = thr;
    int nh = 0;
#pragma unroll 1
    for (int e0 = 0; e0 < nlist; e0 += 32) {
        const int e = e0 + l;
        bool in = false;
        if (e < nlist) {
            const float dx = centre_gap(fx, s.box[0][e], s.box[3][e]), dy = centre_gap(fy, s.box[1][e], s.box[4][e]),
                        dz = centre_gap(fz, s.box[2][e], s.box[5][e]);
            in = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) * (1.f - 4.76837158203125e-07f) <= thr;
        }
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) s.hit[nh + __popc(b & lanemask_lt())] = s.leaf[e];
        nh += __popc(b);
    }
    __syncwarp();
    leaves += nh;
    int cnt = 0;
    kth = 0.f;
    auto admit = [&](uint32_t r, float4 p, bool on) {
        const float d = point_dist2(fx, fy, fz, lx, ly, lz, p);
        const bool in = on && d <= thr;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int pos = cnt + __popc(b & lanemask_lt());
            s.cd[pos] = d;
            s.cp[pos] = make_uint2(r, __float_as_uint(p.w));
        }
        cnt += __popc(b);
    };
#pragma unroll 1
    for (int i = 0; i < nh; i += 2) {
        // two leaves' records in flight at a time
        const uint32_t r0 = s.hit[i] * 32u + l, r1 = s.hit[min(i + 1, nh - 1)] * 32u + l;
        const float4 p0 = m.a[r0], p1 = m.a[r1];  // a partial leaf is padded with far points
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            admit(h ? r1 : r0, h ? p1 : p0, h == 0 || i + 1 < nh);
            if (cnt > S::kSelectAt) {
                // more candidates than the guess allows for: shrink to the k best so far
                __syncwarp();
                float v[R], x;
#pragma unroll
                for (int j = 0; j < R; ++j) v[j] = j * 32 + l < cnt ? s.cd[j * 32 + l] : FLT_MAX;
                if (!find_cut<G>(v, cnt, k, thr, x)) return -1;
                thr = fminf(thr, x * (1.0f + 2.0f * kRelMargin));
                int out = 0;
#pragma unroll
                for (int j = 0; j < R; ++j) {
                    const bool keep = v[j] <= thr;
                    const unsigned b = __ballot_sync(0xffffffffu, keep);
                    const uint2 c = s.cp[j * 32 + l];
                    __syncwarp();
                    if (keep) {
                        const int pos = out + __popc(b & lanemask_lt());
                        s.cd[pos] = v[j];
                        s.cp[pos] = c;
                    }
                    out += __popc(b);
                    __syncwarp();
                }
                cnt = out;
                if (cnt > S::kSelectAt) return -1;
            }
        }
    }
    __syncwarp();
    if (cnt < k) return 0;
    float v[R], x;
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = j * 32 + l < cnt ? s.cd[j * 32 + l] : FLT_MAX;
    if (!find_cut<G>(v, cnt, k, thr, x)) return -1;
    // the k-th, and whether another candidate lies within the screening margin of it
    unsigned mx = 0u;
#pragma unroll
    for (int j = 0; j < R; ++j) mx = max(mx, v[j] <= x ? __float_as_uint(v[j]) : 0u);
    kth = __uint_as_float(__reduce_max_sync(0xffffffffu, mx));
    const float blo = kth * (1.0f - 2.0f * kRelMargin), bhi = kth * (1.0f + 2.0f * kRelMargin);
    if (!(bhi <= guess)) return 0;
    int band = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) band += v[j] >= blo && v[j] <= bhi ? 1 : 0;
    if (__reduce_add_sync(0xffffffffu, band) != 1) return -1;
    int out = 0;
    uint32_t own = 0u;
    bool mine = false;
#pragma unroll
    for (int j = 0; j < R; ++j) {
        if (j * 32 < cnt) {
            const bool keep = v[j] <= x;
            const unsigned b = __ballot_sync(0xffffffffu, keep);
            const uint2 c = s.cp[j * 32 + l];
            if (v[j] == kth) {
                own = c.x;
                mine = true;
            }
            __syncwarp();
            if (keep) s.cp[out + __popc(b & lanemask_lt())] = c;
            out += __popc(b);
            __syncwarp();
        }
    }
    kid = __shfl_sync(0xffffffffu, own, __ffs(__ballot_sync(0xffffffffu, mine)) - 1);
    return 1;
}

// float32(sqrt(x)) of the float64 squared distance x from the query (f + l per axis) to p, equal
// to sqrt_to_f32(point_dist2_f64(...)), from the double-float distance hi + lo: with s =
// sqrtf(hi) the residual hi - s^2 is exact, and sqrt(x) rounds to s, or to the float next to it,
// by where hi - s^2 + lo lies against the midpoints s^2 +- s ulp(s). The distance is good to
// 2^-44, so only values within 2^-10 of a midpoint's offset take the float64 path. GB300 issues
// two FP64 lanes per SM and cycle: about 25 FP64 instructions per query cost more of the SM
// than the whole search of a query here.
ALB_DEVICE float dist_f32(float fx, float fy, float fz, float lx, float ly, float lz, float4 p, float& d2) {
    float hi, lo;
    point_dist2_df(fx, fy, fz, lx, ly, lz, p, hi, lo);
    d2 = hi;
    if (hi > 1.0e-20f && hi < 1.0e30f) {
        const float s = __fsqrt_rn(hi);
        const float e = __fadd_rn(fmaf(-s, s, hi), lo);
        const float up = __int_as_float(__float_as_int(s) + 1);
        const float half = s * (up - s);  // s ulp(s): the midpoints' offset (to 2^-24 of itself)
        if (e > half * (1.f + 1.f / 1024.f)) return up;
        // below a power of two the spacing halves: leave those to float64
        if (e >= 0.f || (__float_as_int(s) & 0x7fffff)) {
            if (fabsf(e) < half * (1.f - 1.f / 1024.f)) return s;
            if (e < -half * (1.f + 1.f / 1024.f)) return __int_as_float(__float_as_int(s) - 1);
        }
    }
    const double x = point_dist2_f64((double)fx + (double)lx, (double)fy + (double)ly, (double)fz + (double)lz, p);
    d2 = (float)x;
    return sqrt_to_f32(x);
}

}  // namespace alb
