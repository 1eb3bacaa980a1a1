// knn_fit.cu - the ROV's regressions: k nearest neighbours and multiple
// local linear regression, a thread per grid query.
//
// Reference: knn_cuda_with_indexes::knn (include/gpuCode/
// knn_cuda_with_indexes.cu:475-618) and multiLocLinReg (SimulateGPU.cu:
// 2934-3053).
//
// A CTA takes a tile of 128 grid queries of one (road, control) group.  The
// group's points pass through shared memory, every thread reads the same
// one at a time (a broadcast) and keeps its own query's state, so no lane
// ever idles over a short list and the per-query bookkeeping - scans,
// selections, solves - costs a thread what it used to cost a warp.  The
// neighbours do not depend on the values of later years, so they are
// selected (k_knn_rov) for as many years at once as half a gigabyte holds the
// lists of, every grid query counted (a road: all; 256 roads: one):
//   1 a histogram of a sample of the squared distances, 8 buckets an octave,
//     estimates the k-th;
//   2 a histogram of all of them, 32 buckets an octave around the estimate,
//     finds the bucket that holds the k-th (the window moves, or narrows
//     onto a bucket of many, until it holds at most kSide distances);
//   3 the points below that bucket's end are listed in index order, those in
//     it marked, and the farthest of these dropped until k are left - the k
//     smallest by (squared distance, index), the set the reference's stable
//     insertion sort returns.
// Then, year by year (k_knn_fit): the normal equations over the k points in
// ascending index, neighbour m into partial m mod 32, partials added in
// order (the order of the CPU oracle), and the FP64 solve.
// Squared distances are compared as bits (they are >= 0, so their bits order
// as the values; a distance that is not a number comes last).
//
// What bounds it: instruction issue and, at the few warps an SM that the
// histograms (256 bytes a query) and the sums (registers, up to three
// species; four take 880 bytes a thread of local memory for the solve) leave
// room for, the latency of dependent instructions.  Two kernels instead of
// one for that reason: selecting needs no registers to speak of, fitting no
// shared memory.  256 roads, 24.7 M queries of about 256 points and k = 65 (a
// generation): kNN and solves 44.1 -> 19.9 ms (select 10.5, fit 9.4; 528 warp
// instructions a query, 1,588 with a warp a query).  One road of 10,000
// paths, 100,000 queries of about 3,300 points: 4.2 -> 1.2 ms.
#include <cmath>

#include "to_f2.cuh"
#include "to_internal.cuh"
#include "to_lsm_math.h"
#include "to_rov.cuh"

namespace {

constexpr int kT = TO_ROV_TILE;            // threads = queries worked on at a time
constexpr int kW = 32;                     // lanes
constexpr int kPts = 512;                  // points in shared memory at a time (selection)
constexpr int kFitBytes = 56 * 1024;       // shared memory of the fit: four CTAs an SM
constexpr int kBuckets = 64;               // 62 and the two ends
constexpr int kSide = 16;                  // most distances in the last bucket
constexpr unsigned kMark = 0x8000u;        // a listed point of the last bucket
static_assert(TO_ROV_SCAN_PATHS <= 32768, "point numbers of 15 bits");
constexpr unsigned kAll = 0xffffffffu;

// squared distances (as bits) of points i .. i+3 of the tile to the query;
// nq holds its negated coordinates, each twice
template <int D>
__device__ __forceinline__ void dist4(const float* pts, int i, const f2 (&nq)[D], unsigned (&b)[4]) {
    f2 s0, s1;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pts + j * kPts + i);
        const f2 t0 = add2(v.x, nq[j]), t1 = add2(v.y, nq[j]);
        s0 = j ? fma2(t0, t0, s0) : mul2(t0, t0);
        s1 = j ? fma2(t1, t1, s1) : mul2(t1, t1);
    }
    bits2(s0, b[0], b[1]);
    bits2(s1, b[2], b[3]);
}

template <int D>
__device__ __forceinline__ unsigned dist1(const float* pts, int i, const f2 (&nq)[D]) {
    f2 s;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        const f2 t = add2(both2(pts[j * kPts + i]), nq[j]);
        s = j ? fma2(t, t, s) : mul2(t, t);
    }
    return (unsigned)s;
}

// to_lsm_weight_within of two neighbours, the same operations packed: nh is
// -h, and the exponent k = rint(w / ln 2) of w in [-1/2, 0] is -1 or 0 (a tie
// rounds to 0), so its power is 1/2 or 1.
__device__ __forceinline__ f2 weight2(float d0, float d1, f2 nh, f2 rh) {
    const f2 d = pack2(d0, d1);
    const f2 q = mul2(d, rh);
    const f2 t = fma2(fma2(q, nh, d), rh, q);
    const f2 w = mul2(mul2(t, t), both2(-0.5f));
    float x0, x1;
    unpack2(mul2(w, both2(0x1.715476p+0f)), x0, x1);
    const bool e0 = x0 < -0.5f, e1 = x1 < -0.5f;
    const f2 mk = pack2(e0 ? 1.0f : 0.0f, e1 ? 1.0f : 0.0f);        // -k
    f2 r = fma2(mk, both2(0x1.62e430p-1f), w);
    r = fma2(mk, both2(-0x1.05c610p-29f), r);
    f2 p = fma2(r, both2(0x1.a01a02p-13f), both2(0x1.6c16c2p-10f));
    p = fma2(r, p, both2(0x1.111112p-7f));
    p = fma2(r, p, both2(0x1.555556p-5f));
    p = fma2(r, p, both2(0x1.555556p-3f));
    p = fma2(r, p, both2(0.5f));
    p = fma2(r, p, both2(1.0f));
    p = fma2(r, p, both2(1.0f));
    return mul2(mul2(p, pack2(e0 ? 0.5f : 1.0f, e1 ? 0.5f : 1.0f)), both2(0.3989422804f));
}

// Window of 62 buckets of 2^shift bit patterns from first << shift; bucket 0
// holds what lies below, bucket 63 what lies above.
struct Window {
    int shift, first;
};
__device__ __forceinline__ int bucket_of(unsigned bits, Window w) {
    return __viaddmin_s32_relu((int)(bits >> w.shift), 1 - w.first, kBuckets - 1);
}

// adds points [0, cnt) of the tile to the thread's histogram (column of
// hist, kW wide)
template <int D>
__device__ __forceinline__ void histogram(const float* pts, int cnt, const f2 (&nq)[D], Window w,
                                          unsigned* hist) {
    const int c4 = cnt & ~3;
#pragma unroll 2
    for (int i = 0; i < c4; i += 4) {
        unsigned b[4];
        dist4<D>(pts, i, nq, b);
#pragma unroll
        for (int u = 0; u < 4; ++u) atomicAdd(&hist[bucket_of(b[u], w) * kW], 1u);
    }
    for (int i = c4; i < cnt; ++i)
        atomicAdd(&hist[bucket_of(dist1<D>(pts, i, nq), w) * kW], 1u);
}

// bucket where the running count reaches `rank` (63: above the window), and
// the count below it; eight loads in flight
__device__ __forceinline__ int find_bucket(const unsigned* hist, int rank, int& below) {
    int c = 0, at = -1;
    below = 0;
    for (int b0 = 0; b0 < kBuckets && at < 0; b0 += 8) {
        unsigned h[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) h[u] = hist[(b0 + u) * kW];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (at < 0 && c + (int)h[u] >= rank) { at = b0 + u; below = c; }
            c += (int)h[u];
        }
    }
    return at < 0 ? kBuckets - 1 : at;
}

__device__ __forceinline__ void clear_hist(unsigned* hist) {
#pragma unroll 8
    for (int b = 0; b < kBuckets; ++b) hist[b * kW] = 0u;
}

// per thread: the histogram, later the distances of the last bucket and the
// list of neighbours (one place past the end of each is written)
__host__ __device__ inline size_t select_thread_bytes(int kmax) {
    const size_t lists = (kSide + 1) * 4 + (size_t)(kmax + kSide + 1) * 2;
    const size_t hist = kBuckets * 4;
    return lists > hist ? ((lists + 3) & ~size_t(3)) : hist;
}
size_t select_smem(int d, int kmax) {
    return (size_t)d * kPts * 4 + (size_t)kT * select_thread_bytes(kmax);
}

// blockIdx.y: slot of the year, from a.sel0
template <int D>
__global__ void __launch_bounds__(kT, 5) k_knn_rov(to_rov_args a) {
    extern __shared__ __align__(16) unsigned char sm_fit[];
    __shared__ int s_tile;
    float* pts = reinterpret_cast<float*>(sm_fit);                    // [D][kPts]
    // a warp's own area (its lists take the place of its histograms while
    // other warps may still be counting), each array a column a lane
    const int tid = threadIdx.x, P = a.P, Q = a.Q;
    unsigned* area = reinterpret_cast<unsigned*>(
        sm_fit + D * kPts * 4 + (size_t)(tid >> 5) * kW * select_thread_bytes(a.kmax));
    unsigned* hist = area + (tid & 31);                               // [kBuckets]
    unsigned* side = hist;                                            // [kSide + 1]
    unsigned short* list = reinterpret_cast<unsigned short*>(area + (kSide + 1) * kW) + (tid & 31);
    const int slot = a.sel0 + blockIdx.y;
    const int ntiles = a.ntiles[slot], tcap = a.G * ((Q + kT - 1) / kT);
    const int2* tiles = a.tiles + (size_t)slot * tcap;
    for (;;) {
        if (tid == 0) s_tile = atomicAdd(a.ntiles + a.slots + slot, 1);
        __syncthreads();                       // also: the last tile is done with
        const int ti = s_tile;
        if (ti >= ntiles) break;
        const int g = tiles[ti].x, start = tiles[ti].y;
        const size_t gs = (size_t)slot * a.G + g;
        const int n = a.npts[gs], k = a.kc[gs];
        if (n < 3 || k <= 0) {                 // too few points
            __syncthreads();
            continue;
        }
        const bool live = start + tid < a.gcount[gs];
        const int at = live ? start + tid : start;
        const int qi = a.touched ? a.qlist[gs * Q + at] : at;
        const float* xs = a.xn + gs * D * P;
        f2 nq[D];
        {
            float qn[D], xq[D];
            to_rov_query<D>(a, slot, g / a.C, qi, qn, xq);
#pragma unroll
            for (int j = 0; j < D; ++j) nq[j] = both2(-qn[j]);
        }
        auto load = [&](int p0) {              // points p0 .. of the group
            const int c = min(kPts, n - p0);
            for (int i = tid; i < c; i += kT)
#pragma unroll
                for (int j = 0; j < D; ++j) pts[j * kPts + i] = xs[(size_t)j * P + p0 + i];
            return c;
        };
        const bool many = n > kPts;            // more points than fit at once
        load(0);
        __syncthreads();
        // 1: the sample is the group's first points (path order: independent)
        Window w;
        {
            const int ns = min(min(n, kPts), max(48, n >> 3));
            // the k-th lies within two octaves up and six down of the radius
            // that a uniform density over the unit cube gives
            const float rho = __powf(__fdividef((float)k, (float)n), 2.0f / (float)D);
            w.shift = 20;
            w.first = max((int)(__float_as_uint(rho) >> 20) - 50, 0);
            clear_hist(hist);
            histogram<D>(pts, ns, nq, w, hist);
            int below;
            const int rank = max(1, (int)(((float)k * (float)ns) / (float)n + 0.5f));
            const int b = find_bucket(hist, rank, below);
            w.first = max(((w.first + b - 1) << 2) + 2 - 31, 0);
            w.shift = 18;
        }
        // 2
        unsigned lo = 0, hi = 0;               // bucket of the k-th: bits in [lo, hi)
        int need = 0;                          // how many of it
        bool ties = false;                     // it is one value: the first of it
        bool found = !live;
        for (;;) {
            if (!found) clear_hist(hist);
            for (int p0 = 0; p0 < n; p0 += kPts) {
                int c = n;
                if (many) { __syncthreads(); c = load(p0); __syncthreads(); }
                if (!found) histogram<D>(pts, c, nq, w, hist);
            }
            if (!found) {
                int below;
                const int b = find_bucket(hist, k, below);
                if (b == 0) {                  // the window lies too high
                    const int f = w.first >> (21 - w.shift);
                    w.first = max(f - 61, 0);
                    w.shift = 21;
                } else if (b == kBuckets - 1) {
                    w.first = (w.first + 62) >> (21 - w.shift);
                    w.shift = 21;
                } else {
                    lo = (unsigned)(w.first + b - 1) << w.shift;
                    hi = lo + (1u << w.shift);
                    need = k - below;
                    ties = w.shift == 0;
                    if (ties || (int)hist[b * kW] <= kSide) {
                        found = true;
                    } else {
                        const int s = max(w.shift - 5, 0);
                        w.first = (int)(lo >> s);
                        w.shift = s;
                    }
                }
            }
            if (many ? !__syncthreads_or(!found) : !__any_sync(kAll, !found)) break;
        }
        __syncwarp();                          // the histograms make room for the lists
        // 3: every point is written at the list's end, which moves past it
        // where it is taken; so are the last bucket's distances
        int cl = 0, eq = 0;
        const bool any_ties = __any_sync(kAll, ties);
        for (int p0 = 0; p0 < n; p0 += kPts) {
            int c = n;
            if (many) { __syncthreads(); c = load(p0); __syncthreads(); }
            if (!live) continue;
            auto take = [&](unsigned b, int i) {
                const bool in = b < hi, last = in && b >= lo;
                list[cl * kW] = (unsigned short)(last ? i | kMark : i);
                side[eq * kW] = b;
                cl += in ? 1 : 0;
                eq += last ? 1 : 0;
            };
            auto take_ties = [&](unsigned b, int i) {      // any mix of lanes
                const bool last = b >= lo && b < hi;
                if (b < lo || (last && (!ties || eq < need))) {
                    list[cl * kW] = (unsigned short)(last && !ties ? i | kMark : i);
                    if (last && !ties) side[eq * kW] = b;
                    ++cl;
                    eq += last ? 1 : 0;
                }
            };
            const int c4 = c & ~3;
            if (!any_ties) {
#pragma unroll 2
                for (int i = 0; i < c4; i += 4) {
                    unsigned b[4];
                    dist4<D>(pts, i, nq, b);
#pragma unroll
                    for (int u = 0; u < 4; ++u) take(b[u], p0 + i + u);
                }
                for (int i = c4; i < c; ++i) take(dist1<D>(pts, i, nq), p0 + i);
            } else {
                for (int i = 0; i < c; ++i) take_ties(dist1<D>(pts, i, nq), p0 + i);
            }
        }
        // the farthest of the last bucket out (equal: the later ones first)
        float kth = __uint_as_float(lo);
        if (live && !ties) {
            unsigned v[kSide];
#pragma unroll
            for (int i = 0; i < kSide; ++i) v[i] = i < eq ? side[i * kW] + 1u : 0u;
            unsigned out = 0;
            for (int drop = eq - need; drop > 0; --drop) {
                unsigned best = 1u;
                int e = 0;
#pragma unroll
                for (int i = 0; i < kSide; ++i)
                    if (v[i] >= best) { best = v[i]; e = i; }
#pragma unroll
                for (int i = 0; i < kSide; ++i)
                    if (i == e) v[i] = 0u;
                out |= 1u << e;
            }
            unsigned top = 0;
#pragma unroll
            for (int i = 0; i < kSide; ++i) top = max(top, v[i]);
            kth = __uint_as_float(top - 1u);
            if (out) {
                int m = 0, e = 0;
                for (int i0 = 0; i0 < cl; i0 += 8) {
                    unsigned short x[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) x[u] = list[min(i0 + u, cl) * kW];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const bool last = (x[u] & kMark) != 0;
                        const bool keep = i0 + u < cl && !(last && (out >> e & 1u));
                        if (keep) list[m * kW] = x[u];
                        m += keep ? 1 : 0;
                        e += last && i0 + u < cl ? 1 : 0;
                    }
                }
            }
        }
        __syncwarp();
        const size_t tg = (size_t)blockIdx.y * tcap + ti;
        a.kthv[tg * kT + tid] = kth;
        unsigned short* nb = a.nbr + tg * a.kmax * kT + tid;
        if (live)
            for (int m = 0; m < k; ++m) nb[(size_t)m * kT] = list[m * kW] & (unsigned short)~kMark;
        __syncthreads();
    }
}

template <int D>
__host__ __device__ constexpr int fit_sums() { return (D + 1) + (D + 1) * (D + 2) / 2; }

// One query's neighbours and what its sums read
template <int D>
struct PairArgs {
    const unsigned short* nb;          // its list, `stride` apart
    int stride, k, n, P, np;
    bool many;                         // the points stay in global memory
    const float* pts;                  // [D + 1][np] points and values in shared memory
    const float *xs, *xr, *ynext;      // [D][P] points, [D][P] raw states, values by path
    const int* path;
    f2 nq[D], nh2, rh2;                // minus the query, minus the bandwidth, its reciprocal
    float xq[D];                       // regression centre (reference semantics)
};

// partials l and l + 1 of the normal equations (neighbours m with m mod 32 =
// l and l + 1), packed
template <int D, bool REF>
__device__ __forceinline__ void pair_sums(const PairArgs<D>& c, int l, f2 (&acc)[fit_sums<D>()]) {
    constexpr int M = D + 1;
#pragma unroll
    for (int e = 0; e < fit_sums<D>(); ++e) acc[e] = 0ull;
    for (int m = l; m < c.k; m += 32) {
        const bool two = m + 1 < c.k;    // the second exists (else weight 0)
        const int i0 = c.nb[m * c.stride], i1 = two ? c.nb[(m + 1) * c.stride] : i0;
        f2 dx[D], y2;
        if (c.many) {
#pragma unroll
            for (int j = 0; j < D; ++j)
                dx[j] = pack2(c.xs[(size_t)j * c.P + i0], c.xs[(size_t)j * c.P + i1]);
            y2 = pack2(c.ynext[c.path[i0]], c.ynext[c.path[i1]]);
        } else {
#pragma unroll
            for (int j = 0; j < D; ++j)
                dx[j] = pack2(c.pts[j * c.np + i0], c.pts[j * c.np + i1]);
            y2 = pack2(c.pts[D * c.np + i0], c.pts[D * c.np + i1]);
        }
        f2 s2;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            dx[j] = add2(dx[j], c.nq[j]);
            s2 = j ? fma2(dx[j], dx[j], s2) : mul2(dx[j], dx[j]);
        }
        if (REF) {
            // the reference reads its dim-major buffer (stride n)
            // point-major (multiLocLinReg, SimulateGPU.cu:3002) and
            // centres on the unit grid
#pragma unroll
            for (int j = 0; j < D; ++j) {
                const int f0 = i0 * D + j, j0 = f0 / c.n, f1 = i1 * D + j, j1 = f1 / c.n;
                dx[j] = pack2(c.xr[(size_t)j0 * c.P + (f0 - j0 * c.n)] - c.xq[j],
                              c.xr[(size_t)j1 * c.P + (f1 - j1 * c.n)] - c.xq[j]);
            }
        }
        float s0, s1;
        unpack2(s2, s0, s1);
        f2 z = weight2(sqrtf(s0), sqrtf(s1), c.nh2, c.rh2);
        if (!two) {
            float z0, z1;
            unpack2(z, z0, z1);
            z = pack2(z0, 0.0f);
        }
        // to_lsm_acc_add: B, then the upper triangle of A by rows
        acc[0] = fma2(y2, z, acc[0]);
#pragma unroll
        for (int j = 0; j < D; ++j) acc[1 + j] = fma2(mul2(y2, dx[j]), z, acc[1 + j]);
        int e = M;
        acc[e] = add2(acc[e], z);
        ++e;
#pragma unroll
        for (int j = 0; j < D; ++j, ++e) acc[e] = fma2(dx[j], z, acc[e]);
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int j = i; j < D; ++j, ++e) acc[e] = fma2(mul2(dx[j], dx[i]), z, acc[e]);
    }
}

// the arguments of the group and query (dd <= h: every neighbour lies within
// the k-th distance)
template <int D>
__device__ __forceinline__ PairArgs<D> pair_args(const to_rov_args& a, int slot, int t, int g,
                                                 int qi, float kth) {
    const size_t gs = (size_t)slot * a.G + g;
    PairArgs<D> c;
    c.k = a.kc[gs];
    c.n = a.npts[gs];
    c.P = a.P;
    c.xs = a.xn + gs * D * a.P;
    c.xr = a.xraw + gs * D * a.P;
    c.ynext = a.condExp + (size_t)(t + 1) * a.PT;
    c.path = a.pidx + gs * a.P;
    float qn[D];
    to_rov_query<D>(a, slot, g / a.C, qi, qn, c.xq);
#pragma unroll
    for (int j = 0; j < D; ++j) c.nq[j] = both2(-qn[j]);
    const float h = sqrtf(kth);
    c.nh2 = both2(-h);
    c.rh2 = both2(1.0f / h);
    return c;
}

// the group's points and their values into shared memory [D + 1][np]; all but
// the values, the year before's result, ahead of the wait for that year
template <int D>
__device__ __forceinline__ void load_points(const to_rov_args& a, int slot, int t, int g, int np,
                                            float* pts) {
    const size_t gs = (size_t)slot * a.G + g;
    const int n = a.npts[gs], P = a.P;
    const float* xs = a.xn + gs * D * P;
    const int* path = a.pidx + gs * P;
    const float* ynext = a.condExp + (size_t)(t + 1) * a.PT;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
#pragma unroll
        for (int j = 0; j < D; ++j) pts[j * np + i] = xs[(size_t)j * P + i];
        pts[D * np + i] = __int_as_float(path[i]);
    }
    to_pdl_wait();
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        pts[D * np + i] = ynext[__float_as_int(pts[D * np + i])];
}

// shared memory of the fit: a tile's neighbour lists and, of groups small
// enough, the points and their values
__host__ __device__ inline int fit_points(int d, int P, int kmax) {
    const int most = (kFitBytes - kmax * kT * 2) / ((d + 1) * 4);
    return P < most ? (P + 3) & ~3 : (most > 0 ? most & ~3 : 0);
}
size_t fit_smem(int d, int P, int kmax) {
    return (size_t)kmax * kT * 2 + (size_t)(d + 1) * fit_points(d, P, kmax) * 4;
}

// REF: reference semantics
template <int D, bool REF>
__global__ void __launch_bounds__(kT, 4) k_knn_fit(to_rov_args a, int t) {
    extern __shared__ __align__(16) unsigned char sm_fit[];
    constexpr int NS = fit_sums<D>();
    const int tid = threadIdx.x, Q = a.Q, slot = t - a.slot0, np = fit_points(D, a.P, a.kmax);
    unsigned short* lists = reinterpret_cast<unsigned short*>(sm_fit);     // [kmax][kT]
    float* pts = reinterpret_cast<float*>(sm_fit + (size_t)a.kmax * kT * 2);   // [D + 1][np]
    const int ntiles = a.ntiles[slot], tcap = a.G * ((Q + kT - 1) / kT);
    const int2* tiles = a.tiles + (size_t)slot * tcap;
    to_pdl_next();
    if (blockIdx.x >= ntiles) to_pdl_wait();
    for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
        const int g = tiles[ti].x, start = tiles[ti].y;
        const size_t gs = (size_t)slot * a.G + g;
        const int n = a.npts[gs], k = a.kc[gs];
        const bool live = start + tid < a.gcount[gs];
        const int at = live ? start + tid : start;
        const int qi = a.touched ? a.qlist[gs * Q + at] : at;
        float* out = to_rov_reg_block(a, t, g) + (size_t)a.R * D;
        if (n < 3 || k <= 0) {                 // too few points
            to_pdl_wait();
            if (live) out[qi] = 0.0f;
            continue;
        }
        const size_t tg = (size_t)(slot - a.sel0) * tcap + ti;
        __syncthreads();                       // the last tile is done with
        {
            const uint4* src = reinterpret_cast<const uint4*>(a.nbr + tg * a.kmax * kT);
            uint4* dst = reinterpret_cast<uint4*>(lists);
#pragma unroll 4
            for (int i = tid; i < k * (kT / 8); i += kT) dst[i] = src[i];
        }
        if (n <= np) load_points<D>(a, slot, t, g, np, pts);
        else to_pdl_wait();
        __syncthreads();
        if (!live) continue;
        PairArgs<D> pc = pair_args<D>(a, slot, t, g, qi, a.kthv[tg * kT + tid]);
        pc.nb = lists + tid;
        pc.stride = kT;
        pc.pts = pts;
        pc.np = np;
        pc.many = n > np;
        float tot[NS];
        for (int l = 0; l < 32 && l < k; l += 2) {
            f2 acc[NS];
            pair_sums<D, REF>(pc, l, acc);
#pragma unroll
            for (int e = 0; e < NS; ++e) {
                float a0, a1;
                unpack2(acc[e], a0, a1);
                tot[e] = (l ? tot[e] + a0 : a0) + a1;
            }
        }
        double sums[NS];
#pragma unroll
        for (int e = 0; e < NS; ++e) sums[e] = (double)tot[e];
        out[qi] = to_lsm_solve_compact(D, sums);
    }
}

// The same for few queries a year (a road, a small batch), where a thread's
// walk through all its neighbours is what a year waits for: a CTA of 16
// warps takes 32 queries (lane = query), warp w partials 2w and 2w + 1; the
// partials meet in shared memory, where a thread per (sum, query) adds them
// in order, and the first warp solves.
constexpr int kWide = 512;
constexpr int kWidePts = 3072;
__host__ __device__ inline int wide_points(int P) { return ((P < kWidePts ? P : kWidePts) + 3) & ~3; }
template <int D>
size_t wide_smem(int P, int kmax) {
    return (size_t)32 * fit_sums<D>() * kW * 4 + (size_t)(D + 1) * wide_points(P) * 4 +
           (size_t)kmax * kW * 2;
}

template <int D, bool REF>
__global__ void __launch_bounds__(kWide) k_knn_fit_wide(to_rov_args a, int t) {
    extern __shared__ __align__(16) unsigned char sm_fit[];
    constexpr int NS = fit_sums<D>(), SUB = kT / kW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Q = a.Q, slot = t - a.slot0, np = wide_points(a.P);
    float* part = reinterpret_cast<float*>(sm_fit);                   // [32][NS][kW]
    float* pts = part + 32 * NS * kW;                                 // [D + 1][np]
    unsigned short* lists = reinterpret_cast<unsigned short*>(pts + (D + 1) * np);  // [kmax][kW]
    const int nsub = a.ntiles[slot] * SUB, tcap = a.G * ((Q + kT - 1) / kT);
    const int2* tiles = a.tiles + (size_t)slot * tcap;
    to_pdl_next();
    if (blockIdx.x >= nsub) to_pdl_wait();
    for (int si = blockIdx.x; si < nsub; si += gridDim.x) {
        const int ti = si / SUB, q0 = si % SUB * kW;
        const int g = tiles[ti].x, start = tiles[ti].y + q0;
        const size_t gs = (size_t)slot * a.G + g;
        const int n = a.npts[gs], k = a.kc[gs], cnt = a.gcount[gs] - start;
        if (cnt <= 0) {
            to_pdl_wait();
            continue;
        }
        const bool live = lane < cnt;
        const int at = live ? start + lane : start;
        const int qi = a.touched ? a.qlist[gs * Q + at] : at;
        float* out = to_rov_reg_block(a, t, g) + (size_t)a.R * D;
        if (n < 3 || k <= 0) {                 // too few points
            to_pdl_wait();
            if (live && warp == 0) out[qi] = 0.0f;
            continue;
        }
        const size_t tg = (size_t)(slot - a.sel0) * tcap + ti;
        __syncthreads();                       // the last queries are done with
        for (int i = tid; i < k * 4; i += kWide)      // a row: 32 of the tile's 128
            reinterpret_cast<uint4*>(lists)[i] = reinterpret_cast<const uint4*>(
                a.nbr + (tg * a.kmax + (i >> 2)) * kT + q0)[i & 3];
        if (n <= np) load_points<D>(a, slot, t, g, np, pts);
        else to_pdl_wait();
        __syncthreads();
        PairArgs<D> pc = pair_args<D>(a, slot, t, g, qi, live ? a.kthv[tg * kT + q0 + lane] : 1.0f);
        pc.nb = lists + lane;
        pc.stride = kW;
        pc.pts = pts;
        pc.np = np;
        pc.many = n > np;
        if (live) {
            f2 acc[NS];
            pair_sums<D, REF>(pc, 2 * warp, acc);
#pragma unroll
            for (int e = 0; e < NS; ++e)
                unpack2(acc[e], part[(2 * warp * NS + e) * kW + lane],
                        part[((2 * warp + 1) * NS + e) * kW + lane]);
        }
        __syncthreads();
        for (int i = tid; i < NS * kW; i += kWide) {
            float x = part[i];
#pragma unroll
            for (int l = 1; l < 32; ++l) x = x + part[l * NS * kW + i];
            part[i] = x;
        }
        __syncthreads();
        if (warp == 0 && live) {
            double sums[NS];
#pragma unroll
            for (int e = 0; e < NS; ++e) sums[e] = (double)part[e * kW + lane];
            out[qi] = to_lsm_solve_compact(D, sums);
        }
    }
}

template <int D>
to_status launch_select(to_ctx ctx, const to_rov_args& a, int years) {
    const size_t smem = select_smem(D, a.kmax);
    const auto k = k_knn_rov<D>;
    TO_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    TO_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kT, smem));
    if (per_sm < 1) per_sm = 1;
    const int sms = ctx->sm_count > 0 ? ctx->sm_count : TO_SM_TARGET;
    const int tiles = a.G * ((a.Q + kT - 1) / kT);
    to_prof_begin(ctx, "knn");
    k<<<dim3(tiles < sms * per_sm ? tiles : sms * per_sm, years), kT, smem, ctx->stream>>>(a);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

template <int D, bool REF>
to_status launch_fit(to_ctx ctx, const to_rov_args& a, int t, bool ahead) {
    const int sms = ctx->sm_count > 0 ? ctx->sm_count : TO_SM_TARGET;
    const int tiles = a.G * ((a.Q + kT - 1) / kT);
    // few queries: at most two tiles an SM even if every grid query is
    // fitted.  Whole valuations, wide against not: one road of 10,000 paths
    // (96 tiles) 5.35 against 6.53 ms, one of reference semantics 2.0 against
    // 2.8; eight roads (768 tiles) 4.7 against 4.3, 24 roads 11.6 against 9.6
    const bool wide = tiles <= 2 * sms;
    const size_t smem = wide ? wide_smem<D>(a.P, a.kmax) : fit_smem(D, a.P, a.kmax);
    const auto k = wide ? k_knn_fit_wide<D, REF> : k_knn_fit<D, REF>;
    TO_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    to_prof_begin(ctx, "knn_solve");
    const int units = wide ? tiles * (kT / kW) : tiles;
    TO_CUDA(ctx, to_pdl_launch(ahead, k, units < 16 * sms ? units : 16 * sms, wide ? kWide : kT, smem,
                               ctx->stream, a, t));
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

}  // namespace

namespace to_k {

size_t knn_select_bytes(const to_rov_args& a, int max_roads) {
    // neighbours and k-th distances of one year, every grid query fitted
    return (size_t)max_roads * a.C * ((a.Q + kT - 1) / kT) * kT * ((size_t)a.kmax * 2 + 4);
}

to_status knn_rov_select(to_ctx ctx, const to_rov_args& a, int years) {
    const int d = a.S + 1;
    if (a.kmax > TO_KNN_KMAX)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "k %d exceeds %d", a.kmax, TO_KNN_KMAX);
    switch (d) {
        case 2: return launch_select<2>(ctx, a, years);
        case 3: return launch_select<3>(ctx, a, years);
        case 4: return launch_select<4>(ctx, a, years);
        case 5: return launch_select<5>(ctx, a, years);
    }
    return to_set_error(ctx, TO_ERR_UNSUPPORTED, "regression dimension %d", d);
}

to_status knn_rov_fit(to_ctx ctx, const to_rov_args& a, int t, bool ahead) {
    const int d = a.S + 1;
    if (a.sem == 0) {                          // one species
        if (d != 2) return to_set_error(ctx, TO_ERR_UNSUPPORTED, "reference semantics, %d dimensions", d);
        return launch_fit<2, true>(ctx, a, t, ahead);
    }
    switch (d) {
        case 2: return launch_fit<2, false>(ctx, a, t, ahead);
        case 3: return launch_fit<3, false>(ctx, a, t, ahead);
        case 4: return launch_fit<4, false>(ctx, a, t, ahead);
        default: return launch_fit<5, false>(ctx, a, t, ahead);
    }
}

}  // namespace to_k
