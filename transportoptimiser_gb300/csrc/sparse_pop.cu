// sparse_pop.cu - population Monte Carlo with the migration matrices in
// compressed-column form, resident in shared memory.
//
// The reference multiplies each path's population vector by a CSC matrix
// (dense2Sparse, SimulateGPU.cu:5973-5996; mteKernel :628-635;
// forwardPathKernel :871-922), one thread per path, reading strided global
// memory.  The matrices are very sparse (local migration: 2-5% non-zero,
// ~8 per column on the benchmark grids), so a dense (paths x N)(N x N)
// product would spend >95% of its work on zeros.  Here:
//   * k_pack_csc packs every (road, species, control) matrix once;
//   * a CTA works on a tile of 16, 32 or 64 paths (a lane is one path, or two
//     on packed FP32) and keeps their populations ([patch][lane],
//     conflict-free) and, where they fit, the lists in shared memory for all
//     years; its warps take the destination patches in groups of four, so one
//     Philox call gives the four growth normals a path needs;
//   * each destination sums its non-zeros in ascending origin order with
//     explicit FMAs - the same chain as the dense form (skipped and padding
//     terms are exact zeros), so results stay bit-identical to the oracle;
//   * patch totals use the fixed grouped order ((v0+v1)+v2)+v3, groups
//     ascending.
#include <cstring>

#include "to_internal.cuh"
#include "to_mbar.cuh"
#include "to_pop.cuh"
#include "to_rov.cuh"
#include "to_rov_dev.cuh"
#include "to_sparse.cuh"

namespace {

constexpr int kLanes = 32;

// One CTA per matrix (rs*C + c): row k of the destination-major matrix is
// destination k's column.  Entries > 0 in ascending origin order.  A warp
// per row reads it coalesced: a count pass, a CTA scan of the row counts,
// then a ballot-compaction pass.
__global__ void __launch_bounds__(1024)
k_pack_csc(const float* __restrict__ mmm, int NP, int C, const int* __restrict__ n_patches,
           int cap, int* __restrict__ ptr, uint16_t* __restrict__ idx, float* __restrict__ val,
           int* __restrict__ nnz, int mtx0) {
    const int mtx = mtx0 + blockIdx.x;
    const int rs = mtx / C;
    const int N = n_patches[rs];
    const float* M = mmm + (size_t)mtx * NP * NP;
    int* p = ptr + (size_t)mtx * (NP + 1);
    uint16_t* ix = idx + (size_t)mtx * cap;
    float* vv = val + (size_t)mtx * cap;
    __shared__ int s_cnt[1024 + 1];
    __shared__ int s_w[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int k = warp; k < NP; k += nw) {
        int c = 0;
        if (k < N)
            for (int l0 = 0; l0 < N; l0 += 32) {
                const int l = l0 + lane;
                c += __popc(__ballot_sync(0xffffffffu, l < N && M[(size_t)k * NP + l] > 0.0f));
            }
        if (lane == 0) s_cnt[k] = c;
    }
    __syncthreads();
    // exclusive scan of s_cnt[0..NP) (NP <= 1024: one value per thread)
    const int v = threadIdx.x < NP ? s_cnt[threadIdx.x] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    int wb = 0, tot = 0;
    for (int w = 0; w < nw; ++w) { if (w < warp) wb += s_w[w]; tot += s_w[w]; }
    __syncthreads();
    if (threadIdx.x < NP) s_cnt[threadIdx.x] = wb + x - v;
    if (threadIdx.x == 0) { s_cnt[NP] = tot; nnz[mtx] = (tot <= cap) ? tot : -1; }
    __syncthreads();
    for (int k = threadIdx.x; k <= NP; k += blockDim.x) p[k] = s_cnt[k];
    if (tot > cap) return;
    for (int k = warp; k < N; k += nw) {
        int o = s_cnt[k];
        for (int l0 = 0; l0 < N; l0 += 32) {
            const int l = l0 + lane;
            const float m = (l < N) ? M[(size_t)k * NP + l] : 0.0f;
            const unsigned b = __ballot_sync(0xffffffffu, m > 0.0f);
            if (m > 0.0f) {
                const int q = o + __popc(b & lt);
                ix[q] = (uint16_t)l;
                vv[q] = m;
            }
            o += __popc(b);
        }
    }
}

__device__ __forceinline__ float grouped4(float a, float b, float c, float d) {
    return ((a + b) + c) + d;
}

constexpr int kMaxG = 4;
constexpr int kGmChunk = 16;

// The launch order of the MTE's (road, species): by descending packed
// entries of the used control (ties by index), so the widest models start
// first and the last wave holds the narrow ones.  A thread ranks one against
// all, which a CTA reads 128 at a time (768 models: 35 us by one CTA of 1,024
// threads, 9 us by six of 128).
constexpr int kOrder = 128;

__global__ void __launch_bounds__(kOrder) k_mte_order(int n_rs, int rs0, int C, int c_use,
                                                      const int* __restrict__ nnz, int* order) {
    __shared__ int s_w[kOrder];
    const int tid = threadIdx.x, i = blockIdx.x * kOrder + tid;
    const int w = i < n_rs ? nnz[(size_t)(rs0 + i) * C + c_use] : 0;
    int rank = 0;
    for (int j0 = 0; j0 < n_rs; j0 += kOrder) {
        const int nj = min(kOrder, n_rs - j0);
        __syncthreads();
        if (tid < nj) s_w[tid] = nnz[(size_t)(rs0 + j0 + tid) * C + c_use];
        __syncthreads();
#pragma unroll 8
        for (int j = 0; j < nj; ++j) {
            const int wj = s_w[j];
            rank += (wj > w) || (wj == w && j0 + j < i);
        }
    }
    if (i < n_rs) order[rank] = i;
}

// ---------------------------------------------------------------------------
// Union of the C <= 3 controls' packed columns of one (road, species): one
// CTA; a thread per destination merges its C ascending origin lists (count,
// CTA scan, write).
// ---------------------------------------------------------------------------
constexpr int kNoOrigin = 0xFFFF;                  // a zero term: the row of zeros
__device__ __forceinline__ int union_step(const int* b, const int* e, const uint16_t* const* ix,
                                          int C, int* pos) {
    int lo = 0x7fffffff;
    for (int c = 0; c < C; ++c)
        if (pos[c] < e[c] && (int)ix[c][pos[c]] < lo) lo = ix[c][pos[c]];
    return lo;
}

__global__ void __launch_bounds__(256)
k_union_csc(int NP, int C, const int* __restrict__ n_patches, to_csc csc) {
    const int rs = blockIdx.x;
    const int N = n_patches[rs];
    __shared__ int s_tmp[32];
    int* up = csc.uptr + (size_t)rs * (NP + 1);
    const uint16_t* ix[3];
    const float* vv[3];
    bool ok = true;
    for (int c = 0; c < C; ++c) {
        const size_t mtx = (size_t)rs * C + c;
        ix[c] = csc.idx + mtx * csc.cap;
        vv[c] = csc.val + mtx * csc.cap;
        ok = ok && csc.nnz[mtx] >= 0;
    }
    if (!ok) {                                    // a control above its capacity
        if (threadIdx.x == 0) csc.unnz[rs] = -1;
        return;
    }
    // pass 1: union size of each column; a thread takes a run of columns
    const int chunk = (NP + (int)blockDim.x - 1) / (int)blockDim.x;
    const int k0 = (int)threadIdx.x * chunk, k1 = min(NP, k0 + chunk);
    int cnt = 0;
    for (int k = k0; k < k1; ++k) {
        int b[3], e[3], pos[3];
        for (int c = 0; c < C; ++c) {
            const int* p = csc.ptr + ((size_t)rs * C + c) * (NP + 1);
            b[c] = pos[c] = k < N ? p[k] : 0;
            e[c] = k < N ? p[k + 1] : 0;
        }
        int n = 0;
        for (;;) {
            const int lo = union_step(b, e, ix, C, pos);
            if (lo == 0x7fffffff) break;
            for (int c = 0; c < C; ++c) if (pos[c] < e[c] && (int)ix[c][pos[c]] == lo) ++pos[c];
            ++n;
        }
        n = (n + 1) & ~1;                          // an even number, the last a zero term
        up[k] = n;
        cnt += n;
    }
    // CTA exclusive scan of the per-thread totals
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_tmp[warp] = x;
    __syncthreads();
    int base = 0, total = 0;
    for (int w = 0; w < nw; ++w) { if (w < warp) base += s_tmp[w]; total += s_tmp[w]; }
    base += x - cnt;
    for (int k = k0; k < k1; ++k) { const int n = up[k]; up[k] = base; base += n; }
    if (threadIdx.x == 0) {
        up[NP] = total;
        csc.unnz[rs] = total <= csc.ucap ? total : -1;
    }
    if (total > csc.ucap) return;
    // pass 2: the entries
    int4* out = csc.uent + (size_t)rs * csc.ucap;
    for (int k = k0; k < k1; ++k) {
        int b[3], e[3], pos[3];
        for (int c = 0; c < C; ++c) {
            const int* p = csc.ptr + ((size_t)rs * C + c) * (NP + 1);
            b[c] = pos[c] = k < N ? p[k] : 0;
            e[c] = k < N ? p[k + 1] : 0;
        }
        int q = up[k];
        for (;;) {
            const int lo = union_step(b, e, ix, C, pos);
            if (lo == 0x7fffffff) break;
            float v[3] = {0.0f, 0.0f, 0.0f};
            for (int c = 0; c < C; ++c)
                if (pos[c] < e[c] && (int)ix[c][pos[c]] == lo) { v[c] = vv[c][pos[c]]; ++pos[c]; }
            out[q++] = make_int4(lo, __float_as_int(v[0]), __float_as_int(v[1]),
                                 __float_as_int(v[2]));
        }
        if ((q - up[k]) & 1) out[q] = make_int4(kNoOrigin, 0, 0, 0);
    }
}

// ---------------------------------------------------------------------------
// ROV forward paths on the union columns (C <= 3 controls), two paths a
// lane.  Persistent: one CTA an SM, taking 64-path tiles of the roads from a
// counter.  Bound by instruction issue (and shared-memory latency below it),
// so the work is laid out for few instructions a path:
//  * a row of the populations holds two paths a lane, so that an entry of a
//    destination's list, its address and the loop around it serve both, and
//    the growth, the sums and the arithmetic of the normals run on packed
//    pairs (to_f2.cuh);
//  * the growth normals' Philox blocks share what does not change between
//    groups, years or paths and read their round keys from the constant bank;
//  * the year's populations are read from one buffer and written to another,
//    so a warp takes groups of four destinations from a shared counter,
//    widest first, and a year has one barrier, split: a warp that is done
//    arrives, draws the normals of its own first group of the next year and
//    only then waits (39.1 -> 37.5 ms).  Where two buffers do not fit
//    beside the lists, the other one is in global memory (it stays in L2)
//    and copied back after the barrier.  What the year's end needs
//    summed over the groups - each control's migrated totals, in group order -
//    goes through a small global scratch (it stays in L2) and is added up
//    during the next year by whichever warp takes it, like the total of the
//    populations: no warp waits for a chain of 80 additions.
// 256 roads, 768 paths, 3 species, 50 years: 50.4 -> 37.5 ms (one path a
// lane before), 65% of the issue slots, the FMA pipe at about the same.  The values
// are those of k_rov_forward_sparse bit for bit: every group's arithmetic
// and every sum's order is unchanged, only who computes it.
// ---------------------------------------------------------------------------
constexpr int kPairPaths = 64;

// shared memory of one (road, species): with both populations buffers, or
// with the next year's in global memory
__host__ __device__ inline size_t pair_bytes(int N4, int nu, bool two) {
    return (size_t)((nu + 1) & ~1) * 16 + (size_t)(two ? 2 : 1) * (N4 + 1) * kLanes * 8 +
           (size_t)N4 * 16 + (size_t)kGmChunk * 3 * kPairPaths * 4 + (size_t)2 * kLanes * 8 +
           (size_t)(N4 + 4 + N4 / 4 + 4) * 4;
}
constexpr int kPairStatic = 3072;          // static shared memory and slack
constexpr int kPairThreads = 1024;         // 512, 640 and 768: 39.9, 39.7 and 40.3 ms where 1024 takes 37.5

template <bool REF>
__global__ void __launch_bounds__(kPairThreads, 1)
k_rov_forward_union(to_rov_args a, to_csc csc, int smem) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    __shared__ int s_item, s_grab[2];
    __shared__ to_bm_tables s_tab;
    __shared__ __align__(8) uint64_t s_bar;    // end of a year: an arrival a warp
    const int C = a.C, Y = a.Y, P = a.P, S = a.S;
    const size_t PT = (size_t)a.PT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tiles = (P + kPairPaths - 1) / kPairPaths, items = tiles * a.nr * S;
    const int ngcap = a.np / 4;
    f2* part = a.fwd_part + (size_t)blockIdx.x * 2 * C * ngcap * kLanes;   // [2][C][ngcap][32]
    to_bm_load(s_tab);                         // before the barriers below
    if (tid == 0) to_mbar::init(&s_bar, kPairThreads / 32);
    uint32_t phase = 0;
    for (;;) {
        if (tid == 0) s_item = atomicAdd(a.fwd_next, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();                       // read before it is written again
        if (item >= items) break;
        const int s = item % S, rd = item / S / tiles, rs = rd * S + s;
        const int path0 = (item / S - rd * tiles) * kPairPaths + lane, path1 = path0 + kLanes;
        const bool live0 = path0 < P, live1 = path1 < P;
        const size_t gp = (size_t)rd * P + path0;
        const int N = a.n_patches[rs], nu = csc.unnz[rs];
        const int N4 = (N + 3) & ~3, NGr = N4 >> 2;
        if (nu < 0 || N > a.ne || pair_bytes(N4, nu, false) > (size_t)smem) {
            // outside the shape this launch was planned for: flag, no result
            if (tid == 0 && a.flags) atomicExch(a.flags, TO_DEVERR_PLAN);
            for (int t = warp; t <= Y; t += blockDim.x >> 5) {
                float* out = a.totalPops + ((size_t)s * (Y + 1) + t) * PT + gp;
                if (live0) out[0] = NAN;
                if (live1) out[kLanes] = NAN;
            }
            continue;
        }
        const uint32_t road = (uint32_t)a.road_ids[rd];
        const uint32_t stream_road = TO_STREAM_GROWTH | (road << 8);
        to_path_stream ps0, ps1;
        to_stream_path(ps0, (uint32_t)path0);
        to_stream_path(ps1, (uint32_t)path1);
        int4* ue = reinterpret_cast<int4*>(sm_raw);                    // [nu]
        f2* cur = reinterpret_cast<f2*>(ue + ((nu + 1) & ~1));         // [N4 + 1][32], row N4 zero
        const bool two = pair_bytes(N4, nu, true) <= (size_t)smem;
        f2* nxt = two ? cur + (size_t)(N4 + 1) * kLanes : cur;         // the same
        f2* far = a.fwd_far + (size_t)blockIdx.x * a.np * kLanes;      // [N4][32] otherwise
        float4* capr = reinterpret_cast<float4*>(nxt + (size_t)(N4 + 1) * kLanes);  // [N4]
        // draws of the growth mean, then [0] the means and [1] the controls
        float* xs = reinterpret_cast<float*>(capr + N4);               // [kGmChunk][3][64]
        f2* tot = reinterpret_cast<f2*>(xs + kGmChunk * 3 * kPairPaths);   // [2][32]
        int* uptr = reinterpret_cast<int*>(tot + 2 * kLanes);          // [N4 + 1]
        int* order = uptr + N4 + 4;                                    // [NGr]
        const float* sp = a.params + 8 * s;
        const float* ip = a.init_pops + (size_t)rs * a.np;
        for (int q = tid; q < (N4 + 1) * kLanes; q += blockDim.x) {
            const int k = q / kLanes;
            cur[q] = both2(k < N ? ip[k] : 0.0f);
            if (k == N4) nxt[q] = both2(0.0f);
        }
        for (int k = tid; k < N4; k += blockDim.x) {
            const float cp = a.caps[(size_t)rs * a.np + k], nr = -(1.0f / cp);
            capr[k] = make_float4(cp, cp, nr, nr);     // capacity, minus its reciprocal
        }
        for (int k = tid; k <= N4; k += blockDim.x)
            uptr[k] = csc.uptr[(size_t)rs * (a.np + 1) + k];
        for (int e = tid; e < nu; e += blockDim.x) {
            int4 v = csc.uent[(size_t)rs * csc.ucap + e];
            // origin -> row byte offset
            v.x = (v.x == kNoOrigin ? N4 : v.x) * kLanes * (int)sizeof(f2);
            ue[e] = v;
        }
        if (tid < 2) s_grab[tid] = 0;
        __syncthreads();
        // the groups in descending order of entries (ties: lower group first)
        for (int gq = tid; gq < NGr; gq += blockDim.x) {
            const int w = uptr[4 * gq + 4] - uptr[4 * gq];
            int rank = 0;
            for (int u = 0; u < NGr; ++u) {
                const int wu = uptr[4 * u + 4] - uptr[4 * u];
                rank += (wu > w) || (wu == w && u < gq);
            }
            order[rank] = gq;
        }
        const float jp = REF ? sp[5] : sp[6];
        const float s5 = sp[5] * sp[5];
        const f2 s7 = both2(sp[7]), one = both2(1.0f), mone = both2(-1.0f);
        float gmean = sp[0];                           // of path `tid` of the tile (tid < 64)
        f2 z[4];                                       // normals of the group worked on
        // totals of the populations at the start of year t
        auto total = [&](int t) {
            f2 tt = both2(0.0f);
#pragma unroll 4
            for (int grp = 0; grp < NGr; ++grp) {
                const f2* v = cur + (size_t)grp * 4 * kLanes + lane;
                tt = add2(tt, add2(add2(add2(v[0], v[kLanes]), v[2 * kLanes]), v[3 * kLanes]));
            }
            tot[(t & 1) * kLanes + lane] = tt;
            float t0, t1;
            unpack2(tt, t0, t1);
            float* out = a.totalPops + ((size_t)s * (Y + 1) + t) * PT + gp;
            if (live0) out[0] = t0;
            if (live1) out[kLanes] = t1;
        };
        // control c's share of the animals left after the migration of year t
        auto at_risk = [&](int t, int c) {
            const f2* v = part + ((size_t)(t & 1) * C + c) * ngcap * kLanes + lane;
            f2 tt = both2(0.0f);
#pragma unroll 8
            for (int grp = 0; grp < NGr; ++grp) tt = add2(tt, v[(size_t)grp * kLanes]);
            float t0, t1, p0, p1;
            unpack2(tt, t0, t1);
            unpack2(tot[(t & 1) * kLanes + lane], p0, p1);
            float* out = a.aars + (((size_t)s * C + c) * Y + t) * PT + gp;
            if (live0) out[0] = t0 / p0;
            if (live1) out[kLanes] = t1 / p1;
        };
        auto normals = [&](int grp) {
            to_normal4x2(ps0, ps1,
                         to_stream_group((uint32_t)((s * N4) >> 2) + grp, stream_road, a.rk),
                         a.rk, s_tab, z);
        };
        auto next_year = [&](int t) {
            to_stream_year(ps0, (uint32_t)t, a.rk);
            to_stream_year(ps1, (uint32_t)t, a.rk);
        };
        for (int t = 0; t < Y; ++t) {
            if (t % kGmChunk == 0) {
                // the next years' growth-mean draws, one thread each
                const int nc = min(kGmChunk, Y - t);
                for (int q = tid; q < nc * 3 * kPairPaths; q += blockDim.x) {
                    const int yy = q / (3 * kPairPaths), r = q - yy * 3 * kPairPaths;
                    const int which = r / kPairPaths, i = r - which * kPairPaths;
                    const uint32_t pth = (uint32_t)(path0 - lane + i);
                    const int ty = t + yy;
                    float v;
                    if (which == 0) {
                        v = (to_uniform1(a.seed, TO_STREAM_SP_JUMP, road, pth, ty, s) < jp)
                                ? 1.0f : 0.0f;
                    } else if (which == 1) {
                        v = to_normal1(a.seed, TO_STREAM_SP_BROWNIAN, road, pth, ty, s) * sp[2];
                    } else {
                        const float zj =
                            to_normal1(a.seed, TO_STREAM_SP_JUMPSIZE, road, pth, ty, s);
                        const float jsz = REF ? (zj * s5 - s5 / 2.0f) : (zj * sp[5] - s5 / 2.0f);
                        v = to_expf(jsz) - 1.0f;
                    }
                    xs[q] = v;
                }
                __syncthreads();
                // the growth means do not depend on the populations: the
                // years' recursion, a thread a path
                if (tid < kPairPaths) {
                    const int pth = path0 - lane + tid;
                    int ctl[kGmChunk];
#pragma unroll
                    for (int yy = 0; yy < kGmChunk; ++yy)
                        ctl[yy] = (yy < nc && pth < P)
                                      ? a.controls[(size_t)(t + yy) * PT + (size_t)rd * P + pth] : 0;
#pragma unroll
                    for (int yy = 0; yy < kGmChunk; ++yy)
                        if (yy < nc) {
                            float* x = xs + yy * 3 * kPairPaths + tid;
                            gmean = gmean + sp[4] * (sp[1] - gmean) * a.dt + gmean * x[kPairPaths] +
                                    x[2 * kPairPaths] * gmean * x[0];
                            x[0] = gmean;
                            x[kPairPaths] = __int_as_float(ctl[yy]);
                            if (a.gmY && pth < P)
                                a.gmY[((size_t)(t + yy) * S + s) * P + pth] = gmean;
                        }
                }
                __syncthreads();
            }
            const float* xt = xs + (t % kGmChunk) * 3 * kPairPaths + lane;
            const float g0 = xt[0], g1 = xt[kLanes];
            const int c0 = __float_as_int(xt[kPairPaths]), c1 = __float_as_int(xt[kPairPaths + kLanes]);
            if (a.popsY)
                for (int q = tid; q < a.ne * kPairPaths; q += blockDim.x) {
                    const int k = q / kPairPaths, i = q - k * kPairPaths;
                    const int pth = path0 - lane + i;
                    if (pth < P)
                        a.popsY[(((size_t)t * S + s) * a.ne + k) * P + pth] =
                            k < N4 ? reinterpret_cast<const float*>(
                                         cur + (size_t)k * kLanes + (i & 31))[i >> 5] : 0.0f;
                }
            const f2 g = pack2(g0, g1);
            const unsigned char* curb = reinterpret_cast<const unsigned char*>(cur + lane);
            f2* py = part + (size_t)(t & 1) * C * ngcap * kLanes + lane;
            // the year's work: a group each, then from the counter the totals and
            // last year's shares, then the other groups
            if (t == 0) {
                next_year(0);
                if (warp < NGr) normals(order[warp]);
            }
            const int lead = t ? 1 + C : 1;
            int* gc = s_grab + (t & 1);
            bool own = warp < NGr;
            for (;;) {
                int grp;
                if (own) {
                    grp = order[warp];
                    own = false;
                } else {
                    int i = 0;
                    if (lane == 0) i = atomicAdd(gc, 1);
                    i = __shfl_sync(0xffffffffu, i, 0) - lead;
                    if (i < 0) {
                        if (i == -1) total(t);
                        else at_risk(t - 1, -2 - i);
                        continue;
                    }
                    i += kPairThreads / 32;
                    if (i >= NGr) break;
                    grp = order[i];
                    normals(grp);
                }
                // the group's column pointers: one 16-byte load and one word
                const int4 u4 = reinterpret_cast<const int4*>(uptr)[grp];
                const int ub[5] = {u4.x, u4.y, u4.z, u4.w, uptr[grp * 4 + 4]};
                f2 m0, m1, m2;             // the group's migrated sums by control
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int k = grp * 4 + j;
                    f2 q0 = 0ull, q1 = 0ull, q2 = 0ull;        // migrated, by control
                    const int e1 = ub[j + 1];
#pragma unroll 2
                    for (int e = ub[j]; e < e1; e += 2) {      // an even number of terms
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int4 en = ue[e + u];
                            const f2 x = *reinterpret_cast<const f2*>(curb + en.x);
                            q0 = fma2(x, both2(__int_as_float(en.y)), q0);
                            q1 = fma2(x, both2(__int_as_float(en.z)), q1);
                            q2 = fma2(x, both2(__int_as_float(en.w)), q2);
                        }
                    }
                    float a00, a01, a10, a11, a20, a21;
                    unpack2(q0, a00, a01);
                    unpack2(q1, a10, a11);
                    unpack2(q2, a20, a21);
                    m0 = j ? add2(m0, q0) : q0;
                    m1 = j ? add2(m1, q1) : q1;
                    m2 = j ? add2(m2, q2) : q2;
                    const f2 mv = pack2(c0 == 0 ? a00 : (c0 == 1 ? a10 : a20),
                                        c1 == 0 ? a01 : (c1 == 1 ? a11 : a21));
                    f2 gr;
                    if (REF) {
                        // scalar: ptxas joins a packed multiply and add
                        float z0, z1;
                        unpack2(z[j], z0, z1);
                        gr = pack2(g0 + z0 * sp[7], g1 + z1 * sp[7]);
                    } else {
                        gr = fma2(mul2(s7, z[j]), g, g);
                    }
                    // (gr (cap - mv)) / cap as to_div_rcp, with minus the
                    // reciprocal: minus the quotient, the same bits
                    const ulonglong2 cr = *reinterpret_cast<const ulonglong2*>(capr + k);
                    const f2 x = mul2(gr, fma2(mv, mone, cr.x));
                    const f2 nq = mul2(x, cr.y);
                    f2 nd = fma2(fma2(nq, cr.x, x), cr.y, nq);
                    f2 v;
                    if (REF) {
                        // and / 100, the same way
                        const f2 q = mul2(nd, both2(0.01f));
                        const f2 r = fma2(neg2(q), both2(100.0f), nd);
                        nd = fma2(r, both2(0.01f), q);
                        v = mul2(mv, fma2(nd, mone, one));
                    } else {
                        float v0, v1;
                        unpack2(mul2(mv, fma2(nd, mone, one)), v0, v1);
                        v = pack2(fmaxf(v0, 0.0f), fmaxf(v1, 0.0f));
                    }
                    if (two) nxt[k * kLanes + lane] = v;
                    else far[k * kLanes + lane] = v;
                }
                py[(size_t)grp * kLanes] = m0;
                if (C > 1) py[((size_t)ngcap + grp) * kLanes] = m1;
                if (C > 2) py[((size_t)2 * ngcap + grp) * kLanes] = m2;
            }
            // last used in the year before the last barrier
            if (tid == 0) s_grab[(t + 1) & 1] = 0;
            // done: while the others finish, the normals of next year's own group
            __syncwarp();
            if (lane == 0) to_mbar::arrive(&s_bar);
            if (t + 1 < Y) {
                next_year(t + 1);
                if (warp < NGr) normals(order[warp]);
            }
            if (!to_mbar::wait(&s_bar, phase)) {
                if (a.flags) atomicExch(a.flags, TO_DEVERR_SPIN);
                return;
            }
            phase ^= 1u;
            if (two) {
                f2* tmp = cur;
                cur = nxt;
                nxt = tmp;
            } else {
#pragma unroll 4
                for (int q = tid; q < N4 * kLanes; q += blockDim.x) cur[q] = far[q];
                __syncthreads();
            }
        }
        if (warp == 0) total(Y);
        else if (warp <= C && Y > 0) at_risk(Y - 1, warp - 1);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// MTE (mteKernel :595-717).  Persistent, the layout of k_rov_forward_union:
// tiles of 64 paths (two a lane, packed) or 32 from a counter, the (road,
// species) widest first (k_mte_order), a warp's own group of four
// destinations and then others from a counter, one split barrier a year with
// the next year's normals drawn behind it.  Bound by instruction issue (67%
// of the slots, 725 instructions a group of 64 paths before the lists were
// laid out by steps), and by a year's latency where there are few tiles.  So
// a group's four lists run together: a step holds two entries of each
// destination, the short ones padded by zero terms from a row of zeros, so
// that there is one loop a group and eight gathers in flight.
// 40,000 paths, 2 species of 115 patches, 50 years: 1.93 -> 1.50 ms (one CTA
// an SM with the next year's values in registers and two barriers a year
// before); 256 roads of 3 species, 64 paths: 2.86 -> 2.53 ms.
// The values do not depend on which warp computes a group.
// ---------------------------------------------------------------------------
// a lane's paths and the arithmetic on them: two (packed) or one
template <class V> struct to_lane;
template <> struct to_lane<f2> {
    static constexpr int paths = 2;
    struct __align__(16) cap { f2 v, nr; };        // capacity, minus its reciprocal
    to_path_stream ps0, ps1;
    __device__ __forceinline__ void path(uint32_t p) {
        to_stream_path(ps0, p);
        to_stream_path(ps1, p + kLanes);
    }
    __device__ __forceinline__ void year(uint32_t t, const to_round_keys& rk) {
        to_stream_year(ps0, t, rk);
        to_stream_year(ps1, t, rk);
    }
    __device__ __forceinline__ void normals(const to_group_stream& g, const to_round_keys& rk,
                                            const to_bm_tables& tab, f2 (&z)[4]) const {
        to_normal4x2(ps0, ps1, g, rk, tab, z);
    }
    static __device__ __forceinline__ f2 load(const float* x) { return pack2(x[0], x[kLanes]); }
    static __device__ __forceinline__ f2 all(float v) { return both2(v); }
    static __device__ __forceinline__ f2 add(f2 a, f2 b) { return add2(a, b); }
    static __device__ __forceinline__ f2 mul(f2 a, f2 b) { return mul2(a, b); }
    static __device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) { return fma2(a, b, c); }
    static __device__ __forceinline__ void store(float* out, int live, f2 v) {
        float v0, v1;
        unpack2(v, v0, v1);
        if (live > 0) out[0] = v0;
        if (live > kLanes) out[kLanes] = v1;
    }
};
template <> struct to_lane<float> {
    static constexpr int paths = 1;
    struct __align__(8) cap { float v, nr; };
    to_path_stream ps;
    __device__ __forceinline__ void path(uint32_t p) { to_stream_path(ps, p); }
    __device__ __forceinline__ void year(uint32_t t, const to_round_keys& rk) {
        to_stream_year(ps, t, rk);
    }
    __device__ __forceinline__ void normals(const to_group_stream& g, const to_round_keys& rk,
                                            const to_bm_tables& tab, float (&z)[4]) const {
        const to_u32x4 w = to_stream_words(ps, g, rk);
        f2 c, s;                                   // of both Box-Muller pairs
        to_box_muller2(w.v[0], w.v[1], w.v[2], w.v[3], tab, c, s);
        unpack2(c, z[0], z[2]);
        unpack2(s, z[1], z[3]);
    }
    static __device__ __forceinline__ float load(const float* x) { return x[0]; }
    static __device__ __forceinline__ float all(float v) { return v; }
    static __device__ __forceinline__ float add(float a, float b) { return a + b; }
    static __device__ __forceinline__ float mul(float a, float b) { return a * b; }
    static __device__ __forceinline__ float fma(float a, float b, float c) { return fmaf(a, b, c); }
    static __device__ __forceinline__ void store(float* out, int live, float v) {
        if (live > 0) out[0] = v;
    }
};

// shared memory of one (road, species) of N4 destinations: its lists (`list`
// steps, 0 if they stay in global memory) and one or two population buffers
__host__ __device__ inline size_t mte_bytes(int N4, int list, bool two, int paths) {
    return (size_t)kGmChunk * 3 * kLanes * paths * 4 + (size_t)N4 * 8 * paths +
           (size_t)((N4 + 4 + 2 * (N4 / 4 + 1) + 3) & ~3) * 4 +
           (size_t)(two ? 2 : 1) * (N4 + 1) * kLanes * 4 * paths + (size_t)list * 64;
}

template <class V>
__global__ void __launch_bounds__(kPairThreads, 1)
k_mte_sparse(to_mte_args a, to_csc csc, to_round_keys rk, int n_rs, int smem, bool far_ok) {
    using L = to_lane<V>;
    constexpr int PW = kLanes * L::paths;      // paths of a tile
    extern __shared__ __align__(16) unsigned char sm_raw[];
    __shared__ int s_item, s_steps, s_grab[2];
    __shared__ to_bm_tables s_tab;
    __shared__ __align__(8) uint64_t s_bar;    // end of a year: an arrival a warp
    const int Y = a.n_years, P = a.n_paths, NP = a.npad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, W = blockDim.x >> 5;
    const int tiles = (P + PW - 1) / PW, items = tiles * n_rs;
    int* next = a.order_buf + n_rs;
    to_bm_load(s_tab);                         // before the barriers below
    if (tid == 0) to_mbar::init(&s_bar, W);
    uint32_t phase = 0;
    for (;;) {
        if (tid == 0) s_item = atomicAdd(next, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();                       // read before it is written again
        if (item >= items) break;
        const int rq = item / tiles, rs = a.rs0 + (a.order ? a.order[rq] : rq);
        const int road = rs / a.S, s = rs - road * a.S;
        const int path0 = (item - rq * tiles) * PW + lane;
        const int mtx = rs * a.C + a.c_use;
        const int N = a.n_patches[rs], nnz = csc.nnz[mtx];
        const int N4 = (N + 3) & ~3, NGr = N4 >> 2;
        if (nnz < 0 || N > a.npe || mte_bytes(N4, 0, !far_ok, L::paths) > (size_t)smem) {
            // outside the shape this launch was planned for: flag, no result
            if (tid == 0 && a.flags) atomicExch(a.flags, TO_DEVERR_PLAN);
            if (warp == 0) L::store(a.end_pops + (size_t)rs * P + path0, P - path0, L::all(NAN));
            continue;
        }
        const uint32_t road_id = (uint32_t)(a.road0 + road);
        const uint32_t stream_road = TO_STREAM_GROWTH | (road_id << 8);
        L lp;
        lp.path((uint32_t)path0);
        const float* sp = a.params + 8 * s;
        const float* ip = a.init_pops + (size_t)rs * NP;
        const int* gptr = csc.ptr + (size_t)mtx * (NP + 1);
        const uint16_t* gidx = csc.idx + (size_t)mtx * csc.cap;
        const float* gval = csc.val + (size_t)mtx * csc.cap;

        // draws of the growth mean, then [0] the means
        float* xs = reinterpret_cast<float*>(sm_raw);                  // [kGmChunk][3][PW]
        auto* capr = reinterpret_cast<typename L::cap*>(xs + kGmChunk * 3 * PW);   // [N4]
        int* cptr = reinterpret_cast<int*>(capr + N4);                 // [N4 + 1]
        int* order = cptr + N4 + 4;                                    // [NGr]
        int* start = order + NGr + 1;                                  // [NGr + 1] first step
        V* cur = reinterpret_cast<V*>(cptr + ((N4 + 4 + 2 * (NGr + 1) + 3) & ~3));
        for (int k = tid; k < N4; k += blockDim.x) {
            const float cp = a.caps[(size_t)rs * NP + k];
            capr[k].v = L::all(cp);
            capr[k].nr = L::all(-(1.0f / cp));
        }
        for (int k = tid; k <= N4; k += blockDim.x) cptr[k] = gptr[k];
        for (int q = tid; q < (N4 + 1) * kLanes; q += blockDim.x) {    // row N4 stays zero
            const int k = q / kLanes;
            cur[q] = L::all(k < N ? ip[k] : 0.0f);
        }
        if (tid < 2) s_grab[tid] = 0;
        __syncthreads();
        // the groups in descending order of entries (ties: lower group first)
        for (int gq = tid; gq < NGr; gq += blockDim.x) {
            const int w = cptr[4 * gq + 4] - cptr[4 * gq];
            int rank = 0;
            for (int u = 0; u < NGr; ++u) {
                const int wu = cptr[4 * u + 4] - cptr[4 * u];
                rank += (wu > w) || (wu == w && u < gq);
            }
            order[rank] = gq;
        }
        if (warp == W - 1) {                   // the groups' first steps, 32 groups a scan
            int base = 0;
            for (int g0 = 0; g0 < NGr; g0 += 32) {
                const int gq = g0 + lane;
                int n = 0;
                if (gq < NGr)
                    for (int j = 0; j < 4; ++j) n = max(n, cptr[4 * gq + j + 1] - cptr[4 * gq + j]);
                n = (n + 1) >> 1;
                int x = n;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (gq < NGr) start[gq] = base + x - n;
                base += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) start[NGr] = s_steps = base;
        }
        __syncthreads();
        const int list = s_steps;
        bool two = true, near = true;
        if (mte_bytes(N4, list, true, L::paths) > (size_t)smem) {
            two = !far_ok;
            near = far_ok && mte_bytes(N4, list, false, L::paths) <= (size_t)smem;
        }
        V* nxt = two ? cur + (size_t)(N4 + 1) * kLanes : cur;
        V* far = reinterpret_cast<V*>(a.far_buf) + (size_t)blockIdx.x * a.npe * kLanes;
        int4* ent = reinterpret_cast<int4*>(nxt + (size_t)(N4 + 1) * kLanes);
        if (two)
            for (int q = tid; q < kLanes; q += blockDim.x) nxt[(size_t)N4 * kLanes + q] = L::all(0.0f);
        if (near)
            for (int gq = warp; gq < NGr; gq += W) {
                const int s0 = start[gq], n8 = (start[gq + 1] - s0) * 8;
                int2* en = reinterpret_cast<int2*>(ent + (size_t)s0 * 4);
                for (int q = lane; q < n8; q += 32) {  // [step][destination][2]
                    const int j = (q >> 1) & 3, e = cptr[4 * gq + j] + 2 * (q >> 3) + (q & 1);
                    en[q] = e < cptr[4 * gq + j + 1]
                                ? make_int2(gidx[e] * kLanes * (int)sizeof(V), __float_as_int(gval[e]))
                                : make_int2(N4 * kLanes * (int)sizeof(V), 0);
                }
            }
        const float s5 = sp[5] * sp[5];
        // a species without jumps: their indicator is 0 and their factor
        // finite, so that their term is 0 whatever is drawn
        const bool jumps = sp[6] > 0.0f || !(fabsf(sp[5]) <= 1.0f);
        const V s7 = L::all(sp[7]), one = L::all(1.0f), mone = L::all(-1.0f);
        float gmean = sp[0];                           // of path `tid` of the tile (tid < PW)
        V z[4];                                        // normals of the group worked on
        auto normals = [&](int grp) {
            lp.normals(to_stream_group((uint32_t)((s * N4) >> 2) + grp, stream_road, rk), rk, s_tab, z);
        };
        for (int t = 0; t < Y; ++t) {
            if (t % kGmChunk == 0) {
                // the next years' growth-mean draws, one thread each
                const int nc = min(kGmChunk, Y - t);
                for (int q = tid; q < nc * 3 * PW; q += blockDim.x) {
                    const int yy = q / (3 * PW), r = q - yy * 3 * PW;
                    const int which = r / PW, i = r - which * PW;
                    const uint32_t pth = (uint32_t)(path0 - lane + i);
                    const int ty = t + yy;
                    float v = 0.0f;
                    if (which == 1) {
                        v = to_normal1(a.seed, TO_STREAM_SP_BROWNIAN, road_id, pth, ty, s) * sp[2];
                    } else if (jumps) {
                        if (which == 0) {
                            v = (to_uniform1(a.seed, TO_STREAM_SP_JUMP, road_id, pth, ty, s) < sp[6])
                                    ? 1.0f : 0.0f;
                        } else {
                            const float zj =
                                to_normal1(a.seed, TO_STREAM_SP_JUMPSIZE, road_id, pth, ty, s);
                            const float jsz =
                                (a.sem == 0) ? (zj * s5 - s5 / 2.0f) : (zj * sp[5] - s5 / 2.0f);
                            v = to_expf(jsz) - 1.0f;
                        }
                    }
                    xs[q] = v;
                }
                __syncthreads();
                // the growth means do not depend on the populations: the
                // years' recursion, a thread a path
                if (tid < PW)
#pragma unroll 4
                    for (int yy = 0; yy < nc; ++yy) {
                        float* x = xs + yy * 3 * PW + tid;
                        gmean = gmean + sp[4] * (sp[1] - gmean) * a.dt + gmean * x[PW] +
                                x[2 * PW] * gmean * x[0];
                        x[0] = gmean;
                    }
                __syncthreads();
            }
            const V g = L::load(xs + (t % kGmChunk) * 3 * PW + lane);
            const unsigned char* curb = reinterpret_cast<const unsigned char*>(cur + lane);
            V* dst = (two ? nxt : far) + lane;
            const bool migrated = a.sem == 0 && t == Y - 1;    // what the end population sums
            if (t == 0) {
                lp.year(0u, rk);
                if (warp < NGr) normals(order[warp]);
            }
            // a group a warp, the rest from the counter
            int* gc = s_grab + (t & 1);
            for (int i = warp; i < NGr;) {
                const int grp = order[i];
                if (i != warp) normals(grp);
                V q[4] = {};                           // migrated
                if (near) {
                    const int4* en = ent + (size_t)start[grp] * 4;
                    for (const int4* e1 = ent + (size_t)start[grp + 1] * 4; en < e1; en += 4) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int4 e = en[j];
                            q[j] = L::fma(*reinterpret_cast<const V*>(curb + e.x),
                                          L::all(__int_as_float(e.y)), q[j]);
                            q[j] = L::fma(*reinterpret_cast<const V*>(curb + e.z),
                                          L::all(__int_as_float(e.w)), q[j]);
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        for (int e = cptr[grp * 4 + j]; e < cptr[grp * 4 + j + 1]; ++e)
                            q[j] = L::fma(cur[gidx[e] * kLanes + lane], L::all(gval[e]), q[j]);
                }
                if (migrated)
                    dst[(size_t)grp * 4 * kLanes] = L::add(L::add(L::add(q[0], q[1]), q[2]), q[3]);
                else
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int k = grp * 4 + j;
                        const V gr = L::fma(L::mul(s7, z[j]), g, g);
                        // (gr (cap - q)) / cap as to_div_rcp, with minus the
                        // reciprocal: minus the quotient, the same bits
                        const typename L::cap cr = capr[k];
                        const V x = L::mul(gr, L::fma(q[j], mone, cr.v));
                        const V nq = L::mul(x, cr.nr);
                        const V nd = L::fma(L::fma(nq, cr.v, x), cr.nr, nq);
                        dst[k * kLanes] = L::mul(q[j], L::fma(nd, mone, one));
                    }
                if (lane == 0) i = atomicAdd(gc, 1);
                i = __shfl_sync(0xffffffffu, i, 0) + W;
            }
            // last used in the year before the last barrier
            if (tid == 0) s_grab[(t + 1) & 1] = 0;
            // done: while the others finish, the normals of next year's own group
            __syncwarp();
            if (lane == 0) to_mbar::arrive(&s_bar);
            if (t + 1 < Y) {
                lp.year((uint32_t)(t + 1), rk);
                if (warp < NGr) normals(order[warp]);
            }
            if (!to_mbar::wait(&s_bar, phase)) {
                if (a.flags) atomicExch(a.flags, TO_DEVERR_SPIN);
                return;
            }
            phase ^= 1u;
            if (two) {
                V* tmp = cur;
                cur = nxt;
                nxt = tmp;
            } else {
#pragma unroll 4
                for (int q = tid; q < N4 * kLanes; q += blockDim.x) cur[q] = far[q];
                __syncthreads();
            }
        }
        if (warp == 0) {
            const bool migrated = a.sem == 0 && Y > 0;
            V tt = L::all(0.0f);
#pragma unroll 4
            for (int grp = 0; grp < NGr; ++grp) {
                const V* v = cur + (size_t)grp * 4 * kLanes + lane;
                tt = L::add(tt, migrated ? v[0]
                                         : L::add(L::add(L::add(v[0], v[kLanes]), v[2 * kLanes]),
                                                  v[3 * kLanes]));
            }
            L::store(a.end_pops + (size_t)rs * P + path0, P - path0, tt);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// ROV forward paths (forwardPathKernel :789-956) - grid ceil(P/32)
// ---------------------------------------------------------------------------
template <int CMAX, int MAXG>
__global__ void __launch_bounds__(1024, 1)
k_rov_forward_sparse(to_rov_args a, to_csc csc) {
    extern __shared__ unsigned char sm_raw[];
    // grid (path tiles of a road, roads): lane = path of road blockIdx.y
    const int NE = a.ne, NG = NE >> 2, NP = a.np, C = a.C, Y = a.Y, P = a.P;
    const size_t PT = (size_t)a.PT;
    const int rd = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int path = blockIdx.x * kLanes + lane;
    const size_t gp = (size_t)rd * P + path;                    // path of the batch
    float* cur = reinterpret_cast<float*>(sm_raw);                 // [NE][32]
    float* part = cur + (size_t)NE * kLanes;                       // [C+1][NG][32]
    float* capv = part + (size_t)(C + 1) * NG * kLanes;            // [NE]
    float* gm = capv + NE;                                         // [32]
    float* tot = gm + kLanes;                                      // [32]
    float* ntot = tot + kLanes;                                    // [32]
    int* ctl = reinterpret_cast<int*>(ntot + kLanes);              // [32]
    int* cptr = ctl + kLanes;                                      // [C][NE+1]
    float* cval = reinterpret_cast<float*>(cptr + (size_t)C * (NE + 1));  // [C][cap_smem]
    uint16_t* cidx = reinterpret_cast<uint16_t*>(cval + (size_t)C * csc.cap_smem);
    const uint32_t road = (uint32_t)a.road_ids[rd];

    for (int s = 0; s < a.S; ++s) {
        const int rs = rd * a.S + s;
        const int N = a.n_patches[rs];
        const int N4 = (N + 3) & ~3;
        const int NGr = N4 >> 2;           // this road's groups (see k_mte_sparse)
        const float* sp = a.params + 8 * s;
        const float* ip = a.init_pops + (size_t)rs * NP;
        __syncthreads();
        for (int q = threadIdx.x; q < NE * kLanes; q += blockDim.x) {
            int k = q / kLanes;
            cur[q] = (k < N) ? ip[k] : 0.0f;
        }
        for (int k = threadIdx.x; k < NE; k += blockDim.x) capv[k] = a.caps[(size_t)rs * NP + k];
        for (int c = 0; c < C; ++c) {
            const int mtx = rs * C + c;
            const int nnz = csc.nnz[mtx];
            for (int k = threadIdx.x; k <= NE; k += blockDim.x)
                cptr[c * (NE + 1) + k] = csc.ptr[(size_t)mtx * (NP + 1) + (k <= NP ? k : NP)];
            for (int e = threadIdx.x; e < nnz; e += blockDim.x) {
                cval[(size_t)c * csc.cap_smem + e] = csc.val[(size_t)mtx * csc.cap + e];
                cidx[(size_t)c * csc.cap_smem + e] = csc.idx[(size_t)mtx * csc.cap + e];
            }
        }
        __syncthreads();
        if (warp == 0) {
            float tt = 0.0f;
            for (int grp = 0; grp < NGr; ++grp) {
                const float* v = cur + (size_t)grp * 4 * kLanes + lane;
                tt = tt + grouped4(v[0], v[kLanes], v[2 * kLanes], v[3 * kLanes]);
            }
            tot[lane] = tt;
            gm[lane] = sp[0];
            if (path < P) a.totalPops[((size_t)s * (Y + 1)) * PT + gp] = tt;
        }
        __syncthreads();
        for (int t = 0; t < Y; ++t) {
            if (warp == 0) {
                float uj = to_uniform1(a.seed, TO_STREAM_SP_JUMP, road, path, t, s);
                float zb = to_normal1(a.seed, TO_STREAM_SP_BROWNIAN, road, path, t, s);
                float zj = to_normal1(a.seed, TO_STREAM_SP_JUMPSIZE, road, path, t, s);
                float jp = (a.sem == 0) ? sp[5] : sp[6];
                float jump = (uj < jp) ? 1.0f : 0.0f;
                float brown = zb * sp[2];
                float s5 = sp[5] * sp[5];
                float jsz = (a.sem == 0) ? (zj * s5 - s5 / 2.0f) : (zj * sp[5] - s5 / 2.0f);
                float g = gm[lane];
                gm[lane] = g + sp[4] * (sp[1] - g) * a.dt + g * brown
                           + (to_expf(jsz) - 1.0f) * g * jump;
                ctl[lane] = (path < P) ? a.controls[(size_t)t * PT + gp] : 0;
                if (a.gmY && path < P) a.gmY[((size_t)t * a.S + s) * P + path] = gm[lane];
            }
            __syncthreads();
            if (a.popsY) {
                // ALGO6 restarts paths from here: the year's starting patch
                // populations, 32 consecutive paths per row
                for (int q = threadIdx.x; q < NE * kLanes; q += blockDim.x) {
                    const int pth = blockIdx.x * kLanes + (q & (kLanes - 1));
                    if (pth < P)
                        a.popsY[(((size_t)t * a.S + s) * NE + (q >> 5)) * P + pth] = cur[q];
                }
            }
            const float g = gm[lane];
            const int my_c = ctl[lane];
            float nv[MAXG][4];
#pragma unroll
            for (int gi = 0; gi < MAXG; ++gi) {
                const int grp = warp + gi * W;
                if (grp < NGr) {
                float z[4];
                to_normal4(a.seed, TO_STREAM_GROWTH, road, path, t,
                           (uint32_t)((s * N4) >> 2) + grp, z);
                float mc[CMAX][4];
                float np4[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    int k = grp * 4 + j;
                    float mv = 0.0f;
#pragma unroll
                    for (int c = 0; c < CMAX; ++c) {
                        if (c >= C) break;
                        const int* cp = cptr + c * (NE + 1);
                        const float* cv = cval + (size_t)c * csc.cap_smem;
                        const uint16_t* ci = cidx + (size_t)c * csc.cap_smem;
                        float acc = 0.0f;
                        for (int e = cp[k]; e < cp[k + 1]; ++e)
                            acc = fmaf(cur[(int)ci[e] * kLanes + lane], cv[e], acc);
                        mc[c][j] = acc;
                        if (c == my_c) mv = acc;
                    }
                    float gr = (a.sem == 0) ? g + z[j] * sp[7] : fmaf(sp[7] * z[j], g, g);
                    float cpk = capv[k];
                    float v = (a.sem == 0) ? mv * (1.0f + gr * (cpk - mv) / cpk / 100.0f)
                                           : fmaxf(mv * (1.0f + gr * (cpk - mv) / cpk), 0.0f);
                    nv[gi][j] = v;
                    np4[j] = v;
                }
#pragma unroll
                for (int c = 0; c < CMAX; ++c) {
                    if (c >= C) break;
                    part[((size_t)c * NG + grp) * kLanes + lane] =
                        grouped4(mc[c][0], mc[c][1], mc[c][2], mc[c][3]);
                }
                part[((size_t)C * NG + grp) * kLanes + lane] =
                    grouped4(np4[0], np4[1], np4[2], np4[3]);
                }
            }
            __syncthreads();
            // totals: warp c sums control c's AAR numerator, warp C the new
            // populations (groups ascending)
            for (int c = warp; c <= C; c += W) {
                float tt = 0.0f;
                for (int grp = 0; grp < NGr; ++grp)
                    tt = tt + part[((size_t)c * NG + grp) * kLanes + lane];
                if (path < P) {
                    if (c < C) a.aars[(((size_t)s * C + c) * Y + t) * PT + gp] = tt / tot[lane];
                    else a.totalPops[((size_t)s * (Y + 1) + t + 1) * PT + gp] = tt;
                }
                if (c == C) ntot[lane] = tt;
            }
            __syncthreads();                   // every warp has read tot
            if (warp == 0) tot[lane] = ntot[lane];
#pragma unroll
            for (int gi = 0; gi < MAXG; ++gi) {
                const int grp = warp + gi * W;
                if (grp < NGr) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) cur[(grp * 4 + j) * kLanes + lane] = nv[gi][j];
                }
            }
            __syncthreads();
        }
    }
}


// ---------------------------------------------------------------------------
// ALGO6 path re-simulation (optimalForwardPaths :1199-2206, as its comments
// describe it).  A CTA re-simulates a tile of 32 or 16 paths (lane = path)
// from year t0 to the horizon with every species together, since each
// year's control depends on all species' states.  A warp owns groups of four
// patches; a year has three barriers:
//   A. every control's migration of the group's populations into shared
//      memory (ascending origins, as forward) and the groups' sums; then the
//      group's growth normals, which need nothing of the decision;
//   B. warp c, as soon as all warps are through with A's first part: control
//      c's adjusted populations tot * (total / tot) from the groups' sums in
//      order, its payoff under the year's regression (the terminal rule in
//      the last year);
//   C. the least valid payoff's control, the growth of its migrated
//      populations with the forward pass's growth mean (stored by it); warp 0
//      adds flows[c] * profit, discounted by (1 + r dt / 100) per year.
// The year-t0 value replaces condExp[t0] and the year-t0 control optCont[t0].
//
// Bound by latency: the years of a restart follow one another, the restarts
// too, and the tiles seldom fill the GPU.  So the lists are the union
// ones where they fit (a loop for all controls, its loads in flight
// together), the payoffs are a warp's each with everything unrolled, and the
// profits come from the table the regressions use.  2,000 paths, 2 species of
// 61 patches, 50 years: 24 -> 7.2 us a year of a restart (five barriers, a
// loop for every control, one warp deciding and drawing the ore's noise again
// before), then 4.6: what a year runs through exceeded the instruction cache,
// so one layout is one kernel, one group's normals wait instead of four (8.1
// against 9.7 ms a valuation) and nothing divides by a run-time count; half a
// warp a group spreads 2,000 paths over 125 SMs instead of 63.  The lists
// side by side, or the next year's regressions fetched ahead, cost more in
// code than they hid (8.1 -> 8.6 ms).
// ---------------------------------------------------------------------------

// shared memory: bytes of the lists, [S] reciprocals and groups' sums beside
// what every layout has
__host__ __device__ inline size_t resim_bytes(int NE, int S, int C, size_t lists, bool sums, int tp) {
    const size_t rows = (size_t)S * (C + 1) * NE * tp * 4;
    return rows + (size_t)S * NE * 4 + (size_t)C * tp * 4 + lists +
           (sums ? (size_t)S * NE * 4 + (size_t)S * (C + 1) * (NE >> 2) * tp * 4 : 0);
}
__host__ __device__ inline size_t resim_lists(int NE, int S, int C, int cap_smem) {
    return (size_t)S * C * ((NE + 1) * 4 + (size_t)cap_smem * 6) + 16;
}

// TP paths a tile: 32, a warp a group, or 16, half a warp a group ("warp"
// below).  UNI: union lists, the groups' sums and the tables of the normals
// all fit; the other layouts are a kernel of their own, since what the years
// run through has to stay in the instruction cache.
template <int S, int TP, bool UNI>
__global__ void __launch_bounds__(1024, 1)
k_rov_resim(to_rov_args a, to_csc csc, int t0, int smem) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int NE = a.ne, NG = NE >> 2, NP = a.np, C = a.C, Y = a.Y, P = a.P, R = a.R;
    const int SC = S * C;
    const int tid = threadIdx.x, lane = tid % TP, warp = tid / TP, W = blockDim.x / TP;
    const int path = blockIdx.x * TP + lane;
    const bool live = path < P;
    // the layout: union lists and the groups' sums, or the controls' own
    // lists, with the sums where they fit
    int nu = 0;
    if (UNI)
        for (int s = 0; s < S; ++s) nu += csc.unnz[s];
    const size_t clists = resim_lists(NE, S, C, csc.cap_smem);
    constexpr bool uni = UNI;
    const bool sums = UNI || resim_bytes(NE, S, C, clists, true, TP) <= (size_t)smem;
    unsigned char* at = sm_raw;
    auto take = [&](size_t bytes) { unsigned char* r = at; at += bytes; return r; };
    int4* ue = reinterpret_cast<int4*>(uni ? take((size_t)nu * 16) : at);      // [nu]
    float* cur = reinterpret_cast<float*>(take((size_t)S * NE * TP * 4));  // [S][NE][32]
    float* mig = reinterpret_cast<float*>(take((size_t)SC * NE * TP * 4)); // [S][C][NE][32]
    float* pay = reinterpret_cast<float*>(take((size_t)C * TP * 4));       // [C][32]
    float* capv = reinterpret_cast<float*>(take((size_t)S * NE * 4));          // [S][NE]
    float *rcap = nullptr, *msum = nullptr, *tsum = nullptr;
    if (sums) {
        rcap = reinterpret_cast<float*>(take((size_t)S * NE * 4));             // [S][NE] 1 / capacity
        msum = reinterpret_cast<float*>(take((size_t)SC * NG * TP * 4));   // [S][C][NG][32]
        tsum = reinterpret_cast<float*>(take((size_t)S * NG * TP * 4));    // [S][NG][32]
    }
    const int lists = uni ? S : SC;
    int* cptr = reinterpret_cast<int*>(take((size_t)lists * (NE + 1) * 4));    // [S] or [S][C], [NE + 1]
    float* cval = reinterpret_cast<float*>(uni ? at : take((size_t)SC * csc.cap_smem * 4));
    uint16_t* cidx = reinterpret_cast<uint16_t*>(at);                          // [S][C][cap_smem]
    to_bm_tables* tab = nullptr;
    if (UNI) {
        at = sm_raw + (((size_t)(at - sm_raw) + 15) & ~(size_t)15);
        tab = reinterpret_cast<to_bm_tables*>(take(sizeof(to_bm_tables)));
        to_bm_load(*tab);
    }
    const uint32_t stream_road = TO_STREAM_GROWTH | ((uint32_t)a.road << 8);

    for (int q = tid; q < S * NE * TP; q += blockDim.x) {
        const int sk = q / TP, pth = blockIdx.x * TP + (q & (TP - 1));
        const int s = sk / NE, k = sk - s * NE;
        cur[q] = (pth < P) ? a.popsY[(((size_t)t0 * S + s) * NE + k) * P + pth] : 0.0f;
    }
    for (int q = tid; q < S * NE; q += blockDim.x) {
        const int s = q / NE, k = q - s * NE;
        const float cp = a.caps[(size_t)s * NP + k];
        capv[q] = cp;
        if (sums) rcap[q] = 1.0f / cp;
    }
    if (uni) {
        int e0 = 0;
        for (int s = 0; s < S; ++s) {
            const int n = csc.unnz[s];
            for (int k = tid; k <= NE; k += blockDim.x)
                cptr[s * (NE + 1) + k] = e0 + csc.uptr[(size_t)s * (NP + 1) + (k <= NP ? k : NP)];
            for (int e = tid; e < n; e += blockDim.x) {
                int4 v = csc.uent[(size_t)s * csc.ucap + e];
                if (v.x == kNoOrigin) v.x = 0;      // its values are zero: no term
                v.x *= TP * (int)sizeof(float);
                ue[e0 + e] = v;
            }
            e0 += n;
        }
    } else {
        for (int m = 0; m < SC; ++m) {
            const int nnz = csc.nnz[m];
            for (int k = tid; k <= NE; k += blockDim.x)
                cptr[m * (NE + 1) + k] = csc.ptr[(size_t)m * (NP + 1) + (k <= NP ? k : NP)];
            for (int e = tid; e < nnz; e += blockDim.x) {
                cval[(size_t)m * csc.cap_smem + e] = csc.val[(size_t)m * csc.cap + e];
                cidx[(size_t)m * csc.cap_smem + e] = csc.idx[(size_t)m * csc.cap + e];
            }
        }
    }
    __syncthreads();
    if (sums) {
        for (int q = warp; q < S * NG; q += W) {
            const float* v = cur + (size_t)q * 4 * TP + lane;
            tsum[q * TP + lane] = grouped4(v[0], v[TP], v[2 * TP], v[3 * TP]);
        }
        __syncthreads();
    }
    // the warp's first group, whose normals and growth mean wait in registers
    // (one only: code for more costs more than it hides)
    const bool own = warp < S * NG;
    const int spec = own ? warp / NG : 0;
    to_path_stream ps;
    to_stream_path(ps, (uint32_t)path);
    // totals over the groups of every species before (ts) and after (tt)
    // control c's migration: 2 S chains side by side
    auto totals = [&](int c, float (&ts)[S], float (&tt)[S]) {
#pragma unroll
        for (int s = 0; s < S; ++s) ts[s] = tt[s] = 0.0f;
        if (sums) {
#pragma unroll 4
            for (int grp = 0; grp < NG; ++grp)
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    ts[s] = ts[s] + tsum[((size_t)s * NG + grp) * TP + lane];
                    tt[s] = tt[s] + msum[((size_t)(s * C + c) * NG + grp) * TP + lane];
                }
        } else {
            for (int grp = 0; grp < NG; ++grp)
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float* v = cur + ((size_t)s * NE + grp * 4) * TP + lane;
                    ts[s] = ts[s] + grouped4(v[0], v[TP], v[2 * TP], v[3 * TP]);
                    v = mig + ((size_t)(s * C + c) * NE + grp * 4) * TP + lane;
                    tt[s] = tt[s] + grouped4(v[0], v[TP], v[2 * TP], v[3 * TP]);
                }
        }
    };
    auto draw = [&](int s, int q, float (&z)[4]) {
        const int grp = q - s * NG, N4 = (a.n_patches[s] + 3) & ~3;
        const to_u32x4 w = to_stream_words(
            ps, to_stream_group((uint32_t)((s * N4) >> 2) + grp, stream_road, a.rk), a.rk);
        if (UNI) {
            f2 cs, sn;                             // of both Box-Muller pairs
            to_box_muller2(w.v[0], w.v[1], w.v[2], w.v[3], *tab, cs, sn);
            unpack2(cs, z[0], z[2]);
            unpack2(sn, z[1], z[3]);
        } else {
            to_box_muller(w.v[0], w.v[1], &z[0], &z[1]);
            to_box_muller(w.v[2], w.v[3], &z[2], &z[3]);
        }
    };
    const float disc = 1.0f + a.rrr * a.dt / 100.0f;
    float val = 0.0f, df = 1.0f;        // warp 0: realised value, discount factor
    int first = 0;
    for (int u = t0; u < Y; ++u) {
        const bool last = u == Y - 1;
        // what the year reads from global memory, requested ahead of its use
        const float prof = live ? a.profS[(size_t)u * P + path] : 0.0f;
        const float gm = live && own ? a.gmY[((size_t)u * S + spec) * P + path] : 0.0f;
        // A
        for (int q = warp, i = 0; q < S * NG; q += W, ++i) {
            const int s = i == 0 ? spec : q / NG, grp = q - s * NG;
            const float* cs = cur + (size_t)s * NE * TP + lane;
            float* mg = mig + ((size_t)s * C * NE + grp * 4) * TP + lane;
            if (uni) {
                const int* up = cptr + s * (NE + 1) + grp * 4;
                float g0 = 0.0f, g1 = 0.0f, g2 = 0.0f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float q0 = 0.0f, q1 = 0.0f, q2 = 0.0f;
                    const int e1 = up[j + 1];
#pragma unroll 2
                    for (int e = up[j]; e < e1; e += 2) {      // an even number of terms
#pragma unroll
                        for (int w = 0; w < 2; ++w) {
                            const int4 en = ue[e + w];
                            const float x = *reinterpret_cast<const float*>(
                                reinterpret_cast<const unsigned char*>(cs) + en.x);
                            q0 = fmaf(x, __int_as_float(en.y), q0);
                            q1 = fmaf(x, __int_as_float(en.z), q1);
                            q2 = fmaf(x, __int_as_float(en.w), q2);
                        }
                    }
                    mg[j * TP] = q0;
                    if (C > 1) mg[(size_t)(NE + j) * TP] = q1;
                    if (C > 2) mg[(size_t)(2 * NE + j) * TP] = q2;
                    g0 = j ? g0 + q0 : q0;
                    g1 = j ? g1 + q1 : q1;
                    g2 = j ? g2 + q2 : q2;
                }
                const float any = g0 + g1 + g2;
                if (any != any) {
                    // an infinite population times a zero: a control's sum
                    // is over its own entries, so without the zeros
#pragma unroll 1
                    for (int j = 0; j < 4; ++j) {
                        float q0 = 0.0f, q1 = 0.0f, q2 = 0.0f;
#pragma unroll 1
                        for (int e = up[j]; e < up[j + 1]; ++e) {
                            const int4 en = ue[e];
                            const float x = *reinterpret_cast<const float*>(
                                reinterpret_cast<const unsigned char*>(cs) + en.x);
                            if (en.y) q0 = fmaf(x, __int_as_float(en.y), q0);
                            if (en.z) q1 = fmaf(x, __int_as_float(en.z), q1);
                            if (en.w) q2 = fmaf(x, __int_as_float(en.w), q2);
                        }
                        mg[j * TP] = q0;
                        if (C > 1) mg[(size_t)(NE + j) * TP] = q1;
                        if (C > 2) mg[(size_t)(2 * NE + j) * TP] = q2;
                        g0 = j ? g0 + q0 : q0;
                        g1 = j ? g1 + q1 : q1;
                        g2 = j ? g2 + q2 : q2;
                    }
                }
                float* o = msum + ((size_t)s * C * NG + grp) * TP + lane;
                o[0] = g0;
                if (C > 1) o[(size_t)NG * TP] = g1;
                if (C > 2) o[(size_t)2 * NG * TP] = g2;
            } else {
                for (int c = 0; c < C; ++c) {
                    const int m = s * C + c;
                    const int* cp = cptr + m * (NE + 1) + grp * 4;
                    const float* cv = cval + (size_t)m * csc.cap_smem;
                    const uint16_t* ci = cidx + (size_t)m * csc.cap_smem;
                    float gs = 0.0f;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float acc = 0.0f;
#pragma unroll 4
                        for (int e = cp[j]; e < cp[j + 1]; ++e)
                            acc = fmaf(cs[(int)ci[e] * TP], cv[e], acc);
                        mg[((size_t)c * NE + j) * TP] = acc;
                        gs = j ? gs + acc : acc;
                    }
                    if (sums) msum[((size_t)m * NG + grp) * TP + lane] = gs;
                }
            }
        }
        __syncthreads();
        // B
        for (int c = warp; c < C; c += W) {
            float st[S], ts[S], tt[S];
            bool valid = true;
            totals(c, ts, tt);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                st[s] = ts[s] * (tt[s] / ts[s]);
                if (st[s] < to_rovd::threshold(a, s) && c > 0) valid = false;
            }
            float r = INFINITY;                    // an invalid control's
            if (valid && live) {
                const float now = a.flows[c] * prof;
                if (last) {
                    r = now > 0.0f ? 0.0f : now;
                } else {
                    r = to_rovd::payoff(
                        now, to_lsm_interp(to_rov_reg_block(a, u, c), R, S, st, prof) / disc);
                }
            }
            pay[c * TP + lane] = r;
        }
        float z[4];
        if (!last && own) {
            to_stream_year(ps, (uint32_t)u, a.rk);
            draw(spec, warp, z);
        }
        __syncthreads();
        // C
        int cu = 0;
        {
            float best = pay[lane];
            for (int c = 1; c < C; ++c) {
                const float r = pay[c * TP + lane];
                if (r < best) { best = r; cu = c; }
            }
        }
        if (u == t0) first = cu;
        if (warp == 0 && live) {
            val = val + (a.flows[cu] * prof) * df;
            df = df / disc;
        }
        if (last) break;
        auto grow = [&](int s, int q, const float (&zz)[4], float g) {
            const int grp = q - s * NG;
            const float s7 = a.params[8 * s + 7];
            const float* mg = mig + (((size_t)s * C + cu) * NE + grp * 4) * TP + lane;
            float* o = cur + ((size_t)s * NE + grp * 4) * TP + lane;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float mv = mg[j * TP], cpk = capv[s * NE + grp * 4 + j];
                const float gr = fmaf(s7 * zz[j], g, g), x = gr * (cpk - mv);
                const float d = sums ? to_div_rcp_inf(x, cpk, rcap[s * NE + grp * 4 + j]) : x / cpk;
                v[j] = fmaxf(mv * (1.0f + d), 0.0f);
                o[j * TP] = v[j];
            }
            if (sums) tsum[q * TP + lane] = grouped4(v[0], v[1], v[2], v[3]);
        };
        if (own) grow(spec, warp, z, gm);
        for (int q = warp + W; q < S * NG; q += W) {
            const int s = q / NG;
            draw(s, q, z);
            grow(s, q, z, live ? a.gmY[((size_t)u * S + s) * P + path] : 0.0f);
        }
        __syncthreads();
    }
    if (warp == 0 && live) {
        a.condExp[(size_t)t0 * P + path] = val;
        a.optCont[(size_t)t0 * P + path] = first;
    }
}

}  // namespace

namespace to_k {

to_status pack_csc(to_ctx ctx, const float* mmm, int NP, int C, const int* n_patches,
                   int n_rs, to_csc& csc, int rs0) {
    if (NP > 1024) return to_set_error(ctx, TO_ERR_UNSUPPORTED, "patches %d", NP);
    to_prof_begin(ctx, "pack_csc");
    k_pack_csc<<<n_rs * C, 1024, 0, ctx->stream>>>(mmm, NP, C, n_patches, csc.cap,
                                                 csc.ptr, csc.idx, csc.val, csc.nnz, rs0 * C);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

// What is admitted: models whose lists fit beside one path a lane (8 bytes an
// entry) with their groups' sums, up to 512 patches.  The kernel lays a model
// out by mte_bytes and can leave its lists in global memory, so this is a rule
// of choice - longer lists go to the dense kernels - and not its limit.
size_t mte_sparse_smem(int NE, int cap_smem) {
    if (NE > 32 * kMaxG * 4) return ~size_t(0);  // 32 warps of kMaxG groups of four
    const int NG = NE / 4;
    return (size_t)cap_smem * 8 + (size_t)(NE * kLanes + NG * kLanes + 2 * NE + kGmChunk * 3 * kLanes) * 4 +
           (size_t)(NE + 1 + NG) * 4 + 16;
}

size_t mte_far_count(to_ctx ctx, int NP) {
    return (size_t)ctx->sm_count * (NP < 32 * kMaxG * 4 ? NP : 32 * kMaxG * 4) * kLanes;
}

// warps per CTA: enough that no warp owns more than kMaxG groups of four
// (32 warps at most, so NE <= 512 for the sparse kernels)
static int warps_for(int NE, int min_warps) {
    int NG = NE / 4;
    int w = (NG + kMaxG - 1) / kMaxG;
    if (w < min_warps) w = min_warps;
    if (w > 32) w = 32;
    return w;
}

to_status mte_sparse(to_ctx ctx, to_mte_args a, int n_rs, to_csc csc) {
    if (a.npe <= 0) a.npe = a.npad;
    if (!a.flags) a.flags = ctx->d_flags;
    const int NE = a.npe, NE4 = (NE + 3) & ~3;
    size_t smem = mte_sparse_smem(NE, csc.cap_smem);
    if (smem > ctx->smem_optin)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "sparse MTE needs %zu B", smem);
    if (n_rs > 1) {
        k_mte_order<<<(n_rs + kOrder - 1) / kOrder, kOrder, 0, ctx->stream>>>(n_rs, a.rs0, a.C, a.c_use, csc.nnz, a.order_buf);
        TO_LAUNCHED(ctx);
        a.order = a.order_buf;
    }
    const size_t limit = ctx->smem_optin - kPairStatic;
    // One path a lane where two would use at most half the SMs (200 patches,
    // 1,000 paths, 2 species: 0.43 against 0.53 ms a call; with 94 tiles of
    // 64 paths on 152 SMs 0.43 against 0.39).
    const int pairs = (a.n_paths + 2 * kLanes - 1) / (2 * kLanes) * n_rs;
    const int paths = a.n_paths <= kLanes || 2 * pairs <= ctx->sm_count ? 1 : 2;
    const int items = (a.n_paths + paths * kLanes - 1) / (paths * kLanes) * n_rs;
    // Up to four CTAs an SM, of 32 warps together, where there are tiles for
    // them and their lists and both buffers fit: few groups leave many warps
    // of a wide CTA idle, and one CTA's barrier hides behind another's work
    // (40,000 paths, 2 species of 20 / 40 / 115 patches, one CTA an SM: 1.23
    // / 1.34 / 2.18 ms a call, four (115: two): 0.73 / 1.00 / 1.93; eight no
    // better).  The lists' padding is taken as half their entries here; a
    // model whose lists need more reads them from global memory.
    int c = (items + ctx->sm_count - 1) / ctx->sm_count;
    if (c > 4) c = 4;
    auto share = [&](int n) { return n == 1 ? limit : (limit + 1024) / n - 1024 - kPairStatic; };
    while (c > 1 && mte_bytes(NE4, csc.cap_smem * 3 / 16 + 8, true, paths) > share(c)) --c;
    const size_t each = share(c);
    int W = 32 / c < NE4 / 4 ? 32 / c : NE4 / 4;
    if (W < 2) W = 2;
    const int ctas = c * ctx->sm_count;
    const auto kern = paths == 2 ? k_mte_sparse<f2> : k_mte_sparse<float>;
    TO_CUDA(ctx, cudaMemsetAsync(a.order_buf + n_rs, 0, sizeof(int), ctx->stream));
    TO_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)each));
    to_prof_begin(ctx, "mte_sparse");
    kern<<<items < ctas ? items : ctas, W * 32, each, ctx->stream>>>(
        a, csc, to_make_round_keys(a.seed), n_rs, (int)each, c == 1);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

size_t rov_sparse_smem(int NE, int C, int cap_smem) {
    if (NE > 32 * kMaxG * 4 || C + 1 > 32) return ~size_t(0);
    int NG = NE / 4;
    return (size_t)(NE * kLanes + (C + 1) * NG * kLanes + NE + 4 * kLanes) * 4 +
           (size_t)C * (NE + 1) * 4 + (size_t)C * cap_smem * 6 + 16;
}

size_t rov_union_smem(int NE, int C, int ucap_smem) {
    if (C > 3) return ~size_t(0);
    return pair_bytes(NE, ucap_smem, false) + kPairStatic;
}

to_status union_csc(to_ctx ctx, int NP, int C, const int* n_patches, int n_rs, to_csc& csc) {
    if (C > 3 || !csc.uent || !csc.uptr || !csc.unnz)
        return to_set_error(ctx, TO_ERR_INVALID, "union form: %d controls", C);
    k_union_csc<<<n_rs, 256, 0, ctx->stream>>>(NP, C, n_patches, csc);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

to_status rov_forward_sparse(to_ctx ctx, const to_rov_args& a, to_csc csc) {
    if (csc.uent && a.C <= 3) {
        // every (road, species) lays its own sizes out in all of the shared
        // memory, so a plan's margin costs nothing
        const int smem = (int)ctx->smem_optin - kPairStatic;
        const int items = (a.P + kPairPaths - 1) / kPairPaths * a.nr * a.S;
        const auto pair = a.sem == 0 ? k_rov_forward_union<true> : k_rov_forward_union<false>;
        TO_CUDA(ctx, cudaMemsetAsync(a.fwd_next, 0, sizeof(int), ctx->stream));
        TO_CUDA(ctx, cudaFuncSetAttribute(pair, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        to_prof_begin(ctx, "rov_forward_sparse");
        pair<<<items < a.ctas ? items : a.ctas, kPairThreads, smem, ctx->stream>>>(a, csc, smem);
        to_prof_end(ctx);
        TO_LAUNCHED(ctx);
        return TO_OK;
    }
    size_t smem = rov_sparse_smem(a.ne, a.C, csc.cap_smem);
    if (smem > ctx->smem_optin)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "sparse ROV needs %zu B", smem);
    int warps = warps_for(a.ne, a.C + 1 > 4 ? a.C + 1 : 4);
    if ((a.ne / 4 + warps - 1) / warps > kMaxG)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "patches %d", a.ne);
    const dim3 blocks((a.P + kLanes - 1) / kLanes, a.nr);
    to_prof_begin(ctx, "rov_forward_sparse");
    if (a.C <= 3) {
        TO_CUDA(ctx, cudaFuncSetAttribute(k_rov_forward_sparse<3, kMaxG>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_rov_forward_sparse<3, kMaxG><<<blocks, warps * 32, smem, ctx->stream>>>(a, csc);
    } else {
        TO_CUDA(ctx, cudaFuncSetAttribute(k_rov_forward_sparse<TO_ROV_MAXC, kMaxG>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_rov_forward_sparse<TO_ROV_MAXC, kMaxG><<<blocks, warps * 32, smem, ctx->stream>>>(a, csc);
    }
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return TO_OK;
}


to_status rov_resim_sparse(to_ctx ctx, const to_rov_args& a, to_csc csc, int t0) {
    // the smallest layout has to fit
    const size_t least =
        resim_bytes(a.ne, a.S, a.C, resim_lists(a.ne, a.S, a.C, csc.cap_smem), false, kLanes);
    const size_t limit = ctx->smem_optin;
    if (least > limit)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "ALGO6 re-simulation needs %zu B", least);
    // Tiles of 16 paths while the SMs take them all at once (2 species of 61 /
    // 130 patches, 1,999 / 1,000 paths: 9.7 / 13.4 ms a valuation against
    // 10.2 / 16.2 in tiles of 32; 2,500 paths fill the SMs either way)
    const int tp = (a.P + 15) / 16 <= ctx->sm_count ? 16 : 32;
    const size_t ulists = (size_t)a.S * ((size_t)csc.ucap_smem * 16 + (size_t)(a.ne + 1) * 4);
    const bool uni = csc.uent && resim_bytes(a.ne, a.S, a.C, ulists, true, tp) + 16 +
                                         sizeof(to_bm_tables) <= limit;
    using kern_t = void (*)(to_rov_args, to_csc, int, int);
    const auto pick = [&](kern_t u16, kern_t u32, kern_t c16, kern_t c32) {
        return tp == 16 ? (uni ? u16 : c16) : (uni ? u32 : c32);
    };
#define TO_RESIM(S) \
    pick(k_rov_resim<S, 16, true>, k_rov_resim<S, 32, true>, k_rov_resim<S, 16, false>, \
         k_rov_resim<S, 32, false>)
    const kern_t kern = a.S == 1 ? TO_RESIM(1) : a.S == 2 ? TO_RESIM(2) : a.S == 3 ? TO_RESIM(3)
                                                                                   : TO_RESIM(4);
#undef TO_RESIM
    const int blocks = (a.P + tp - 1) / tp;
    to_prof_begin(ctx, "rov_resim");
    TO_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
    kern<<<blocks, 1024, limit, ctx->stream>>>(a, csc, t0, (int)limit);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

}  // namespace to_k
