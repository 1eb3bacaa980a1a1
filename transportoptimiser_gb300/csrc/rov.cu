// rov.cu - controlled-traffic real-options valuation on the device
// (ALGO4: forward paths under random controls, regression Monte Carlo
// backward induction with multiple local linear regression on k nearest
// neighbours).
//
// Reference (include/gpuCode/SimulateGPU.cu): simulateROVCUDA :3870-5003,
// randControls :720, forwardPathKernel :789, computePathStates :959,
// allocateXYRegressionData :1012, computeStateMinMax :1073,
// createQueryPoints :1152, firstPeriodInduction :2210, backwardInduction
// :2333, multiLocLinReg :2934, knn_cuda_with_indexes::knn (kNN).
//
// What changes on GB300:
//  * the forward pass keeps every path tile's populations in shared memory
//    for all years and evaluates all controls' migrations from one read of
//    the populations; the random streams are regenerated from Philox where
//    they are consumed (nothing of size P*Y*N is stored);
//  * the reference's serial <<<1,1>>> compaction and min/max kernels become a
//    CTA per (road, year), all years independent of one another;
//  * kNN and regressions run on the device (knn_fit.cu): a thread per grid
//    query, the same neighbour set as the reference's stable insertion sort
//    without its P x Q distance matrix or host round trips;
//  * the local linear systems are accumulated in FP32 and solved in FP64
//    (Cholesky); expectations are reduced in FP64;
//  * several roads can be valued in one batch: paths are road-major and the
//    regressions are grouped by (road, control).
// Every per-query / per-path formula comes from to_lsm_math.h so the SIMT
// path reproduces the oracle bit for bit.
#include <cmath>
#include <cstring>
#include <vector>

#include "to_internal.cuh"
#include "to_lsm_math.h"
#include "to_rov.cuh"
#include "to_rov_dev.cuh"
#include "to_rov_years.h"
#include "to_sparse.cuh"

namespace {

using to_rovd::adj_pop;
using to_rovd::ore_at;
using to_rovd::threshold;
using to_rovd::unit_profit;

// ---------------------------------------------------------------------------
// exogenous processes and random controls (forwardPathKernel :930-952,
// randControls :720-730): uRes[u][t][p], controls[t][p]
// ---------------------------------------------------------------------------
// Lane = path.  What a year draws does not depend on the years before, so the
// CTA's warps draw the (year, process) pairs of 16 years and four processes
// at a time, and then one warp a process runs through those years (a thread a
// path drew everything in the chain before: one road of 10,000 paths, three
// processes, 50 years 98 -> 23 us, 256 roads of 768 paths 448 -> 240).
constexpr int kExYears = 16, kExProc = 4, kExThreads = 256;

__global__ void __launch_bounds__(kExThreads) k_rov_exog(to_rov_args a) {
    __shared__ float s_brown[kExYears][kExProc][32], s_size[kExYears][kExProc][32],
        s_jump[kExYears][kExProc][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kExThreads / 32;
    const int Y = a.Y, U = a.U, P = a.PT, p = min((int)blockIdx.x * 32 + lane, P - 1);
    const bool live = (int)blockIdx.x * 32 + lane < P;
    const int r = p / a.P, pl = p - r * a.P;      // road, path within it
    const uint32_t road = (uint32_t)a.road_ids[r];
    for (int t = warp; t < Y; t += nw) {
        float uc = to_uniform1(a.seed, TO_STREAM_CONTROL, road, pl, t, 0);
        int control = (int)(uc * (float)a.C);
        if (control == a.C) control--;
        if (live) a.controls[(size_t)t * P + p] = control;
    }
    for (int u0 = 0; u0 < U; u0 += kExProc) {
        const int nu = min(kExProc, U - u0);
        const float* up = a.uncert + 6 * (u0 + min(warp, nu - 1));   // of the warp's chain
        float curr = up[0];
        float* out = a.uRes + (size_t)(u0 + min(warp, nu - 1)) * (Y + 1) * P + p;
        if (warp < nu && live) out[0] = curr;
        for (int t0 = 0; t0 < Y; t0 += kExYears) {
            const int ny = min(kExYears, Y - t0);
            __syncthreads();                   // the years before are run through
            for (int q = warp; q < ny * nu; q += nw) {
                const int y = q / nu, j = q - y * nu, t = t0 + y, u = u0 + j;
                const float* uq = a.uncert + 6 * u;
                s_brown[y][j][lane] = to_normal1(a.seed, TO_STREAM_EX_BROWNIAN, road, pl, t, u) * uq[2];
                float jump = 0.0f, size = 0.0f;
                // without jumps their term is 0 whatever is drawn, as long
                // as their size is finite
                if (uq[5] > 0.0f || !(fabsf(uq[4]) <= 1.0f)) {
                    const float uj = to_uniform1(a.seed, TO_STREAM_EX_JUMP, road, pl, t, u);
                    const float zj = to_normal1(a.seed, TO_STREAM_EX_JUMPSIZE, road, pl, t, u);
                    const float s4 = uq[4] * uq[4];
                    const float jsz = (a.sem == 0) ? (zj * s4 - s4 / 2.0f) : (zj * uq[4] - s4 / 2.0f);
                    jump = (uj < uq[5]) ? 1.0f : 0.0f;
                    size = to_expf(jsz) - 1.0f;
                }
                s_jump[y][j][lane] = jump;
                s_size[y][j][lane] = size;
            }
            __syncthreads();
            if (warp < nu)
#pragma unroll 4
                for (int y = 0; y < ny; ++y) {
                    curr = curr + up[3] * (up[1] - curr) * a.dt + curr * s_brown[y][warp][lane]
                           + s_size[y][warp][lane] * curr * s_jump[y][warp][lane];
                    if (live) out[(size_t)(t0 + y + 1) * P] = curr;
                }
        }
    }
}

// ---------------------------------------------------------------------------
// forward paths (forwardPathKernel :789-956).  One CTA = a tile of TP paths,
// one species at a time, all years; thread (pg, kg) owns paths 4pg..4pg+3
// and patches 4kg..4kg+3 for every control.
// ---------------------------------------------------------------------------
template <int CMAX>
__global__ void __launch_bounds__(512)
k_rov_forward(to_rov_args a) {
    extern __shared__ float smem[];
    const int NE = a.ne, KG = NE >> 2, TP = a.tile_paths, LC = a.l_chunk;
    const int C = a.C, Y = a.Y, P = a.P;
    const int tid = threadIdx.x, pg = tid / KG, kg = tid - pg * KG;
    const bool active = pg < (TP >> 2);
    const int path0 = blockIdx.x * TP;
    float* Mt = smem;                               // [C][LC][NE]
    float* pop = Mt + (size_t)C * LC * NE;          // [TP][NE]
    float* mig = pop + (size_t)TP * NE;             // [TP][NE]
    float* gm = mig + (size_t)TP * NE;              // [TP]
    float* tot = gm + TP;                           // [TP]
    int* ctl = reinterpret_cast<int*>(tot + TP);    // [TP]
    const uint32_t road = (uint32_t)a.road;
    const bool resident = (LC == NE);

    for (int s = 0; s < a.S; ++s) {
        const int N = a.n_patches[s];
        const int N4 = (N + 3) & ~3;
        const float* sp = a.params + 8 * s;
        const float* M = a.mmm + (size_t)s * C * a.np * a.np;
        const float* ip = a.init_pops + (size_t)s * a.np;
        float cap4[4];
        for (int j = 0; j < 4; ++j) cap4[j] = a.caps[(size_t)s * a.np + kg * 4 + j];
        __syncthreads();
        for (int q = tid; q < TP * NE; q += blockDim.x) {
            int l = q % NE;
            pop[q] = (l < N) ? ip[l] : 0.0f;
        }
        if (resident) {
            for (int q = tid; q < C * NE * NE; q += blockDim.x) {
                int c = q / (NE * NE), r = q - c * NE * NE;
                int k = r / NE, l = r - k * NE;
                Mt[((size_t)c * NE + l) * NE + k] = M[((size_t)c * a.np + k) * a.np + l];
            }
        }
        __syncthreads();
        for (int q = tid; q < TP; q += blockDim.x) {
            gm[q] = sp[0];
            const float* v = pop + (size_t)q * NE;
            float tt = 0.0f;    // groups of four, ((v0 + v1) + v2) + v3, ascending
            for (int g4 = 0; g4 < NE; g4 += 4) tt = tt + (((v[g4] + v[g4 + 1]) + v[g4 + 2]) + v[g4 + 3]);
            tot[q] = tt;
            int path = path0 + q;
            if (path < P) a.totalPops[((size_t)s * (Y + 1) + 0) * P + path] = tt;
        }
        __syncthreads();
        for (int t = 0; t < Y; ++t) {
            for (int q = tid; q < TP; q += blockDim.x) {
                uint32_t path = (uint32_t)(path0 + q);
                float uj = to_uniform1(a.seed, TO_STREAM_SP_JUMP, road, path, t, s);
                float zb = to_normal1(a.seed, TO_STREAM_SP_BROWNIAN, road, path, t, s);
                float zj = to_normal1(a.seed, TO_STREAM_SP_JUMPSIZE, road, path, t, s);
                float jp = (a.sem == 0) ? sp[5] : sp[6];
                float jump = (uj < jp) ? 1.0f : 0.0f;
                float brown = zb * sp[2];
                float s5 = sp[5] * sp[5];
                float jsz = (a.sem == 0) ? (zj * s5 - s5 / 2.0f) : (zj * sp[5] - s5 / 2.0f);
                float g = gm[q];
                gm[q] = g + sp[4] * (sp[1] - g) * a.dt + g * brown
                        + (to_expf(jsz) - 1.0f) * g * jump;
                ctl[q] = (path0 + q < P) ? a.controls[(size_t)t * P + path0 + q] : 0;
            }
            float acc[CMAX][4][4];
#pragma unroll
            for (int c = 0; c < CMAX; ++c)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[c][i][j] = 0.0f;
            for (int l0 = 0; l0 < NE; l0 += LC) {
                if (!resident) {
                    __syncthreads();
                    for (int q = tid; q < C * LC * NE; q += blockDim.x) {
                        int c = q / (LC * NE), r = q - c * LC * NE;
                        int k = r / LC, l = r - k * LC;
                        Mt[((size_t)c * LC + l) * NE + k] =
                            M[((size_t)c * a.np + k) * a.np + l0 + l];
                    }
                    __syncthreads();
                }
                if (active) {
                    const float* pr = pop + (size_t)(pg * 4) * NE + l0;
                    for (int l = 0; l < LC; ++l) {
                        float a0 = pr[l], a1 = pr[NE + l], a2 = pr[2 * NE + l],
                              a3 = pr[3 * NE + l];
#pragma unroll
                        for (int c = 0; c < CMAX; ++c) {
                            if (c >= C) break;
                            float4 m = *reinterpret_cast<const float4*>(
                                Mt + ((size_t)c * LC + l) * NE + kg * 4);
                            acc[c][0][0] = fmaf(a0, m.x, acc[c][0][0]); acc[c][0][1] = fmaf(a0, m.y, acc[c][0][1]);
                            acc[c][0][2] = fmaf(a0, m.z, acc[c][0][2]); acc[c][0][3] = fmaf(a0, m.w, acc[c][0][3]);
                            acc[c][1][0] = fmaf(a1, m.x, acc[c][1][0]); acc[c][1][1] = fmaf(a1, m.y, acc[c][1][1]);
                            acc[c][1][2] = fmaf(a1, m.z, acc[c][1][2]); acc[c][1][3] = fmaf(a1, m.w, acc[c][1][3]);
                            acc[c][2][0] = fmaf(a2, m.x, acc[c][2][0]); acc[c][2][1] = fmaf(a2, m.y, acc[c][2][1]);
                            acc[c][2][2] = fmaf(a2, m.z, acc[c][2][2]); acc[c][2][3] = fmaf(a2, m.w, acc[c][2][3]);
                            acc[c][3][0] = fmaf(a3, m.x, acc[c][3][0]); acc[c][3][1] = fmaf(a3, m.y, acc[c][3][1]);
                            acc[c][3][2] = fmaf(a3, m.z, acc[c][3][2]); acc[c][3][3] = fmaf(a3, m.w, acc[c][3][3]);
                        }
                    }
                }
            }
            // per-control totals (AAR numerators) summed patch-ascending
            for (int c = 0; c < C; ++c) {
                __syncthreads();
                if (active) {
#pragma unroll
                    for (int cc = 0; cc < CMAX; ++cc) {
                        if (cc != c) continue;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            *reinterpret_cast<float4*>(mig + (size_t)(pg * 4 + i) * NE + kg * 4) =
                                make_float4(acc[cc][i][0], acc[cc][i][1], acc[cc][i][2], acc[cc][i][3]);
                    }
                }
                __syncthreads();
                for (int q = tid; q < TP; q += blockDim.x) {
                    const float* v = mig + (size_t)q * NE;
                    float tc = 0.0f;
                    for (int g4 = 0; g4 < NE; g4 += 4)
                        tc = tc + (((v[g4] + v[g4 + 1]) + v[g4 + 2]) + v[g4 + 3]);
                    int path = path0 + q;
                    if (path < P)
                        a.aars[(((size_t)s * C + c) * Y + t) * P + path] = tc / tot[q];
                }
            }
            __syncthreads();
            // growth under the path's random control
            if (active) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    int pl = pg * 4 + i;
                    uint32_t path = (uint32_t)(path0 + pl);
                    float z[4];
                    to_normal4(a.seed, TO_STREAM_GROWTH, road, path, t,
                               (uint32_t)((s * N4) >> 2) + kg, z);
                    int c = ctl[pl];
                    float mv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int cc = 0; cc < CMAX; ++cc)
                        if (cc == c)
#pragma unroll
                            for (int j = 0; j < 4; ++j) mv[j] = acc[cc][i][j];
                    float g = gm[pl];
                    float4 np;
                    float* npv = &np.x;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float m = mv[j];
                        float gr = (a.sem == 0) ? g + z[j] * sp[7] : fmaf(sp[7] * z[j], g, g);
                        float cp = cap4[j];
                        npv[j] = (a.sem == 0) ? m * (1.0f + gr * (cp - m) / cp / 100.0f)
                                              : fmaxf(m * (1.0f + gr * (cp - m) / cp), 0.0f);
                    }
                    *reinterpret_cast<float4*>(pop + (size_t)pl * NE + kg * 4) = np;
                }
            }
            __syncthreads();
            for (int q = tid; q < TP; q += blockDim.x) {
                const float* v = pop + (size_t)q * NE;
                float tt = 0.0f;
                for (int g4 = 0; g4 < NE; g4 += 4)
                    tt = tt + (((v[g4] + v[g4 + 1]) + v[g4 + 2]) + v[g4 + 3]);
                tot[q] = tt;
                int path = path0 + q;
                if (path < P) a.totalPops[((size_t)s * (Y + 1) + t + 1) * P + path] = tt;
            }
            __syncthreads();
        }
    }
}


// Unit profits of every path and year: those the regression states hold
// (profS) and those the decisions use (unitProfits) - the same but for
// reference semantics, whose two kernels read their process arrays with
// different strides.  A profit takes a Philox block and a Box-Muller pair,
// and the states, the query marks and the decisions of a year all use it.
__global__ void __launch_bounds__(256) k_rov_profit(to_rov_args a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = 1 + blockIdx.y, Y = a.Y;
    if (p >= a.PT) return;
    const size_t at = (size_t)t * a.PT + p;
    const float ps = unit_profit(a, p, t, Y + 1, Y + 1);
    a.profS[at] = ps;
    if (a.sem != 0) return;                    // profS is unitProfits
    a.unitProfits[at] = (t == Y - 1) ? unit_profit(a, p, t, Y + 1, Y) : unit_profit(a, p, t, Y, Y);
}

// terminal year (backwardInduction :2375-2463)
__global__ void k_rov_terminal(to_rov_args a) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.PT) return;
    const int t = a.Y - 1, C = a.C, S = a.S;
    float state[TO_ROV_MAXC * (TO_LSM_MAXD - 1) + 1];
    for (int c = 0; c < C; ++c)
        for (int s = 0; s < S; ++s) state[c * S + s] = adj_pop(a, p, t, s, c);
    state[S * C] = a.unitProfits[(size_t)t * a.PT + p];
    float best;
    int bc;
    to_rovd::decide_terminal(a, state, best, bc);
    a.condExp[(size_t)t * a.PT + p] = best;
    a.optCont[(size_t)t * a.PT + p] = bc;
    if (a.adjPops)
        for (int s = 0; s < S; ++s)
            a.adjPops[((size_t)t * S + s) * a.PT + p] = state[(C - 1) * S + s];
}

// order-preserving unsigned key of a float (min/max through integer atomics)
__device__ __forceinline__ unsigned lsm_key(float v) {
    unsigned k = __float_as_uint(v);
    return (k & 0x80000000u) ? ~k : (k | 0x80000000u);
}
__device__ __forceinline__ float lsm_unkey(unsigned k) {
    k = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
    return __uint_as_float(k);
}

// What the regressions of one (road, year) are fitted on, one CTA each:
//  1 the regression states of the road's paths, compacted stably by the
//    year's random control (allocateXYRegressionData :1012-1069; a path
//    whose species miss their thresholds under another control than 0 is
//    left out), with their ranges (computeStateMinMax :1073-1148);
//  2 counts, k, the reference's range rules and the grid axes
//    (createQueryPoints :1187-1190);
//  3 the normalised points (SimulateGPU.cu:4591-4603);
//  4 touched-query mode: k_rov_backward at this year reads control c's
//    regressions at the 2^d corners of the cell holding the path's own state
//    for c (to_lsm_interp), for every control valid for the path; exactly
//    those grid queries are marked in a bitmap;
//  5 the bitmaps as one ascending query list per group, cut into tiles of
//    TO_ROV_TILE for k_knn_rov.
// None of it depends on the values of later years, so a launch takes as many
// years as the scratch holds.  Latency bound (a CTA is a chain of short
// passes over a few hundred paths), which many CTAs an SM hide: 7.7 -> 1.5 ms
// a 256-road generation, 3.6 -> 0.22 ms a road of 10,000 paths (six kernels
// and a cell grid a year before).
constexpr int kPrepThreads = 512;
constexpr int kPrepBitmap = 32 * 1024;     // bytes of shared memory for the marks

__global__ void __launch_bounds__(kPrepThreads) k_lsm_prepare(to_rov_args a) {
    extern __shared__ unsigned s_bits[];
    constexpr int NW = kPrepThreads / 32;
    __shared__ int s_wcnt[NW][TO_ROV_MAXC];
    __shared__ int s_base[TO_ROV_MAXC];
    __shared__ unsigned s_key[TO_ROV_MAXC][TO_LSM_MAXD][2];
    __shared__ float s_mn[TO_ROV_MAXC + 1][TO_LSM_MAXD], s_mx[TO_ROV_MAXC + 1][TO_LSM_MAXD];
    __shared__ float s_lo[TO_LSM_MAXD], s_hi[TO_LSM_MAXD];      // ends of the raw axes
    __shared__ int s_scan[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = blockIdx.x, slot = blockIdx.y, t = a.slot0 + slot;
    const int P = a.P, S = a.S, C = a.C, R = a.R, Q = a.Q, d = S + 1, Y = a.Y;
    const size_t PT = (size_t)a.PT, p_0 = (size_t)r * P;
    const size_t gs0 = (size_t)slot * a.G + (size_t)r * C;      // first group of the slot's road
    float* xraw = a.xraw + gs0 * d * P;
    int* pidx = a.pidx + gs0 * P;

    // 1
    for (int q = tid; q < C * d; q += kPrepThreads) {
        s_key[q / d][q % d][0] = 0xFFFFFFFFu;
        s_key[q / d][q % d][1] = 0u;
    }
    if (tid < C) s_base[tid] = 0;
    for (int p0 = 0; p0 < P; p0 += kPrepThreads) {
        for (int q = tid; q < NW * C; q += kPrepThreads) s_wcnt[q / C][q % C] = 0;
        __syncthreads();                     // counts clear, keys set
        const int pl = p0 + tid;
        const size_t p = p_0 + pl;
        int c = -1;
        float xv[TO_LSM_MAXD];
        if (pl < P) {
            c = a.controls[(size_t)t * PT + p];
            bool ok = true;
            for (int s = 0; s < S; ++s) {
                xv[s] = adj_pop(a, (int)p, t, s, C - 1);
                if (xv[s] < a.params[8 * s + 3]) ok = false;
            }
            if (c != 0 && !ok) c = -1;
            xv[S] = a.profS[(size_t)t * PT + p];
        }
        const unsigned peers = __match_any_sync(0xffffffffu, c);
        const bool leader = lane == __ffs(peers) - 1;
        if (c >= 0) {
            if (leader) s_wcnt[warp][c] = __popc(peers);
            for (int j = 0; j < d; ++j) {
                const unsigned lo = __reduce_min_sync(peers, lsm_key(xv[j]));
                const unsigned hi = __reduce_max_sync(peers, lsm_key(xv[j]));
                if (leader) {
                    atomicMin(&s_key[c][j][0], lo);
                    atomicMax(&s_key[c][j][1], hi);
                }
            }
        }
        __syncthreads();
        if (c >= 0) {
            int pos = s_base[c] + __popc(peers & ((1u << lane) - 1u));
            for (int w = 0; w < warp; ++w) pos += s_wcnt[w][c];
            pidx[(size_t)c * P + pos] = (int)p;
            for (int j = 0; j < d; ++j) xraw[((size_t)c * d + j) * P + pos] = xv[j];
        }
        __syncthreads();
        if (tid < C) {
            int n = s_base[tid];
            for (int w = 0; w < NW; ++w) n += s_wcnt[w][tid];
            s_base[tid] = n;
        }
        __syncthreads();                     // before the next chunk clears the counts
    }
    // 2: each control's own ranges (control 0, and any with more than d + 1
    // points), then the others take control 0's
    for (int q = tid; q < C * d; q += kPrepThreads) {
        const int c = q / d, j = q - c * d;
        if (!((c == 0) || (s_base[c] > d + 1))) continue;
        float lo = 0.0f, hi = 0.0f;
        if (s_base[c] > 0) {
            lo = lsm_unkey(s_key[c][j][0]);
            hi = lsm_unkey(s_key[c][j][1]);
            // the reference scans from the first point with
            // "if (xmin > x) ... else if (xmax < x)": plain min and max,
            // except that a first value of -0/+0 keeps its sign when it is
            // the extreme
            const float first = xraw[((size_t)c * d + j) * P];
            if (lo == first) lo = first;
            if (hi == first) hi = first;
        }
        s_mn[c][j] = lo;
        s_mx[c][j] = hi;
    }
    __syncthreads();
    for (int q = tid; q < C * d; q += kPrepThreads) {
        const int c = q / d, j = q - c * d;
        if ((c == 0) || (s_base[c] > d + 1)) continue;
        s_mn[c][j] = s_mn[0][j];
        s_mx[c][j] = s_mx[0][j];
    }
    __syncthreads();
    if (tid < d) {
        const int j = tid;
        float lo = s_mn[0][j], hi = s_mx[0][j];
        for (int c = 1; c < C; ++c) {
            if (lo > s_mn[c][j]) lo = s_mn[c][j];
            if (hi < s_mx[c][j]) hi = s_mx[c][j];
        }
        s_mn[C][j] = lo;
        s_mx[C][j] = hi;
        s_lo[j] = to_lsm_query_axis(0, lo, hi, R);
        s_hi[j] = to_lsm_query_axis(R - 1, lo, hi, R);
    }
    __syncthreads();
    for (int q = tid; q < d * R; q += kPrepThreads) {
        const int j = q / R, di = q - j * R;
        const float lo = s_mn[C][j], hi = s_mx[C][j];
        const float raw = to_lsm_query_axis(di, lo, hi, R);
        a.qax[((size_t)slot * a.nr + r) * d * R + q] = to_lsm_normalise(raw, lo, hi, j == S, a.scaling);
        for (int c = 0; c < C; ++c) to_rov_reg_block(a, t, (size_t)r * C + c)[q] = raw;
    }
    if (tid < C) {
        const int n = s_base[tid];
        int k = 0;
        if (n > 3) {
            k = (int)((double)a.k_mult * (log((double)n) + 1.0));
            if (k > n) k = n;
        }
        a.npts[gs0 + tid] = n;
        a.kc[gs0 + tid] = k;
    }
    // 3 (in place unless the raw states are kept: reference semantics)
    float* xn = a.xn + gs0 * d * P;
    for (int cj = warp; cj < C * d; cj += NW) {
        const int c = cj / d, j = cj - c * d, n = s_base[c];
        const float lo = s_mn[C][j], hi = s_mx[C][j];
        for (int m = lane; m < n; m += 32)
            xn[(size_t)cj * P + m] = to_lsm_normalise(xraw[(size_t)cj * P + m], lo, hi, j == S,
                                                      a.scaling);
    }
    const int per = (Q + TO_ROV_TILE - 1) / TO_ROV_TILE;
    int2* tiles = a.tiles + (size_t)slot * a.G * per;
    if (!a.touched) {
        // every grid query of every group
        __shared__ int s_t0;
        if (tid == 0) s_t0 = atomicAdd(&a.ntiles[slot], C * per);
        if (tid < C) a.gcount[gs0 + tid] = Q;
        __syncthreads();
        for (int q = tid; q < C * per; q += kPrepThreads)
            tiles[s_t0 + q] = make_int2(r * C + q / per, (q % per) * TO_ROV_TILE);
        return;
    }
    // 4
    const int qw = (Q + 31) >> 5;
    unsigned* bits = a.bmap ? a.bmap + ((size_t)slot * a.nr + r) * C * qw : s_bits;
    for (int q = tid; q < C * qw; q += kPrepThreads) bits[q] = 0u;
    __syncthreads();
    for (int pl = tid; pl < P; pl += kPrepThreads) {
        const int p = (int)(p_0 + pl);
        const float prof = a.profS[(size_t)t * PT + p];
        const int lp = to_lsm_lower_index(prof, s_lo[S], s_hi[S], R);
        for (int c = 0; c < C; ++c) {
            bool valid = true;
            int base = 0;
            int li[TO_LSM_MAXD];
            for (int s = 0; s < S; ++s) {
                const float v = adj_pop(a, p, t, s, c);
                if (v < threshold(a, s) && c > 0) { valid = false; break; }
                li[s] = to_lsm_lower_index(v, s_lo[s], s_hi[s], R);
                base = base * R + li[s];
            }
            if (!valid) continue;
            base = base * R + lp;
            unsigned* mk = bits + (size_t)c * qw;
            for (int corner = 0; corner < (1 << S); ++corner) {
                // the corner's offset; its neighbour along the last dimension
                // lies one query further
                int idx = base, mul = R;
                for (int s = S - 1; s >= 0; --s) {
                    if ((corner >> (S - 1 - s)) & 1) idx += mul;
                    mul *= R;
                }
                const unsigned b0 = 1u << (idx & 31);
                if ((idx & 31) < 31) {
                    atomicOr(&mk[idx >> 5], b0 | (b0 << 1));
                } else {
                    atomicOr(&mk[idx >> 5], b0);
                    atomicOr(&mk[(idx >> 5) + 1], 1u);
                }
            }
        }
    }
    __syncthreads();
    // 5
    int fitted = 0;
    for (int c = 0; c < C; ++c) {
        const unsigned* mk = bits + (size_t)c * qw;
        const int chunk = (qw + kPrepThreads - 1) / kPrepThreads;
        const int w0 = tid * chunk, w1 = min(qw, w0 + chunk);
        int cnt = 0;
        for (int w = w0; w < w1; ++w) cnt += __popc(mk[w]);
        int x = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_scan[warp] = x;
        __syncthreads();
        int pos = x - cnt, total = 0;
        for (int w = 0; w < NW; ++w) { if (w < warp) pos += s_scan[w]; total += s_scan[w]; }
        int* list = a.qlist + (gs0 + c) * Q;
        for (int w = w0; w < w1; ++w)
            for (unsigned b = mk[w]; b; b &= b - 1) list[pos++] = w * 32 + __ffs(b) - 1;
        if (tid == 0) {
            a.gcount[gs0 + c] = total;
            const int nt = (total + TO_ROV_TILE - 1) / TO_ROV_TILE;
            const int t0 = nt > 0 ? atomicAdd(&a.ntiles[slot], nt) : 0;
            for (int i = 0; i < nt; ++i) tiles[t0 + i] = make_int2(r * C + c, i * TO_ROV_TILE);
        }
        fitted += total;
        __syncthreads();
    }
    if (tid == 0 && a.qroad && fitted) atomicAdd(&a.qroad[r], (unsigned)fitted);
}

// the values the year's points regress on, group by group (cell-grid search)
__global__ void __launch_bounds__(256) k_lsm_values(to_rov_args a, int t, int slot) {
    const int g = blockIdx.y, m = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t gs = (size_t)slot * a.G + g;
    if (m < a.npts[gs])
        a.yv[(size_t)g * a.P + m] = a.condExp[(size_t)(t + 1) * a.PT + a.pidx[gs * a.P + m]];
}

}  // namespace

namespace {

// backwardInduction for 0 < t < Y-1 (:2464-2776), a thread per path.  The
// interior decision of corrected semantics is unrolled for the number of
// species: states and corner weights in registers instead of arrays indexed
// at run time in local memory, the profit read instead of drawn again; and
// for up to CU controls, whose loads are then all in flight together (a
// control the path may not take is interpolated too and not looked at).
// Bound by the latency of the dependent loads (states, axes, 2^d corners;
// the regressions stay in L2): 47 -> 29 us a year of 196,608 paths of three
// species, 21 -> 10 us of 10,000 paths of two.  A year's fit and decisions
// follow one another 48 times, so each starts while the one before runs and
// loads what does not depend on it (to_pdl_wait; the fit after a selection
// starts at its end): 19 -> 14 us a year of those
// 10,000 paths, 25 -> 17 us of 2,000 under the reference's semantics.
template <int S, int CU>
__global__ void __launch_bounds__(128) k_rov_backward(to_rov_args a, int t) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    to_pdl_next();
    if (p >= a.PT) {
        to_pdl_wait();
        return;
    }
    const int C = a.C, R = a.R, r = p / a.P;
    const float prof = a.unitProfits[(size_t)t * a.PT + p];
    const float disc = 1.0f + a.rrr * a.dt / 100.0f;
    float tot[S];
#pragma unroll
    for (int s = 0; s < S; ++s) tot[s] = a.totalPops[((size_t)s * (a.Y + 1) + t) * a.PT + p];
    float best = 0.0f;
    int bc = 0;
    for (int c0 = 0; c0 < C; c0 += CU) {
        float pay[CU], st[CU][S];
        bool valid[CU];
#pragma unroll
        for (int u = 0; u < CU; ++u) {
            const int c = c0 + u < C ? c0 + u : C - 1;
            valid[u] = c0 + u < C;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                st[u][s] = tot[s] * a.aars[(((size_t)s * C + c) * a.Y + t) * a.PT + p];
                if (st[u][s] < a.params[8 * s + 3] && c > 0) valid[u] = false;
            }
            if (c == C - 1 && a.adjPops)
#pragma unroll
                for (int s = 0; s < S; ++s) a.adjPops[((size_t)t * S + s) * a.PT + p] = st[u][s];
        }
        to_pdl_wait();                         // the year's regressions
#pragma unroll
        for (int u = 0; u < CU; ++u) {
            const int c = c0 + u < C ? c0 + u : C - 1;
            const float cur = a.flows[c] * prof;
            const float v = to_lsm_interp(to_rov_reg_block(a, t, (size_t)r * C + c), R, S, st[u], prof);
            pay[u] = to_rovd::payoff(cur, v / disc);
        }
#pragma unroll
        for (int u = 0; u < CU; ++u)
            if (valid[u] && (c0 + u == 0 || pay[u] < best)) { best = pay[u]; bc = c0 + u; }
    }
    a.condExp[(size_t)t * a.PT + p] = best;
    a.optCont[(size_t)t * a.PT + p] = bc;
}

// reference semantics (one species)
__global__ void __launch_bounds__(128) k_rov_backward_ref(to_rov_args a, int t) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    to_pdl_next();
    if (p >= a.PT) {
        to_pdl_wait();
        return;
    }
    const int C = a.C, S = a.S;
    float state[TO_ROV_MAXC * (TO_LSM_MAXD - 1) + 1];
    for (int c = 0; c < C; ++c)
        for (int s = 0; s < S; ++s) state[c * S + s] = adj_pop(a, p, t, s, c);
    if (a.adjPops)
        for (int s = 0; s < S; ++s)
            a.adjPops[((size_t)t * S + s) * a.PT + p] = state[(C - 1) * S + s];
    state[S * C] = a.unitProfits[(size_t)t * a.PT + p];
    float best;
    int bc;
    to_pdl_wait();                             // the year's regressions
    to_rovd::decide_interior(a, t, p / a.P, state, best, bc);
    a.condExp[(size_t)t * a.PT + p] = best;
    a.optCont[(size_t)t * a.PT + p] = bc;
}

// firstPeriodInduction (:2210-2330) with FP64 reductions; one CTA a road.  The
// SM's FP64 rate (two lanes a clock) is what it waits for, so paths are
// counted in integers, a warp a control adds up the warps' sums, and what
// follows from them is worked out by one thread instead of all (2,000 paths:
// 71 -> 31 us, 10,000: 103 -> 67).
__global__ void __launch_bounds__(1024) k_rov_first(to_rov_args a) {
    // one CTA per road; its paths are base .. base+P-1 of the batch
    const int P = a.P, C = a.C, S = a.S, Y = a.Y;
    const size_t PT = (size_t)a.PT, base = (size_t)blockIdx.x * P;
    __shared__ double s_sum[TO_ROV_MAXC][32], s_pay[TO_ROV_MAXC], s_m1[32], s_vv[32];
    __shared__ int s_cnt[TO_ROV_MAXC][32], s_n[TO_ROV_MAXC], s_valid[TO_ROV_MAXC];
    __shared__ double s_best, s_mean;
    __shared__ int s_bc;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double discd = (double)(1.0f + a.rrr * a.dt / 100.0f);
    for (int c = 0; c < C; ++c) {
        double sum = 0.0;
        int cnt = 0;
#pragma unroll 4
        for (int p = threadIdx.x; p < P; p += blockDim.x)
            if (a.controls[base + p] == c) {
                sum += (double)a.condExp[PT + base + p];
                ++cnt;
            }
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0) { s_sum[c][warp] = sum; s_cnt[c][warp] = cnt; }
    }
    __syncthreads();
    for (int c = warp; c < C; c += nw)
        if (lane == 0) {
            double sm = 0.0;
            int n = 0;
            for (int w = 0; w < nw; ++w) { sm += s_sum[c][w]; n += s_cnt[c][w]; }
            s_n[c] = n;
            s_pay[c] = n > 0 ? sm / ((double)n * discd) : 0.0;
            bool valid = true;
            for (int s = 0; s < S; ++s) {
                float adj = a.totalPops[((size_t)s * (Y + 1)) * PT + base] *
                            a.aars[(((size_t)s * C + c) * Y) * PT + base];
                if (adj < threshold(a, s) && c > 0) valid = false;
            }
            s_valid[c] = valid;
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        float uf = 0.0f, ore = 0.0f;
        for (int f = 0; f < a.nF; ++f)
            uf = fmaf(a.fuel_costs[f], a.uRes[((size_t)a.fuel_idx[f] * (Y + 1)) * PT + base], uf);
        for (int c = 0; c < a.Cm; ++c)
            ore = fmaf(ore_at(a, (int)base, 0, c),
                       a.uRes[((size_t)(a.nF + c) * (Y + 1)) * PT + base], ore);
        float prof0 = (a.unit_cost + uf) - a.unit_revenue * ore;
        if (a.demand_idx >= 0)
            prof0 = prof0 * a.uRes[((size_t)a.demand_idx * (Y + 1)) * PT + base];
        double pay[TO_ROV_MAXC];
        int stop = C;
        for (int c = 0; c < C; ++c) {
            if (s_n[c] <= 0) { stop = c; break; }
            pay[c] = s_pay[c];
            if (s_valid[c]) {
                pay[c] += (double)(a.flows[c] * prof0);
                if (pay[c] > 0.0) pay[c] = 0.0;
            } else pay[c] = NAN;
        }
        for (int c = stop; c < C; ++c) pay[c] = (c == 0) ? 0.0 : NAN;
        double best = pay[0];
        int bc = 0;
        for (int c = 1; c < C; ++c)
            if (isfinite(pay[c]) && pay[c] < best) { best = pay[c]; bc = c; }
        s_best = best;
        s_bc = bc;
    }
    __syncthreads();
    const double best = s_best;
    const int bc = s_bc;
    double ss = 0.0, m1 = 0.0;
#pragma unroll 4
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        if (a.controls[base + p] == bc) {
            double v = (double)a.condExp[PT + base + p];
            ss += (v - best) * (v - best);
            m1 += v;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        m1 += __shfl_xor_sync(0xffffffffu, m1, o);
    }
    if (lane == 0) { s_sum[0][warp] = ss; s_m1[warp] = m1; }
    __syncthreads();
    const double N1 = (double)s_n[bc];
    if (threadIdx.x == 0) {
        double M1 = 0.0;
        for (int w = 0; w < nw; ++w) M1 += s_m1[w];
        s_mean = N1 > 0.0 ? M1 / N1 : 0.0;
    }
    __syncthreads();
    // sample variance of the chosen control's year-1 values
    const double mean = s_mean;
    double vv = 0.0;
#pragma unroll 4
    for (int p = threadIdx.x; p < P; p += blockDim.x)
        if (a.controls[base + p] == bc) {
            double v = (double)a.condExp[PT + base + p] - mean;
            vv += v * v;
        }
    for (int o = 16; o > 0; o >>= 1) vv += __shfl_xor_sync(0xffffffffu, vv, o);
    if (lane == 0) s_vv[warp] = vv;
    __syncthreads();
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        a.condExp[base + p] = (float)best;
        a.optCont[base + p] = bc;
    }
    if (threadIdx.x == 0) {
        double SS = 0.0, V = 0.0;
        for (int w = 0; w < nw; ++w) { SS += s_sum[0][w]; V += s_vv[w]; }
        double sdfac = (a.sem == 0) ? (1.0 + (double)a.rrr / (100.0 * (double)a.dt)) : discd;
        double* st = a.stats + 5 * (size_t)blockIdx.x;
        st[0] = (double)(float)best;
        st[1] = (double)bc;
        st[2] = (N1 > 0.0) ? sqrt(SS / (N1 * sdfac)) : 0.0;
        st[3] = (N1 > 1.0) ? sqrt(V / (N1 - 1.0)) / sqrt(N1) / discd : 0.0;
        st[4] = N1;
    }
}

}  // namespace

namespace to_k {

to_status rov_backward(to_ctx ctx, const to_rov_args& a, int pblocks, int tpb,
                       const to_csc* csc);

to_status rov_run(to_ctx ctx, to_rov_args a, const to_csc* csc) {
    const int P = a.PT;                        // every path of the batch
    a.rk = to_make_round_keys(a.seed);
    const int tpb = 128;
    const int pblocks = (P + tpb - 1) / tpb;
    to_prof_begin(ctx, "rov_exog");
    k_rov_exog<<<(P + 31) / 32, kExThreads, 0, ctx->stream>>>(a);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    if (csc) {
        TO_TRY(rov_forward_sparse(ctx, a, *csc));
        return rov_backward(ctx, a, pblocks, tpb, csc);
    }
    if (a.nr != 1)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "batched roads need the sparse migration form");
    // forward tile shape
    const int NE = a.ne, KG = NE / 4;
    int pgroups = 256 / KG;
    if (pgroups < 1) pgroups = 1;
    if (pgroups > 16) pgroups = 16;
    if (pgroups * KG > 1024) return to_set_error(ctx, TO_ERR_UNSUPPORTED, "patches %d", NE);
    a.tile_paths = 4 * pgroups;
    size_t fixed = (size_t)(2 * a.tile_paths * NE + 3 * a.tile_paths) * sizeof(float);
    size_t budget = 200 * 1024;
    if (fixed + (size_t)a.C * NE * NE * 4 <= budget) a.l_chunk = NE;
    else {
        int lc = 64;
        while (lc > 4 && (fixed + (size_t)a.C * lc * NE * 4 > budget || NE % lc)) lc >>= 1;
        if (NE % lc) lc = 4;
        a.l_chunk = lc;
    }
    size_t smem = fixed + (size_t)a.C * a.l_chunk * NE * sizeof(float);
    dim3 grid((P + a.tile_paths - 1) / a.tile_paths);
    int threads = ((pgroups * KG + 31) / 32) * 32;
    if (a.C > TO_ROV_MAXC) return to_set_error(ctx, TO_ERR_UNSUPPORTED, "controls %d", a.C);
    to_prof_begin(ctx, "rov_forward");
    if (a.C <= 3) {
        TO_CUDA(ctx, cudaFuncSetAttribute(k_rov_forward<3>,
                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_rov_forward<3><<<grid, threads, smem, ctx->stream>>>(a);
    } else {
        TO_CUDA(ctx, cudaFuncSetAttribute(k_rov_forward<TO_ROV_MAXC>,
                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_rov_forward<TO_ROV_MAXC><<<grid, threads, smem, ctx->stream>>>(a);
    }
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return rov_backward(ctx, a, pblocks, tpb, nullptr);
}

// bytes of one prepared year, besides the fixed ones
static size_t slot_bytes(const to_rov_args& a, int max_roads) {
    const size_t G = (size_t)max_roads * a.C, d = a.S + 1;
    const size_t per = (a.Q + TO_ROV_TILE - 1) / TO_ROV_TILE;
    return G * d * a.P * 4 * (a.sem == 0 ? 2 : 1) + G * a.P * 4 + (a.touched ? G * a.Q * 4 : 0) +
           G * per * 8 + (a.reg_by_slot ? G * ((size_t)a.R * d + 2 * (size_t)a.Q) * 4 : 0);
}

void rov_plan(to_rov_args& a, int max_roads) {
    // all years where they fit in half a gigabyte (a road, a small batch); a
    // 256-road generation takes a few at a time, enough CTAs a launch
    const auto fit = [&](size_t bytes, size_t most) {
        const size_t n = ((size_t)512 << 20) / (bytes > 0 ? bytes : 1);
        return (int)(n < 1 ? 1 : (n > most ? most : n));
    };
    a.slots = fit(slot_bytes(a, max_roads), (size_t)a.Y - 2);
    a.sel_slots = fit(knn_select_bytes(a, max_roads), (size_t)a.slots);
}

size_t rov_scratch(to_rov_args& a, int max_roads, char* base) {
    const size_t T = a.slots, NR = max_roads, G = NR * a.C, d = a.S + 1, P = a.P, Q = a.Q;
    const size_t per = (Q + TO_ROV_TILE - 1) / TO_ROV_TILE, qw = (Q + 31) / 32;
    size_t off = 0;
    auto take = [&](size_t b) {
        char* p = base ? base + off : nullptr;
        off += to_align256(b);
        return p;
    };
    a.xn = (float*)take(T * G * d * P * 4);
    a.xraw = a.sem == 0 ? (float*)take(T * G * d * P * 4) : a.xn;
    a.pidx = (int*)take(T * G * P * 4);
    a.npts = (int*)take(T * G * 4);
    a.kc = (int*)take(T * G * 4);
    a.qax = (float*)take(T * NR * d * a.R * 4);
    a.qlist = a.touched ? (int*)take(T * G * Q * 4) : nullptr;
    a.gcount = (int*)take(T * G * 4);
    a.tiles = (int2*)take(T * G * per * 8);
    a.ntiles = (int*)take(2 * T * 4);
    a.bmap = (a.touched && a.C * qw * 4 > (size_t)kPrepBitmap)
                 ? (unsigned*)take(T * NR * a.C * qw * 4) : nullptr;
    a.profS = a.sem == 0 ? (float*)take((size_t)a.Y * NR * P * 4) : a.unitProfits;
    a.fwd_next = (int*)take(4);
    if (a.C <= 3) {
        a.fwd_part = (f2*)take((size_t)a.ctas * 2 * a.C * (a.np / 4) * 32 * 8);
        a.fwd_far = (f2*)take((size_t)a.ctas * a.np * 32 * 8);
    }
    if (a.P <= TO_ROV_SCAN_PATHS) {
        const size_t tiles = (size_t)a.sel_slots * G * per;
        a.nbr = (unsigned short*)take(tiles * TO_ROV_TILE * a.kmax * 2);
        a.kthv = (float*)take(tiles * TO_ROV_TILE * 4);
    } else {
        a.yv = (float*)take(G * P * 4);
        a.gsx = (float*)take(G * d * P * 4);
        a.gsi = (int*)take(G * P * 4);
        a.gcell = (int*)take(G * (TO_KNN_GCELLS + 1) * 4);
        a.ggrid = (to_knn_grid*)take(G * sizeof(to_knn_grid));
        a.kth = (float*)take(G * Q * 4);
        a.knn_acc = (double*)take(G * Q * ((d + 1) * (d + 4) / 2) * 8);
    }
    return off;
}

to_status rov_backward(to_ctx ctx, const to_rov_args& args, int pblocks, int tpb,
                       const to_csc* csc) {
    to_rov_args a = args;
    if (a.algo == 6 && (!csc || !a.popsY || !a.gmY || a.nr != 1))
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "ALGO6 needs the sparse forward pass, one road");
    if (a.touched && (a.sem != 1 || a.algo != 4 || !a.qlist))
        return to_set_error(ctx, TO_ERR_INVALID, "touched-query mode: sem 1, ALGO4, scratch");
    if (a.slots < 1 || (size_t)a.G * a.Q > (size_t)0x7fffffff)
        return to_set_error(ctx, TO_ERR_INVALID, "regression scratch: %d years", a.slots);
    if (a.S < 1 || a.S + 1 > TO_LSM_MAXD)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "%d species", a.S);
    const bool scan = a.P <= TO_ROV_SCAN_PATHS;
    // the cell-grid search starts a query from its k-th distance a year
    // later; cleared so that every valuation starts the same way
    if (!scan) TO_CUDA(ctx, cudaMemsetAsync(a.kth, 0, (size_t)a.G * a.Q * 4, ctx->stream));
    if (a.qroad) TO_CUDA(ctx, cudaMemsetAsync(a.qroad, 0, (size_t)a.nr * sizeof(unsigned), ctx->stream));
    to_prof_begin(ctx, "lsm_prepare");
    k_rov_profit<<<dim3((a.PT + 255) / 256, a.Y - 1), 256, 0, ctx->stream>>>(a);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    k_rov_terminal<<<pblocks, tpb, 0, ctx->stream>>>(a);
    TO_LAUNCHED(ctx);
    const size_t bits = (a.touched && !a.bmap) ? (size_t)a.C * ((a.Q + 31) / 32) * 4 : 0;
    TO_CUDA(ctx, cudaFuncSetAttribute(k_lsm_prepare, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kPrepBitmap));
    to_rov_years y(a.Y, a.slots, a.sel_slots);
    while (y.next()) {
        const int t = y.t;
        if (y.prepare) {
            a.slot0 = y.low;
            to_prof_begin(ctx, "lsm_prepare");
            TO_CUDA(ctx, cudaMemsetAsync(a.ntiles, 0, 2 * (size_t)a.slots * sizeof(int), ctx->stream));
            k_lsm_prepare<<<dim3(a.nr, y.prepare), kPrepThreads, bits, ctx->stream>>>(a);
            to_prof_end(ctx);
            TO_LAUNCHED(ctx);
        }
        if (scan) {
            if (y.select) {
                a.sel0 = y.sel - y.low;
                TO_TRY(knn_rov_select(ctx, a, y.select));
            }
            TO_TRY(knn_rov_fit(ctx, a, t, y.fit_ahead()));
        } else {
            k_lsm_values<<<dim3((a.P + 255) / 256, a.G), 256, 0, ctx->stream>>>(a, t, t - a.slot0);
            TO_LAUNCHED(ctx);
            TO_TRY(knn_rov_grid(ctx, a, t));
        }
        to_prof_begin(ctx, "rov_backward");
        TO_CUDA(ctx, to_pdl_launch(true, a.sem == 0 ? k_rov_backward_ref
                                   : a.S == 1 ? k_rov_backward<1, 3>
                                   : a.S == 2 ? k_rov_backward<2, 3>
                                   : a.S == 3 ? k_rov_backward<3, 3>
                                              : k_rov_backward<4, 3>,
                                   pblocks, tpb, 0, ctx->stream, a, t));
        to_prof_end(ctx);
        TO_LAUNCHED(ctx);
        // ALGO6: the year's value becomes the realised payoff of each path
        // re-simulated from year t under the regression-optimal controls
        if (a.algo == 6) TO_TRY(rov_resim_sparse(ctx, a, *csc, t));
    }
    k_rov_first<<<a.nr, 1024, 0, ctx->stream>>>(a);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

}  // namespace to_k
