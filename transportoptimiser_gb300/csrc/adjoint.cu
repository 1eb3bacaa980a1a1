// adjoint.cu - pathwise sensitivities of the controlled road valuation with
// the exercise policy frozen (no counterpart in the reference, which only
// estimates values).
//
// The frozen-policy model, per path p and year t = 0..Y-1, control c_{p,t}
// fixed (e.g. the optimal controls of a forward LSM pass):
//   exogenous processes (forwardPathKernel, SimulateGPU.cu:930-952)
//     U_{t+1} = U_t + theta (mu - U_t) dt + U_t sigma z_t + (e^{j_t} - 1) U_t J_t
//   unit profit (as the ROV's, SimulateGPU.cu:2375-2420)
//     pi_t = (unit_cost + sum_f fuel_f U_f - revenue sum_c ore_c U_{nF+c}) U_demand
//   PV = sum_t (1 + rrr dt / 100)^-t flows[c_t] pi_t
//   per species s: growth-rate mean g (mteKernel :691-701), migration with
//   the control's matrix M_c (survival exp(-crossings * hazard_c) inside),
//   corrected logistic growth x' = max(m (1 + gr (cap - m) / cap), 0) with
//   gr = g (1 + v z), and end population E_s = sum_k x_Y[k].
// Parameters theta (2U + 2S + C): reversion theta_u, volatility sigma_u,
// growth-rate mean mu_s (params[1]), growth variability v_s (params[7]),
// crossing hazard h_c (scales entry (k, l) of M_c by exp(-cross_lk dh_c)).
// Outputs: E[PV], E[E_s].
//
// Forward: PV per path (a thread per path) and the population recursion with
// the states checkpointed every K years.  Backward (vector-Jacobian
// product): forward tangents for the scalar recursions (OU, growth-rate
// mean), and a reverse sweep for the patch populations: each K-year segment
// is recomputed from its checkpoint, then lambda_t = M_c^T (lambda_{t+1} .
// dF/dm) with the parameter terms accumulated on the way.  Per-path
// contributions are averaged in FP64.
//
// The population sweeps run a CTA of 16 warps on 64 paths of one species:
// lane = two paths, packed (to_f2.cuh); the warps take groups of four
// patches, so that one Philox block serves the four normals it holds; a
// patch's migration is one list of the patches it exchanges animals with,
// each entry holding every control's value, of which a lane reads its own
// control's - one multiply-add a path and entry whatever the number of
// controls.  The states that other patches read are in shared memory, a
// segment's states and migrated states in global memory (they stay in L2).
// Bound by instruction issue and the latency of the lists' loads: two species
// of 115 patches, 10,000 paths, 50 years: forward 9.1 -> 0.9 ms, a species'
// reverse sweep 20 -> 2.0 ms (a thread a path over all patches and every
// control's pairs before).
#include <cmath>
#include <vector>

#include "to_f2.cuh"
#include "to_internal.cuh"

namespace {

constexpr int kCk = 10;                 // checkpoint interval (years)

struct AdjArgs {
    int P, Y, S, C, U, NP, nF, Cm, demand_idx, road;
    float dt, rrr, unit_cost, unit_revenue;
    uint64_t seed;
    const float* theta;                 // [2U + 2S + C] device
    const float* uncert;                // [U][6]
    const float* flows;                 // [C]
    const float* fuel_costs;            // [nF]
    const int* fuel_idx;                // [nF]
    const float* ore_content;           // [Cm]
    const float* ore_sd;                // [Cm]
    const int* controls;                // [Y][P]
    const int* n_patches;               // [S]
    const float* params;                // [S][8]
    const float* init_pops;             // [S][NP]
    const float* caps;                  // [S][NP]
    // migration lists of every species: patch k's entries [uptr[s][k],
    // uptr[s][k + 1]) are the patches it receives from, ascending; the
    // transposed lists those it sends to.  Entry e holds the values of all
    // controls at the current hazards (k_adj_values) and a zero, which a
    // control outside 0 .. C - 1 reads: under it nothing migrates or earns
    const int *uptr, *tptr;             // [S][NP + 1]
    const int *ul, *tk;                 // [E] the other patch
    const int* tsrc;                    // [E] the transposed entry's place in the first lists
    const int4* uchain;                 // [E] first lists: 32 origin, 32 destination, -crossings
    const float* base_v;                // [E][C + 1] values at the base hazards
    float *uval, *tval;                 // [E][C + 1]
    const float* base_h;                // [C] hazards the values were built with
    int E;
    to_round_keys rk;
    // tape
    float* ckpt;                        // [S][Y/K + 1][NP][P]
    // scratch of a sweep's CTAs, which take one (species, tile) after another:
    // a tile's own would be 25 rows a path beside the 6 of its checkpoints
    int slots;                          // of the scratch: the most CTAs at work
    f2* segx;                           // [slots][K][NP][32] a segment's states
    f2* segm;                           // [slots][K][NP][32] and migrated states
    f2* terms;                          // [slots][2][2][NP][32] a year's terms of mu_s and v_s
    f2* lam;                            // [slots][NP][32] adjoint of a segment's first state
    f2* rows;                           // [slots][NP][32] rows shared memory has no room for
    float* gtab;                        // [S][Y][P] growth-rate mean used in year t
    float* gdot;                        // [S][Y][P] its derivative in mu_s
    double* pv;                         // [P]
    double* endp;                       // [S][P]
    double* gpath;                      // [P][ntheta] per-path vector-Jacobian products
    const float* gout;                  // [1 + S] output weights
};

__device__ __forceinline__ float th_theta(const AdjArgs& a, int u) { return a.theta[u]; }
__device__ __forceinline__ float th_sigma(const AdjArgs& a, int u) { return a.theta[a.U + u]; }
__device__ __forceinline__ float th_mu(const AdjArgs& a, int s) { return a.theta[2 * a.U + s]; }
__device__ __forceinline__ float th_v(const AdjArgs& a, int s) { return a.theta[2 * a.U + a.S + s]; }
__device__ __forceinline__ float th_h(const AdjArgs& a, int c) { return a.theta[2 * a.U + 2 * a.S + c]; }

__device__ __forceinline__ float ore_at(const AdjArgs& a, int p, int t, int c) {
    const long f = (long)c * a.Y * a.P + (long)p * a.Y + t;
    const float z = to_normal1(a.seed, TO_STREAM_ORE, (uint32_t)a.road, (uint32_t)(f >> 2), 0,
                               (uint32_t)(f & 3));
    return a.ore_content[c] + a.ore_sd[c] * z;
}

// OU paths with optional tangents (dU/dtheta_u, dU/dsigma_u) and the PV and
// its gradient.  mode 0: PV only; mode 1: gradient terms weighted by w.
__device__ void exog_path(const AdjArgs& a, int p, bool tangents, double* pv_out, float* gth,
                          float* gsg) {
    constexpr int UMAX = 8;
    float U[UMAX], dth[UMAX], dsg[UMAX];
    for (int u = 0; u < a.U; ++u) { U[u] = a.uncert[6 * u]; dth[u] = 0.0f; dsg[u] = 0.0f; gth[u] = 0.0f; gsg[u] = 0.0f; }
    double pv = 0.0;
    float disc = 1.0f;
    const float dfac = 1.0f / (1.0f + a.rrr * a.dt / 100.0f);   // rrr in percent, as the ROV
    for (int t = 0; t < a.Y; ++t) {
        // unit profit at U_t and its partials
        float uf = 0.0f, ore = 0.0f;
        float dpi_du[UMAX];
        for (int u = 0; u < a.U; ++u) dpi_du[u] = 0.0f;
        for (int f = 0; f < a.nF; ++f) uf = fmaf(a.fuel_costs[f], U[a.fuel_idx[f]], uf);
        float oc[UMAX];
        for (int c = 0; c < a.Cm; ++c) {
            oc[c] = ore_at(a, p, t, c);
            ore = fmaf(oc[c], U[a.nF + c], ore);
        }
        const float base = (a.unit_cost + uf) - a.unit_revenue * ore;
        const float dem = a.demand_idx >= 0 ? U[a.demand_idx] : 1.0f;
        const float pi = base * dem;
        const int ctl = a.controls[(size_t)t * a.P + p];
        const float w = (unsigned)ctl < (unsigned)a.C ? disc * a.flows[ctl] : 0.0f;
        pv += (double)(w * pi);
        if (tangents) {
            for (int f = 0; f < a.nF; ++f) dpi_du[a.fuel_idx[f]] += a.fuel_costs[f] * dem;
            for (int c = 0; c < a.Cm; ++c) dpi_du[a.nF + c] += -a.unit_revenue * oc[c] * dem;
            if (a.demand_idx >= 0) dpi_du[a.demand_idx] += base;
            for (int u = 0; u < a.U; ++u) {
                gth[u] += w * dpi_du[u] * dth[u];
                gsg[u] += w * dpi_du[u] * dsg[u];
            }
        }
        // advance the processes to t + 1
        for (int u = 0; u < a.U; ++u) {
            const float* up = a.uncert + 6 * u;
            const float uj = to_uniform1(a.seed, TO_STREAM_EX_JUMP, (uint32_t)a.road, p, t, u);
            const float zb = to_normal1(a.seed, TO_STREAM_EX_BROWNIAN, (uint32_t)a.road, p, t, u);
            const float zj = to_normal1(a.seed, TO_STREAM_EX_JUMPSIZE, (uint32_t)a.road, p, t, u);
            const float jump = (uj < up[5]) ? 1.0f : 0.0f;
            const float s4 = up[4] * up[4];
            const float jf = (to_expf(zj * up[4] - s4 / 2.0f) - 1.0f) * jump;
            const float th = th_theta(a, u), sg = th_sigma(a, u);
            const float cur = U[u];
            const float mult = 1.0f - th * a.dt + sg * zb + jf;
            if (tangents) {
                dth[u] = dth[u] * mult + (up[1] - cur) * a.dt;
                dsg[u] = dsg[u] * mult + cur * zb;
            }
            U[u] = cur + th * (up[1] - cur) * a.dt + cur * (zb * sg) + jf * cur;
        }
        disc *= dfac;
    }
    *pv_out = pv;
}

__global__ void k_adj_pv(AdjArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.P) return;
    float gth[8], gsg[8];
    double pv;
    exog_path(a, p, false, &pv, gth, gsg);
    a.pv[p] = pv;
}

__global__ void k_adj_pv_grad(AdjArgs a, int ntheta) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.P) return;
    float gth[8], gsg[8];
    double pv;
    exog_path(a, p, true, &pv, gth, gsg);
    const float w = a.gout[0];
    double* g = a.gpath + (size_t)p * ntheta;
    for (int u = 0; u < a.U; ++u) {
        g[u] = (double)(w * gth[u]);
        g[a.U + u] = (double)(w * gsg[u]);
    }
}

// growth-rate mean of species s in year t (updated before the year's
// growth) and its derivative in mu_s, for every year; a thread per (species,
// path)
__global__ void __launch_bounds__(128) k_adj_growth(AdjArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.y;
    if (p >= a.P) return;
    const float* sp = a.params + 8 * s;
    const float mu = th_mu(a, s);
    float g = sp[0], gd = 0.0f;
    for (int t = 0; t < a.Y; ++t) {
        const float uj = to_uniform1(a.seed, TO_STREAM_SP_JUMP, (uint32_t)a.road, p, t, s);
        const float zb = to_normal1(a.seed, TO_STREAM_SP_BROWNIAN, (uint32_t)a.road, p, t, s);
        const float zj = to_normal1(a.seed, TO_STREAM_SP_JUMPSIZE, (uint32_t)a.road, p, t, s);
        const float jump = (uj < sp[6]) ? 1.0f : 0.0f;
        const float s5 = sp[5] * sp[5];
        const float jf = (to_expf(zj * sp[5] - s5 / 2.0f) - 1.0f) * jump;
        const float mult = 1.0f - sp[4] * a.dt + zb * sp[2] + jf;
        gd = gd * mult + sp[4] * a.dt;
        g = g + sp[4] * (mu - g) * a.dt + g * (zb * sp[2]) + jf * g;
        a.gtab[((size_t)s * a.Y + t) * a.P + p] = g;
        a.gdot[((size_t)s * a.Y + t) * a.P + p] = gd;
    }
}

// the lists' values at the hazards theta holds
__global__ void __launch_bounds__(256) k_adj_values(AdjArgs a) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.E) return;
    const int src = a.tsrc[e];
    const float x = __int_as_float(a.uchain[e].z), xs = __int_as_float(a.uchain[src].z);
    const int W = a.C + 1;
    for (int c = 0; c < W; ++c) {
        const float dh = c < a.C ? th_h(a, c) - a.base_h[c] : 0.0f;
        a.uval[(size_t)e * W + c] = a.base_v[(size_t)e * W + c] *
                                    (dh == 0.0f ? 1.0f : to_expf(x * dh));
        a.tval[(size_t)e * W + c] = a.base_v[(size_t)src * W + c] *
                                    (dh == 0.0f ? 1.0f : to_expf(xs * dh));
    }
}

constexpr int kAdjThreads = 512, kAdjWarps = kAdjThreads / 32;
constexpr int kAdjPaths = 64;                  // paths of a CTA, two a lane
constexpr int kAdjStatic = 3072;               // static shared memory and slack

// what the sweeps of one (tile, species) share
struct AdjTile {
    int s, N, N4, p0, p1;                      // species, patches, the lane's paths
    bool live0, live1;
    float v;                                   // growth variability
    const int *up, *tp;                        // list starts
    const float* cap;
    to_path_stream ps0, ps1;
    uint32_t stream_road, group0;
    const to_bm_tables* tab;
};

__host__ __device__ inline int adj_tiles(const AdjArgs& a) { return (a.P + kAdjPaths - 1) / kAdjPaths; }
// item: the (species, tile), tiles of a species in a row
__device__ __forceinline__ AdjTile adj_tile(const AdjArgs& a, const to_bm_tables* tab, int item) {
    AdjTile q;
    const int tiles = adj_tiles(a);
    q.s = item / tiles;
    q.N = a.n_patches[q.s];
    q.N4 = (q.N + 3) & ~3;
    q.p0 = (item - q.s * tiles) * kAdjPaths + (threadIdx.x & 31);
    q.p1 = q.p0 + 32;
    q.live0 = q.p0 < a.P;
    q.live1 = q.p1 < a.P;
    q.v = th_v(a, q.s);
    q.up = a.uptr + (size_t)q.s * (a.NP + 1);
    q.tp = a.tptr + (size_t)q.s * (a.NP + 1);
    q.cap = a.caps + (size_t)q.s * a.NP;
    to_stream_path(q.ps0, (uint32_t)(q.live0 ? q.p0 : 0));
    to_stream_path(q.ps1, (uint32_t)(q.live1 ? q.p1 : 0));
    q.stream_road = TO_STREAM_GROWTH | ((uint32_t)a.road << 8);
    q.group0 = (uint32_t)((q.s * q.N4) >> 2);
    q.tab = tab;
    return q;
}

// the lane's controls (columns of the lists' values) and growth means of
// year t, and its streams set to that year; paths past the end: nothing
// migrates, growth of path 0
struct AdjYear {
    int c0, c1;
    f2 g, gd;
};
__device__ __forceinline__ AdjYear adj_year(const AdjArgs& a, AdjTile& q, int t) {
    AdjYear y;
    const size_t row = (size_t)t * a.P, sr = ((size_t)q.s * a.Y + t) * a.P;
    const int p0 = q.live0 ? q.p0 : 0, p1 = q.live1 ? q.p1 : 0;
    y.c0 = q.live0 ? a.controls[row + p0] : a.C;
    y.c1 = q.live1 ? a.controls[row + p1] : a.C;
    if ((unsigned)y.c0 > (unsigned)a.C) y.c0 = a.C;
    if ((unsigned)y.c1 > (unsigned)a.C) y.c1 = a.C;
    y.g = pack2(a.gtab[sr + p0], a.gtab[sr + p1]);
    y.gd = pack2(a.gdot[sr + p0], a.gdot[sr + p1]);
    to_stream_year(q.ps0, (uint32_t)t, a.rk);
    to_stream_year(q.ps1, (uint32_t)t, a.rk);
    return y;
}

__device__ __forceinline__ void adj_normals(const AdjArgs& a, const AdjTile& q, int grp, f2 (&z)[4]) {
    to_normal4x2(q.ps0, q.ps1, to_stream_group(q.group0 + grp, q.stream_road, a.rk), a.rk, *q.tab, z);
}

// sum over entries [e0, e1) of a list: the values of the lane's controls
// times the other patches' rows.  A value is zero where another control has
// the pair, which is no term of this control's: that matters where the row is
// infinite, and the sum is then made again without the zeros.
__device__ __forceinline__ f2 adj_list_sum(const float* val, const int* other, int W, int e0, int e1,
                                           int c0, int c1, const f2* rows) {
    f2 acc = 0ull;
#pragma unroll 4
    for (int e = e0; e < e1; ++e) {
        const float* v = val + (size_t)e * W;
        acc = fma2(pack2(v[c0], v[c1]), rows[other[e] * 32], acc);
    }
    float s0, s1;
    unpack2(acc, s0, s1);
    if (s0 == s0 && s1 == s1) return acc;
    s0 = s1 = 0.0f;
#pragma unroll 1
    for (int e = e0; e < e1; ++e) {
        const float v0 = val[(size_t)e * W + c0], v1 = val[(size_t)e * W + c1];
        float x0, x1;
        unpack2(rows[other[e] * 32], x0, x1);
        if (v0 != 0.0f) s0 = fmaf(v0, x0, s0);
        if (v1 != 0.0f) s1 = fmaf(v1, x1, s1);
    }
    return pack2(s0, s1);
}

// migrated state of patch k
__device__ __forceinline__ f2 adj_migrated(const AdjArgs& a, const AdjTile& q, int k,
                                           const AdjYear& y, const f2* rows) {
    return adj_list_sum(a.uval, a.ul, a.C + 1, q.up[k], q.up[k + 1], y.c0, y.c1, rows);
}

// minus x / c.  A capacity with a normal reciprocal: multiply by it and
// correct once, which gives the division's bits for quotients in the normal
// range, and an infinite quotient without the correction, whose remainder is
// not a number; any other capacity: divide.
struct AdjCap {
    f2 c, nr;
    float cap;
    bool normal;
};
__device__ __forceinline__ AdjCap adj_cap(float cap) {
    AdjCap r;
    r.cap = cap;
    r.normal = fabsf(cap) > 1e-30f && fabsf(cap) < 1e30f;
    r.c = both2(cap);
    r.nr = both2(-(1.0f / cap));
    return r;
}
__device__ __forceinline__ f2 adj_neg_div(f2 x, const AdjCap& c) {
    if (c.normal) {
        const f2 nq = mul2(x, c.nr);
        float d0, d1, q0, q1;
        unpack2(fma2(fma2(nq, c.c, x), c.nr, nq), d0, d1);
        unpack2(nq, q0, q1);
        return pack2(d0 == d0 ? d0 : q0, d1 == d1 ? d1 : q1);
    }
    float x0, x1;
    unpack2(x, x0, x1);
    return neg2(pack2(x0 / c.cap, x1 / c.cap));
}

// one year forward: the next states from the rows x (to nx), and for the
// reverse sweep the migrated and next states (own patches' rows only)
__device__ __forceinline__ void adj_step(const AdjArgs& a, const AdjTile& q, const AdjYear& y,
                                         const f2* x, f2* nx, f2* segm, f2* segx) {
    const int lane = threadIdx.x & 31;
    const f2 v2 = both2(q.v), one = both2(1.0f), mone = both2(-1.0f);
    for (int grp = threadIdx.x >> 5; grp < q.N4 / 4; grp += kAdjWarps) {
        f2 z[4];
        adj_normals(a, q, grp, z);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = grp * 4 + j;
            if (k >= q.N) break;
            const f2 m = adj_migrated(a, q, k, y, x + lane);
            const AdjCap c = adj_cap(q.cap[k]);
            const f2 gr = fma2(mul2(v2, z[j]), y.g, y.g);
            const f2 nd = adj_neg_div(mul2(gr, fma2(m, mone, c.c)), c);
            float x0, x1;
            unpack2(mul2(m, fma2(nd, mone, one)), x0, x1);
            const f2 r = pack2(fmaxf(x0, 0.0f), fmaxf(x1, 0.0f));
            nx[k * 32 + lane] = r;
            if (segm) {
                segm[k * 32 + lane] = m;
                segx[k * 32 + lane] = r;
            }
        }
    }
}

// through a year's growth: mu = lambda * dF/dm of a patch, and its terms of
// the derivatives in the growth variability and mean
__device__ __forceinline__ f2 adj_through(const AdjTile& q, const AdjYear& y, float cap, f2 z, f2 m,
                                          f2 l, f2& tv, f2& tm) {
    const f2 one = both2(1.0f), mone = both2(-1.0f);
    const AdjCap c = adj_cap(cap);
    const f2 vz = mul2(both2(q.v), z);
    const f2 gr = fma2(vz, y.g, y.g);
    const f2 room = fma2(m, mone, c.c);                                  // cap - m
    const f2 f = mul2(m, fma2(adj_neg_div(mul2(gr, room), c), mone, one));
    const f2 dm = fma2(adj_neg_div(mul2(gr, fma2(m, both2(-2.0f), c.c)), c), mone, one);
    const f2 dg = neg2(adj_neg_div(mul2(m, room), c));
    // dF = 0 where the growth is cut off at zero
    float f0, f1, a0, a1, b0, b1, v0, v1;
    unpack2(f, f0, f1);
    unpack2(mul2(l, dg), a0, a1);
    unpack2(mul2(l, dm), b0, b1);
    unpack2(vz, v0, v1);
    const f2 lg = pack2(f0 > 0.0f ? a0 : 0.0f, f1 > 0.0f ? a1 : 0.0f);
    tv = mul2(mul2(lg, y.g), z);
    // scalar: ptxas joins a packed multiply and add, which rounds once
    tm = mul2(mul2(lg, pack2(1.0f + v0, 1.0f + v1)), y.gd);
    return pack2(f0 > 0.0f ? b0 : 0.0f, f1 > 0.0f ? b1 : 0.0f);
}

// The sums over a year's patches and pairs run in the order one thread a
// path would take - patches ascending; destinations, then origins - in FP32,
// so that they round alike however the patches are dealt out.  Growth: one
// warp adds a year's terms while the others work on the next rows.
__device__ __forceinline__ void adj_growth_chain(const AdjTile& q, const f2* terms, size_t seg, f2* sums) {
    const int lane = threadIdx.x & 31;
    f2 gv = sums[lane], gm = sums[32 + lane];
#pragma unroll 8
    for (int k = 0; k < q.N; ++k) {
        gv = add2(gv, terms[k * 32 + lane]);
        gm = add2(gm, terms[seg + k * 32 + lane]);
    }
    sums[lane] = gv;
    sums[32 + lane] = gm;
}
// Hazards: a chain over all pairs, a load latency every few of them, but the
// years are independent - a segment's years are summed at once, a warp each
// (a year at a time, by one warp beside the others: a sweep of 4.8 ms where
// this takes 2.0).
__device__ __forceinline__ f2 adj_hazard_chain(const AdjArgs& a, const AdjTile& q, const AdjYear& y,
                                               const f2* mu, const f2* xt) {
    const int lane = threadIdx.x & 31, W = a.C + 1, e1 = q.up[q.N];
    const float* v0 = a.uval + y.c0;
    const float* v1 = a.uval + y.c1;
    f2 acc = 0ull;
#pragma unroll 4
    for (int e = q.up[0]; e < e1; ++e) {
        const int4 u = a.uchain[e];
        const f2 v = mul2(both2(__int_as_float(u.z)), pack2(v0[(size_t)e * W], v1[(size_t)e * W]));
        acc = fma2(mul2(v, mu[u.y + lane]), xt[u.x + lane], acc);
    }
    float s0, s1;
    unpack2(acc, s0, s1);
    if (s0 == s0 && s1 == s1) return acc;
    s0 = s1 = 0.0f;                            // without the zeros, as adj_list_sum
#pragma unroll 1
    for (int e = q.up[0]; e < e1; ++e) {
        const int4 u = a.uchain[e];
        const float x = __int_as_float(u.z), w0 = v0[(size_t)e * W], w1 = v1[(size_t)e * W];
        float m0, m1, x0, x1;
        unpack2(mu[u.y + lane], m0, m1);
        unpack2(xt[u.x + lane], x0, x1);
        if (w0 != 0.0f) s0 = fmaf(x * w0 * m0, x0, s0);
        if (w1 != 0.0f) s1 = fmaf(x * w1 * m1, x1, s1);
    }
    return pack2(s0, s1);
}

// the rows a year wrote become the rows the next one reads
__device__ __forceinline__ void adj_turn(f2*& x, f2*& nx, int n, int two) {
    __syncthreads();
    if (two) {
        f2* t = x;
        x = nx;
        nx = t;
    } else {
        for (int i = threadIdx.x; i < n; i += kAdjThreads) x[i] = nx[i];
        __syncthreads();
    }
}

// forward: end population per path and checkpoints.  `two`: shared memory
// holds both years' rows, else the next year's go through global memory
__device__ __forceinline__ void adj_forward(const AdjArgs& a, AdjTile q, int two, unsigned char* sm) {
    const int tid = threadIdx.x, lane = tid & 31;
    f2* x = reinterpret_cast<f2*>(sm);                         // [N][32]
    f2* nx = two ? x + (size_t)q.N * 32 : a.rows + (size_t)blockIdx.x * a.NP * 32;
    const float* ip = a.init_pops + (size_t)q.s * a.NP;
    for (int i = tid; i < q.N * 32; i += kAdjThreads) x[i] = both2(ip[i >> 5]);
    __syncthreads();
    for (int t = 0; t < a.Y; ++t) {
        const AdjYear y = adj_year(a, q, t);
        if (t % kCk == 0)
            for (int k = tid >> 5; k < q.N; k += kAdjWarps) {
                float* o = a.ckpt + (((size_t)q.s * (a.Y / kCk + 1) + t / kCk) * a.NP + k) * a.P;
                float x0, x1;
                unpack2(x[k * 32 + lane], x0, x1);
                if (q.live0) o[q.p0] = x0;
                if (q.live1) o[q.p1] = x1;
            }
        adj_step(a, q, y, x, nx, nullptr, nullptr);
        adj_turn(x, nx, q.N * 32, two);
    }
    if (tid < 32) {
        double e0 = 0.0, e1 = 0.0;
#pragma unroll 4
        for (int k = 0; k < q.N; ++k) {
            float x0, x1;
            unpack2(x[k * 32 + lane], x0, x1);
            e0 += (double)x0;
            e1 += (double)x1;
        }
        if (q.live0) a.endp[(size_t)q.s * a.P + q.p0] = e0;
        if (q.live1) a.endp[(size_t)q.s * a.P + q.p1] = e1;
    }
}

__global__ void __launch_bounds__(kAdjThreads, 2) k_adj_pop_fwd(AdjArgs a, int two) {
    extern __shared__ __align__(16) unsigned char sm_adj[];
    __shared__ to_bm_tables s_tab;
    to_bm_load(s_tab);
    for (int item = blockIdx.x; item < a.S * adj_tiles(a); item += gridDim.x) {
        __syncthreads();                       // the one before is done with
        adj_forward(a, adj_tile(a, &s_tab, item), two, sm_adj);
    }
}

// backward: reverse sweep over the K-year segments.  The rows other patches
// read are a segment's states while it is recomputed, then mu: a warp turns
// year t's mu into lambda_t of four patches and that at once into their
// year t - 1's mu, so a year takes one barrier either way.  In the reverse
// years warps take groups from a counter, one of them after the growth sums.
__device__ __forceinline__ void adj_backward(const AdjArgs& a, AdjTile q, float w, int two, int ntheta,
                                             unsigned char* sm, int* s_grab) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, W = a.C + 1;
    const int NG = q.N4 / 4;
    const size_t slot = blockIdx.x, seg = (size_t)a.NP * 32;
    f2* gsum = reinterpret_cast<f2*>(sm);                          // [2][32] v_s, mu_s
    float* gh = reinterpret_cast<float*>(gsum + 64);               // [W][64]
    float* gy = gh + (size_t)W * kAdjPaths;                        // [kCk][64] a year's
    f2* x = reinterpret_cast<f2*>(gy + kCk * kAdjPaths);           // [N][32]
    f2* nx = two ? x + (size_t)q.N * 32 : a.rows + slot * seg;     // [N][32]
    f2* lam = a.lam + slot * seg;
    f2* segx = a.segx + slot * kCk * seg;
    f2* segm = a.segm + slot * kCk * seg;      // in the reverse years mu takes a year's place
    f2* terms = a.terms + slot * 4 * seg;                          // [t & 1][v_s, mu_s][NP][32]
    if (tid < 64) gsum[tid] = 0ull;
    for (int i = tid; i < W * kAdjPaths; i += kAdjThreads) gh[i] = 0.0f;
    if (tid < 2) s_grab[tid] = 0;
    for (int i = tid; i < q.N * 32; i += kAdjThreads) lam[i] = both2(w);
    int turn = 0;                                                  // of the counters
    const int nseg = (a.Y + kCk - 1) / kCk;
    for (int sg = nseg - 1; sg >= 0; --sg) {
        const int t0 = sg * kCk, t1 = min(a.Y, t0 + kCk);
        // the segment's states from its checkpoint
        __syncthreads();
        for (int k = warp; k < q.N; k += kAdjWarps) {
            const float* c = a.ckpt + (((size_t)q.s * (a.Y / kCk + 1) + sg) * a.NP + k) * a.P;
            segx[k * 32 + lane] = x[k * 32 + lane] =
                pack2(q.live0 ? c[q.p0] : 0.0f, q.live1 ? c[q.p1] : 0.0f);
        }
        __syncthreads();
        for (int t = t0; t < t1 - 1; ++t) {
            const AdjYear y = adj_year(a, q, t);
            adj_step(a, q, y, x, nx, segm + (size_t)(t - t0) * seg, segx + (size_t)(t + 1 - t0) * seg);
            adj_turn(x, nx, q.N * 32, two);
        }
        // the last year's mu
        AdjYear y = adj_year(a, q, t1 - 1);
        f2* tt = terms + (size_t)((t1 - 1) & 1) * 2 * seg + lane;
        for (int grp = warp; grp < NG; grp += kAdjWarps) {
            f2 z[4];
            adj_normals(a, q, grp, z);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = grp * 4 + j;
                if (k >= q.N) break;
                const f2 m = adj_migrated(a, q, k, y, x + lane);
                nx[k * 32 + lane] = segm[(size_t)(t1 - 1 - t0) * seg + k * 32 + lane] =
                    adj_through(q, y, q.cap[k], z[j], m, lam[k * 32 + lane], tt[k * 32],
                                tt[seg + k * 32]);
            }
        }
        adj_turn(x, nx, q.N * 32, two);
        for (int t = t1 - 1; t >= t0; --t) {
            // lambda_t = M_c^T mu_t, then year t - 1's growth
            const int c0 = y.c0, c1 = y.c1;
            f2* mt = segm + (size_t)(t - 1 - t0) * seg;
            if (warp == 0) adj_growth_chain(q, terms + (size_t)(t & 1) * 2 * seg, seg, gsum);
            if (t > t0) y = adj_year(a, q, t - 1);
            tt = terms + (size_t)((t - 1) & 1) * 2 * seg + lane;
            int* counter = s_grab + (turn & 1);
            for (;;) {
                int grp = 0;
                if (lane == 0) grp = atomicAdd(counter, 1);
                grp = __shfl_sync(0xffffffffu, grp, 0);
                if (grp >= NG) break;
                f2 z[4] = {0ull, 0ull, 0ull, 0ull};
                if (t > t0) adj_normals(a, q, grp, z);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int k = grp * 4 + j;
                    if (k >= q.N) break;
                    const f2 l = adj_list_sum(a.tval, a.tk, W, q.tp[k], q.tp[k + 1], c0, c1, x + lane);
                    if (t > t0)
                        nx[k * 32 + lane] = mt[k * 32 + lane] =
                            adj_through(q, y, q.cap[k], z[j], mt[k * 32 + lane], l, tt[k * 32],
                                        tt[seg + k * 32]);
                    else
                        lam[k * 32 + lane] = l;
                }
            }
            ++turn;
            if (tid == 0) s_grab[turn & 1] = 0;        // last used before the last barrier
            adj_turn(x, nx, q.N * 32, two);
        }
        for (int t = t1 - 1 - warp; t >= t0; t -= kAdjWarps) {
            const AdjYear h = adj_year(a, q, t);
            float h0, h1;
            unpack2(adj_hazard_chain(a, q, h, segm + (size_t)(t - t0) * seg,
                                     segx + (size_t)(t - t0) * seg), h0, h1);
            gy[(t - t0) * kAdjPaths + lane] = h0;
            gy[(t - t0) * kAdjPaths + 32 + lane] = h1;
        }
        __syncthreads();
        if (warp == 0)
            for (int t = t1 - 1; t >= t0; --t) {
                const AdjYear h = adj_year(a, q, t);
                gh[h.c0 * kAdjPaths + lane] += gy[(t - t0) * kAdjPaths + lane];
                gh[h.c1 * kAdjPaths + 32 + lane] += gy[(t - t0) * kAdjPaths + 32 + lane];
            }
    }
    __syncthreads();
    const float* gs = reinterpret_cast<const float*>(gsum);
    for (int i = tid; i < (2 + a.C) * kAdjPaths; i += kAdjThreads) {
        const int what = i / kAdjPaths, j = i - what * kAdjPaths, p = q.p0 - lane + j;
        if (p >= a.P) continue;
        double* gp = a.gpath + (size_t)p * ntheta;
        // species blocks are disjoint, so each species writes its own entries
        if (what < 2) gp[2 * a.U + (1 - what) * a.S + q.s] = (double)gs[what * 64 + (j & 31) * 2 + (j >> 5)];
        else atomicAdd(&gp[2 * a.U + 2 * a.S + what - 2], (double)gh[(what - 2) * kAdjPaths + j]);
    }
}

__global__ void __launch_bounds__(kAdjThreads, 2) k_adj_pop_bwd(AdjArgs a, int two, int ntheta) {
    extern __shared__ __align__(16) unsigned char sm_adj[];
    __shared__ to_bm_tables s_tab;
    __shared__ int s_grab[2];
    to_bm_load(s_tab);
    for (int item = blockIdx.x; item < a.S * adj_tiles(a); item += gridDim.x) {
        const AdjTile q = adj_tile(a, &s_tab, item);
        // the sweep is linear in the species' output weight: a zero weight
        // contributes exactly zero (the per-path gradients start zeroed)
        const float w = a.gout[1 + q.s];
        if (w == 0.0f) continue;
        __syncthreads();                       // the one before is done with
        adj_backward(a, q, w, two, ntheta, sm_adj, s_grab);
    }
}

// mean over paths of column j of a [P][ncol] array (FP64), one CTA per column
__global__ void k_col_mean(int P, int ncol, const double* __restrict__ v, double* out) {
    const int j = blockIdx.x;
    double s = 0.0;
    for (int p = threadIdx.x; p < P; p += blockDim.x) s += v[(size_t)p * ncol + j];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ double w[32];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += w[i];
        out[j] = t / (double)P;
    }
}

size_t adj_fwd_smem(int N, bool two) { return (size_t)(two ? 2 : 1) * N * 32 * 8; }
size_t adj_bwd_smem(int N, int C, bool two) {
    return (size_t)(C + 3 + kCk) * kAdjPaths * 4 + adj_fwd_smem(N, two);
}

}  // namespace

// ---- tape and C ABI ---------------------------------------------------------
struct to_tape_s {
    to_ctx ctx = nullptr;
    AdjArgs a;
    int ntheta = 0, nout = 0, maxN = 0;
    bool two_b = false;                 // the reverse sweep's rows fit in shared memory twice
    char* buf = nullptr;
    double* d_out = nullptr;            // [1 + S] forward outputs
    double* d_grad = nullptr;           // [ntheta] backward result
    double outputs[16];
};

extern "C" {

to_status to_adjoint_forward(to_ctx ctx, const to_adjoint_problem* pr, const double* theta,
                             double* outputs, to_tape* tape_out) {
    if (!ctx || !pr || !pr->rov || !theta || !outputs) return TO_ERR_INVALID;
    const to_rov_problem* rp = pr->rov;
    const int S = rp->n_species, C = rp->n_controls, U = rp->n_uncertainties;
    const int P = rp->n_paths, Y = rp->n_years;
    if (S <= 0 || S > 8 || C <= 0 || C > 8 || U < 0 || U > 8 || P <= 0 || Y <= 0 ||
        rp->n_commodities > 8 || !pr->controls || !pr->crossings || !pr->hazard)
        return TO_ERR_INVALID;
    // every process the profits read exists (as the ROV's entry checks)
    if (rp->n_fuels < 0 || rp->n_commodities < 0 || rp->n_fuels + rp->n_commodities > U ||
        rp->demand_idx >= U)
        return TO_ERR_INVALID;
    for (int f = 0; f < rp->n_fuels; ++f)
        if (rp->fuel_idx[f] < 0 || rp->fuel_idx[f] >= U) return TO_ERR_INVALID;
    const int ntheta = 2 * U + 2 * S + C;
    for (int i = 0; i < ntheta; ++i)
        if (!std::isfinite(theta[i])) return to_set_error(ctx, TO_ERR_NONFINITE, "theta %d", i);
    cudaSetDevice(ctx->device);
    int maxN = 4;
    for (int s = 0; s < S; ++s) {
        const int N = rp->species[s].n_patches;
        if (N <= 0 || N > 512) return to_set_error(ctx, TO_ERR_UNSUPPORTED, "patches %d", N);
        if (N > maxN) maxN = N;
    }
    const int NP = (maxN + 3) & ~3;
    // lists of every species: the pairs with a non-zero value under any
    // control, by destination and then by origin
    std::vector<int> uptr((size_t)S * (NP + 1), 0), tptr((size_t)S * (NP + 1), 0), ul, tk, tsrc;
    std::vector<int4> chain;
    std::vector<float> vv;
    for (int s = 0; s < S; ++s) {
        const to_rov_species& sp = rp->species[s];
        const int N = sp.n_patches;
        int* up = &uptr[(size_t)s * (NP + 1)];
        int* tp = &tptr[(size_t)s * (NP + 1)];
        const size_t e0 = ul.size();
        std::vector<int> cnt(N, 0), dest;
        for (int k = 0; k < N; ++k) {
            up[k] = (int)ul.size();
            for (int l = 0; l < N; ++l) {
                bool any = false;
                for (int c = 0; c < C && !any; ++c) any = sp.mmm[((size_t)c * N + k) * N + l] != 0.0f;
                if (!any) continue;
                ul.push_back(l);
                dest.push_back(k);
                ++cnt[l];
                for (int c = 0; c < C; ++c) vv.push_back(sp.mmm[((size_t)c * N + k) * N + l]);
                vv.push_back(0.0f);
                const float nx = -(float)pr->crossings[s][(size_t)l * N + k];
                int bits;
                memcpy(&bits, &nx, 4);
                chain.push_back(make_int4(l * 32, k * 32, bits, 0));
            }
        }
        for (int k = N; k <= NP; ++k) up[k] = (int)ul.size();
        // transposed: by origin, destinations ascending
        int at = (int)e0;
        for (int l = 0; l < N; ++l) { tp[l] = at; at += cnt[l]; }
        for (int l = N; l <= NP; ++l) tp[l] = at;
        tk.resize(ul.size());
        tsrc.resize(ul.size());
        std::vector<int> next(tp, tp + N);
        for (size_t e = e0; e < ul.size(); ++e) {
            const int q = next[ul[e]]++;
            tk[q] = dest[e - e0];
            tsrc[q] = (int)e;
        }
    }
    const size_t nE = ul.size() > 0 ? ul.size() : 1;
    const int tiles = (P + kAdjPaths - 1) / kAdjPaths;
    // two CTAs an SM at most are at work (their registers)
    const int sms = ctx->sm_count > 0 ? ctx->sm_count : TO_SM_TARGET;
    const int slots = S * tiles < 2 * sms ? S * tiles : 2 * sms;
    const size_t rowb = (size_t)slots * NP * 32 * 8;           // one row of each
    const bool two_f = adj_fwd_smem(maxN, true) + kAdjStatic <= ctx->smem_optin;
    const bool two_b = adj_bwd_smem(maxN, C, true) + kAdjStatic <= ctx->smem_optin;
    std::vector<int> np(S);
    std::vector<float> prm((size_t)S * 8), ip((size_t)S * NP, 0.0f), cpv((size_t)S * NP, 1.0f);
    for (int s = 0; s < S; ++s) {
        const to_rov_species& sp = rp->species[s];
        np[s] = sp.n_patches;
        for (int q = 0; q < 8; ++q) prm[(size_t)s * 8 + q] = sp.params[q];
        for (int k = 0; k < sp.n_patches; ++k) { ip[(size_t)s * NP + k] = sp.init_pops[k]; cpv[(size_t)s * NP + k] = sp.caps[k]; }
    }
    std::vector<float> th(ntheta), bh(C);
    for (int i = 0; i < ntheta; ++i) th[i] = (float)theta[i];
    for (int c = 0; c < C; ++c) bh[c] = (float)pr->hazard[c];
    // one allocation holds inputs and tape
    size_t bytes = 0;
    auto acc = [&](size_t b) { bytes += to_align256(b); };
    acc(ntheta * 4); acc((size_t)U * 24 + 4); acc(C * 4); acc(64); acc(64); acc(64); acc(64);
    acc((size_t)Y * P * 4); acc(S * 4); acc((size_t)S * 32); acc((size_t)S * NP * 4);
    acc((size_t)S * NP * 4); acc(uptr.size() * 4); acc(tptr.size() * 4);
    for (int q = 0; q < 3; ++q) acc(nE * 4);
    acc(nE * 16);
    for (int q = 0; q < 3; ++q) acc(nE * (C + 1) * 4);
    acc(C * 4);
    acc((size_t)S * (Y / kCk + 1) * NP * P * 4); acc(rowb * kCk); acc(rowb * kCk);
    acc(rowb); acc(rowb * 4);
    if (!two_f || !two_b) acc(rowb);
    acc((size_t)S * Y * P * 4); acc((size_t)S * Y * P * 4); acc((size_t)P * 8);
    acc((size_t)S * P * 8); acc((size_t)P * ntheta * 8); acc(64); acc(256); acc(ntheta * 8);
    to_tape t = new to_tape_s();
    t->ctx = ctx;
    cudaError_t e = cudaMalloc(&t->buf, bytes);
    if (e != cudaSuccess) { delete t; return to_check_cuda(ctx, e, "adjoint tape"); }
    char* q = t->buf;
    auto take = [&](size_t b) { char* r = q; q += to_align256(b); return r; };
    AdjArgs& a = t->a;
    memset(&a, 0, sizeof(a));
    a.P = P; a.Y = Y; a.S = S; a.C = C; a.U = U; a.NP = NP; a.nF = rp->n_fuels;
    a.Cm = rp->n_commodities; a.demand_idx = rp->demand_idx; a.road = rp->road;
    a.dt = rp->dt; a.rrr = rp->rrr; a.unit_cost = rp->unit_cost; a.unit_revenue = rp->unit_revenue;
    a.seed = rp->seed;
    float* d_th = (float*)take(ntheta * 4);
    float* d_unc = (float*)take((size_t)U * 24 + 4);
    float* d_fl = (float*)take(C * 4);
    float* d_fc = (float*)take(64); int* d_fi = (int*)take(64);
    float* d_oc = (float*)take(64); float* d_os = (float*)take(64);
    int* d_ctl = (int*)take((size_t)Y * P * 4);
    int* d_np = (int*)take(S * 4);
    float* d_prm = (float*)take((size_t)S * 32);
    float* d_ip = (float*)take((size_t)S * NP * 4);
    float* d_cp = (float*)take((size_t)S * NP * 4);
    int* d_up = (int*)take(uptr.size() * 4);
    int* d_tp = (int*)take(tptr.size() * 4);
    int* d_ul = (int*)take(nE * 4); int* d_tk = (int*)take(nE * 4); int* d_ts = (int*)take(nE * 4);
    int4* d_ch = (int4*)take(nE * 16);
    float* d_v = (float*)take(nE * (C + 1) * 4);
    a.uval = (float*)take(nE * (C + 1) * 4); a.tval = (float*)take(nE * (C + 1) * 4);
    float* d_bh = (float*)take(C * 4);
    a.ckpt = (float*)take((size_t)S * (Y / kCk + 1) * NP * P * 4);
    a.slots = slots;
    a.segx = (f2*)take(rowb * kCk);
    a.segm = (f2*)take(rowb * kCk);
    a.lam = (f2*)take(rowb);
    a.terms = (f2*)take(rowb * 4);
    a.rows = (!two_f || !two_b) ? (f2*)take(rowb) : nullptr;
    a.gtab = (float*)take((size_t)S * Y * P * 4);
    a.gdot = (float*)take((size_t)S * Y * P * 4);
    a.pv = (double*)take((size_t)P * 8);
    a.endp = (double*)take((size_t)S * P * 8);
    a.gpath = (double*)take((size_t)P * ntheta * 8);
    float* d_gout = (float*)take(64);
    double* d_out = (double*)take(256);
    t->d_out = d_out;
    t->d_grad = (double*)take(ntheta * 8);
    a.theta = d_th; a.uncert = d_unc; a.flows = d_fl; a.fuel_costs = d_fc; a.fuel_idx = d_fi;
    a.ore_content = d_oc; a.ore_sd = d_os; a.controls = d_ctl; a.n_patches = d_np;
    a.params = d_prm; a.init_pops = d_ip; a.caps = d_cp; a.uptr = d_up; a.tptr = d_tp;
    a.ul = d_ul; a.tk = d_tk; a.tsrc = d_ts; a.base_v = d_v; a.uchain = d_ch; a.base_h = d_bh;
    a.E = (int)ul.size(); a.gout = d_gout; a.rk = to_make_round_keys(a.seed);
    auto h2d = [&](void* d, const void* h, size_t b) {
        return b ? cudaMemcpyAsync(d, h, b, cudaMemcpyHostToDevice, ctx->stream) : cudaSuccess;
    };
    cudaError_t ce = cudaSuccess;
    auto chk = [&](cudaError_t x) { if (ce == cudaSuccess) ce = x; };
    chk(h2d(d_th, th.data(), ntheta * 4));
    chk(h2d(d_unc, rp->uncert, (size_t)U * 24));
    chk(h2d(d_fl, rp->flows, C * 4));
    chk(h2d(d_fc, rp->fuel_costs, (size_t)rp->n_fuels * 4));
    chk(h2d(d_fi, rp->fuel_idx, (size_t)rp->n_fuels * 4));
    chk(h2d(d_oc, rp->ore_content, (size_t)rp->n_commodities * 4));
    chk(h2d(d_os, rp->ore_sd, (size_t)rp->n_commodities * 4));
    chk(h2d(d_ctl, pr->controls, (size_t)Y * P * 4));
    chk(h2d(d_np, np.data(), S * 4));
    chk(h2d(d_prm, prm.data(), prm.size() * 4));
    chk(h2d(d_ip, ip.data(), ip.size() * 4));
    chk(h2d(d_cp, cpv.data(), cpv.size() * 4));
    chk(h2d(d_up, uptr.data(), uptr.size() * 4));
    chk(h2d(d_tp, tptr.data(), tptr.size() * 4));
    chk(h2d(d_ul, ul.data(), ul.size() * 4));
    chk(h2d(d_tk, tk.data(), tk.size() * 4));
    chk(h2d(d_ts, tsrc.data(), tsrc.size() * 4));
    chk(h2d(d_v, vv.data(), vv.size() * 4));
    chk(h2d(d_ch, chain.data(), chain.size() * 16));
    chk(h2d(d_bh, bh.data(), C * 4));
    if (ce != cudaSuccess) { cudaFree(t->buf); delete t; return to_check_cuda(ctx, ce, "adjoint inputs"); }
    t->ntheta = ntheta; t->nout = 1 + S; t->maxN = maxN; t->two_b = two_b;
    // forward
    k_adj_pv<<<(P + 127) / 128, 128, 0, ctx->stream>>>(a);
    const size_t smf = adj_fwd_smem(maxN, two_f);
    cudaFuncSetAttribute(k_adj_pop_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(ctx->smem_optin - kAdjStatic));
    if (a.E > 0) k_adj_values<<<(a.E + 255) / 256, 256, 0, ctx->stream>>>(a);
    k_adj_growth<<<dim3((P + 127) / 128, S), 128, 0, ctx->stream>>>(a);
    to_prof_begin(ctx, "adjoint_forward");
    k_adj_pop_fwd<<<two_f ? S * tiles : slots, kAdjThreads, smf, ctx->stream>>>(a, two_f ? 1 : 0);
    to_prof_end(ctx);
    k_col_mean<<<1, 256, 0, ctx->stream>>>(P, 1, a.pv, d_out);
    for (int s = 0; s < S; ++s)
        k_col_mean<<<1, 256, 0, ctx->stream>>>(P, 1, a.endp + (size_t)s * P, d_out + 1 + s);
    ctx->launches += 5 + S;
    ce = cudaGetLastError();
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(t->outputs, d_out, (size_t)(1 + S) * 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(ctx->stream);
    if (ce != cudaSuccess) { cudaFree(t->buf); delete t; return to_check_cuda(ctx, ce, "adjoint forward"); }
    for (int i = 0; i < 1 + S; ++i) outputs[i] = t->outputs[i];
    if (tape_out) *tape_out = t;
    else { cudaFree(t->buf); delete t; }
    return TO_OK;
}

to_status to_adjoint_backward(to_ctx ctx, to_tape t, const double* grad_outputs,
                              double* grad_theta) {
    if (!ctx || !t || !grad_outputs || !grad_theta || t->ctx != ctx) return TO_ERR_INVALID;
    cudaSetDevice(ctx->device);
    AdjArgs& a = t->a;
    const int S = a.S, P = a.P, ntheta = t->ntheta;
    float go[16];
    for (int i = 0; i < 1 + S; ++i) go[i] = (float)grad_outputs[i];
    TO_CUDA(ctx, cudaMemcpyAsync(const_cast<float*>(a.gout), go, (size_t)(1 + S) * 4,
                                 cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemsetAsync(a.gpath, 0, (size_t)P * ntheta * 8, ctx->stream));
    if (grad_outputs[0] != 0.0) {           // the PV part is linear in its weight too
        k_adj_pv_grad<<<(P + 127) / 128, 128, 0, ctx->stream>>>(a, ntheta);
        TO_LAUNCHED(ctx);
    }
    const size_t smb = adj_bwd_smem(t->maxN, a.C, t->two_b);
    TO_CUDA(ctx, cudaFuncSetAttribute(k_adj_pop_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(ctx->smem_optin - kAdjStatic)));
    to_prof_begin(ctx, "adjoint_backward");
    k_adj_pop_bwd<<<a.slots, kAdjThreads, smb, ctx->stream>>>(a, t->two_b ? 1 : 0, ntheta);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    std::vector<double> g(ntheta);
    double* d_g = t->d_grad;
    k_col_mean<<<ntheta, 256, 0, ctx->stream>>>(P, ntheta, a.gpath, d_g);
    TO_LAUNCHED(ctx);
    TO_CUDA(ctx, cudaMemcpyAsync(g.data(), d_g, (size_t)ntheta * 8, cudaMemcpyDeviceToHost,
                                 ctx->stream));
    TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int i = 0; i < ntheta; ++i) grad_theta[i] = g[i];
    return TO_OK;
}

to_status to_tape_destroy(to_tape t) {
    if (!t) return TO_OK;
    if (t->ctx) {
        cudaSetDevice(t->ctx->device);
        cudaStreamSynchronize(t->ctx->stream);
    }
    cudaFree(t->buf);
    delete t;
    return TO_OK;
}

}  // extern "C"
