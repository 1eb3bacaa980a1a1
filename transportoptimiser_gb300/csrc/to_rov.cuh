// to_rov.cuh - argument block of the ROV kernels and the kNN / regression
// launchers shared with the surrogate builders.
#pragma once
#include "to_f2.cuh"
#include "to_internal.cuh"
#include "to_lsm_math.h"

#define TO_ROV_MAXC 8
#define TO_KNN_KMAX 256
#define TO_KNN_GCELLS 4096

// uniform cell grid over one control's normalised regression points:
// cell_j(x) = clamp(floor((x - lo_j) * inv_j), 0, G_j - 1), dimension 0
// fastest; ok = 0 when a coordinate is not finite (full scan instead)
struct to_knn_grid {
    float lo[TO_LSM_MAXD], hi[TO_LSM_MAXD], inv[TO_LSM_MAXD], w[TO_LSM_MAXD];
    int G[TO_LSM_MAXD];
    int ok;
    float T0;                 // first squared-distance threshold of a query
};

// A batch of nr roads with the same dimensions: path arrays are road-major
// ([..][PT], road r's paths at r*P .. r*P+P-1) and the regressions are
// grouped by (road, control), group g = r*C + c.
struct to_rov_args {
    int P, Y, S, C, U, R, Q;          // paths per road, years, species, controls, processes, dimRes, R^d
    int nr, PT, G;                    // roads, paths of all roads (nr*P), groups (nr*C)
    const int* road_ids;              // [nr] road id of each road (random streams)
    int nF, Cm, demand_idx, sem, road;
    float dt, rrr, unit_cost, unit_revenue, scaling;
    uint64_t seed;
    to_round_keys rk;                 // of the seed (rov_run)
    int ctas;                         // resident CTAs of the paired forward pass
    int* fwd_next;                    // its work counter
    f2* fwd_part;                     // [ctas][2][C][np / 4][32] its per-group sums
    f2* fwd_far;                      // [ctas][np][32] next populations of wide models
    int np, ne;                       // stride / effective width of patch arrays
    int tile_paths, l_chunk;          // forward tile (launcher)
    // inputs (device)
    const int* n_patches;             // [nr][S]
    const float* params;              // [S*8]
    const float* init_pops;           // [nr][S][np]
    const float* caps;                // [nr][S][np] (padding 1)
    const float* mmm;                 // [nr][S][C][np][np] destination-major
    const float* flows;               // [C]
    const float* uncert;              // [U*6]
    const float* fuel_costs;          // [nF]
    const int* fuel_idx;              // [nF]
    const float* ore_content;         // [Cm]
    const float* ore_sd;              // [Cm]
    // path state (device)
    int* controls;                    // [Y][PT]
    float* uRes;                      // [U][Y+1][PT]
    float* totalPops;                 // [S][Y+1][PT]
    float* aars;                      // [S][C][Y][PT]
    // regression scratch (device).  What a year's regressions are fitted on -
    // the states, their ranges and the list of grid queries - does not depend
    // on the values of later years, so it is prepared for up to `slots` years
    // at a time; slot = t - slot0.  Per slot, per group g = r*C + c:
    int slots, slot0;
    int sel0, sel_slots;              // first slot with selected neighbours, how many fit
    float* xraw;                      // [slots][G][d][P] compacted raw states (sem 0 only, else xn)
    float* xn;                        // [slots][G][d][P] normalised
    int* pidx;                        // [slots][G][P] path of the batch behind each point
    int* npts;                        // [slots][G]
    int* kc;                          // [slots][G]
    float* qax;                       // [slots][nr][d][R] normalised grid axes of the year
    int* qlist;                       // [slots][G][Q] grid queries to fit, ascending (touched mode)
    int* gcount;                      // [slots][G] how many
    int2* tiles;                      // [slots][G * ceil(Q / TO_ROV_TILE)] {group, first place in its list}
    int* ntiles;                      // [slots] tiles; [slots] next tile to work on
    unsigned short* nbr;              // [sel_slots][tiles][kmax][TO_ROV_TILE] neighbours, ascending
    float* kthv;                      // [sel_slots][tiles][TO_ROV_TILE] k-th squared distances
    unsigned* bmap;                   // [slots][nr][C][ceil(Q / 32)] query marks too many for shared memory
    float* profS;                     // [Y][PT] unit profit of the regression states
    int k_mult;                       // k = k_mult (ln n + 1): 10 ALGO4, 3 ALGO6
    int algo;                         // 4 or 6
    float* popsY;                     // ALGO6: [Y][S][ne][P] patch populations, start of year
    float* gmY;                       // ALGO6: [Y][S][P] mean growth rate of the year
    int kmax;
    // above TO_ROV_SCAN_PATHS paths a road (the cell-grid search, knn.cu)
    float* yv;                        // [G][P] values of the year after
    float* gsx;                       // [G][d][P] points in cell order
    int* gsi;                         // [G][P] their original indices
    int* gcell;                       // [G][TO_KNN_GCELLS + 1] cell starts
    to_knn_grid* ggrid;               // [G]
    float* kth;                       // [G][Q] k-th squared distance, year before
    double* knn_acc;                  // [G][Q][(d+1)(d+4)/2] normal-equation sums per listed query
    // touched-query mode (corrected semantics, ALGO4, surfaces not
    // returned): a year's regressions are fitted only at the grid queries
    // some path's interpolation reads; the others are never read
    int touched;
    unsigned* qroad;                  // [nr] queries fitted per road over the years (may be null)
    // 1: reg holds only the prepared years' blocks, by slot (the regressions of
    // year t are written and read within year t; nothing returns them)
    int reg_by_slot;
    int* flags;                       // device error word (plan checks), may be null
    // outputs (device)
    float* reg;                       // [Y or slots][G][R*d + 2Q]
    float* condExp;                   // [Y][PT]
    int* optCont;                     // [Y][PT]
    float* unitProfits;               // [Y][PT]
    float* adjPops;                   // [Y][S][PT], or null
    double* stats;                    // [nr][5]: value, control, SD, SE, n
};

// regression block of (year t, group g): axis values [R*d], then the Q
// grid values, then Q standard deviations
__host__ __device__ __forceinline__ float* to_rov_reg_block(const to_rov_args& a, int t, size_t g) {
    const size_t blk = (size_t)a.R * (a.S + 1) + 2 * (size_t)a.Q;
    return a.reg + ((size_t)(a.reg_by_slot ? t - a.slot0 : t) * a.G + g) * blk;
}

// grid query q of the current year: normalised coordinates (for kNN) and
// the coordinates the regression centres on (createQueryPoints + host
// normalisation; sem 0 centres on the unit grid, SimulateGPU.cu:2964-2966)
// grid queries of one group that a CTA fits at a time
#define TO_ROV_TILE 128
// paths a road up to which a query scans every point of its group
#define TO_ROV_SCAN_PATHS 32768

template <int D>
__device__ __forceinline__ void to_rov_query(const to_rov_args& a, int slot, int road, int q,
                                             float* qn, float* xq) {
    const int R = a.R;
    const float* ax = a.qax + ((size_t)slot * a.nr + road) * D * R;
    const bool pow2 = (R & (R - 1)) == 0;
    const int lr = pow2 ? __ffs(R) - 1 : 0;           // log2 R
    int rem = q;
    int div = a.Q / R;
#pragma unroll
    for (int j = 0; j < D; ++j) {
        int di;
        if (pow2) {
            // q's base-R digit of dimension j (dimension 0 most significant)
            di = (q >> (lr * (D - 1 - j))) & (R - 1);
        } else {
            di = rem / div;
            rem -= di * div;
            div /= R;
        }
        // the year's normalised axis values, computed once per road (k_lsm_prepare)
        const float nv = ax[j * R + di];
        qn[j] = nv;
        xq[j] = (a.sem == 0) ? to_lsm_unit_axis(di, R) : nv;
    }
}

struct to_csc;
namespace to_k {
// csc: the packed migration matrices for the sparse forward pass, or null
to_status rov_run(to_ctx ctx, to_rov_args a, const to_csc* csc);
// bytes of regression scratch for a.slots years, and its pointers carved from
// `base` (null: only the size)
size_t rov_scratch(to_rov_args& a, int max_roads, char* base);
// sets the years to prepare and to select neighbours for at a time
void rov_plan(to_rov_args& a, int max_roads);
// the k nearest points of every listed grid query of `years` prepared years,
// from slot a.sel0; then the local linear regressions of one of them (ahead:
// not the kernel after a selection, to_rov_years.h)
size_t knn_select_bytes(const to_rov_args& a, int max_roads);
to_status knn_rov_select(to_ctx ctx, const to_rov_args& a, int years);
to_status knn_rov_fit(to_ctx ctx, const to_rov_args& a, int t, bool ahead);
// both for year t by the cell-grid search (groups of very many points)
to_status knn_rov_grid(to_ctx ctx, const to_rov_args& a, int t);
// generic kNN: ref dim-major [dim][n], query dim-major [dim][Q]
to_status knn(to_ctx ctx, const float* ref, int n, const float* query, int Q,
              int dim, int k, float* dist, int* ind);
}
