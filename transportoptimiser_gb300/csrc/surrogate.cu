// surrogate.cu - local-linear surrogate builders used by the GA fitness.
//
// Reference: SimulateGPU::buildSurrogateMTECUDA (include/gpuCode/
// SimulateGPU.cu:5533-5692: 1-D surrogate of the end population against the
// initial animals-at-risk) and SimulateGPU::buildSurrogateROVCUDA
// (SimulateGPU.cu:5694-5917: d-D surrogate of the ROV value against the
// IARs and unit use), both built from a k-nearest-neighbour local linear
// regression on a dim_res^d grid (createQueryPoints, knn, multiLocLinReg,
// rovCorrection).  The reference copies the samples and the grid between
// host and device around each step; here one preparation kernel (min / max,
// normalisation, grid) feeds the warp-per-query kNN and a thread-per-grid-
// point regression, all on the device.
#include <cmath>
#include <cstring>
#include <vector>

#include "to_internal.cuh"
#include "to_lsm_math.h"
#include "to_rov.cuh"

namespace {

struct SurrArgs {
    int n, d, R, Q, k, normalize, sem, clip0;
    const float* raw;     // [d][n]
    const float* y;       // [n_y][n] the responses
    float* pn;            // [d][n] points the kNN sees
    float* qn;            // [d][Q] queries the kNN sees
    float* xq;            // [d][Q] regression centres
    float* dist;          // [k][Q]
    int* ind;             // [k][Q]
    float* out;           // [n_y][R*d + Q]
    int n_y;
};

// Every CTA finds the ranges for itself (the samples are a few KB in L2) and
// then takes its share of the points and queries: 1,000 samples, 16^3
// queries, 13.5 us by one CTA, 7.0 us by one for each 1,024 queries.
__global__ void __launch_bounds__(1024) k_surr_prepare(SurrArgs a) {
    const int at = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    __shared__ float s_lo[TO_LSM_MAXD], s_hi[TO_LSM_MAXD];
    __shared__ float w_lo[32], w_hi[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int j = 0; j < a.d; ++j) {
        float lo = INFINITY, hi = -INFINITY;
        for (int m = threadIdx.x; m < a.n; m += blockDim.x) {
            float v = a.raw[(size_t)j * a.n + m];
            lo = fminf(lo, v);
            hi = fmaxf(hi, v);
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) { w_lo[warp] = lo; w_hi[warp] = hi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            float l = w_lo[0], h = w_hi[0];
            for (int w = 1; w < nw; ++w) { l = fminf(l, w_lo[w]); h = fmaxf(h, w_hi[w]); }
            s_lo[j] = l;
            s_hi[j] = h;
        }
        __syncthreads();
    }
    for (int q = at; q < a.n * a.d; q += step) {
        int j = q / a.n;
        float v = a.raw[q];
        a.pn[q] = a.normalize ? to_lsm_normalise(v, s_lo[j], s_hi[j], 0, 1.0f) : v;
    }
    for (int q = at; q < a.Q; q += step) {
        int rem = q;
        int div = a.Q / a.R;
        for (int j = 0; j < a.d; ++j) {
            int di = rem / div;
            rem -= di * div;
            div /= a.R;
            float raw = to_lsm_query_axis(di, s_lo[j], s_hi[j], a.R);
            if (rem == 0)
                for (int v = 0; v < a.n_y; ++v) a.out[(size_t)v * (a.R * a.d + a.Q) + j * a.R + di] = raw;
            float nv = a.normalize ? to_lsm_normalise(raw, s_lo[j], s_hi[j], 0, 1.0f) : raw;
            a.qn[(size_t)j * a.Q + q] = nv;
            a.xq[(size_t)j * a.Q + q] = a.normalize ? (a.sem == 0 ? to_lsm_unit_axis(di, a.R) : nv)
                                                    : raw;
        }
    }
}

// A thread per grid query, grid row v on response v.  With the dimension
// known the sums stay in registers (D = 0: any dimension), and CTAs of 64
// spread a surrogate's few thousand queries over the SMs: 16^3 queries, 35
// neighbours, 2 x 56 us in two launches of 128-thread CTAs before, 23 us.
template <int D>
__global__ void __launch_bounds__(64) k_surr_regress(SurrArgs a) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.Q) return;
    const int d = D ? D : a.d, v = blockIdx.y;
    const float* y = a.y + (size_t)v * a.n;
    float* yout = a.out + (size_t)v * (a.R * d + a.Q) + (size_t)a.R * d;
    if (a.n < 3 || a.k <= 0) { yout[q] = 0.0f; return; }
    const bool raw = a.sem == 0 || !a.normalize;
    const float* px = raw ? a.raw : a.pn;      // coordinate j of sample i at i si + j sj
    const size_t si = raw ? d : 1, sj = raw ? 1 : a.n;
    float xq[D ? D : TO_LSM_MAXD];
    for (int j = 0; j < d; ++j) xq[j] = a.xq[(size_t)j * a.Q + q];
    float acc[TO_LSM_ACC];
    to_lsm_acc_init(d, acc);
    const float h = a.dist[(size_t)(a.k - 1) * a.Q + q];
#pragma unroll 4
    for (int kk = 0; kk < a.k; ++kk) {
        const float dd = a.dist[(size_t)kk * a.Q + q];
        const int i = a.ind[(size_t)kk * a.Q + q] - 1;
        float xv[D ? D : TO_LSM_MAXD];
        for (int j = 0; j < d; ++j) xv[j] = px[i * si + j * sj];
        to_lsm_acc_add(d, acc, to_lsm_weight(dd, h), y[i], xv, xq);
    }
    float r = to_lsm_solve_intercept(d, acc);
    if (v == 0 && a.clip0 && r > 0.0f) r = 0.0f;   // rovCorrection (SimulateGPU.cu:3055-3073)
    yout[q] = r;
}

// k rules of the two builders (SimulateGPU.cu:5545-5554, 5711-5722), never
// more than the number of samples
int k_mte(int n) {
    int k;
    if (n < 50) k = 5;
    else if (n < 100) k = 7;
    else if (n < 500) k = (int)std::ceil(0.02 * (n - 100) + 7);
    else k = (int)std::ceil(std::log((double)n) + 8);
    return k < n ? k : n;
}
int k_rov(int n) {
    int k;
    if (n < 50) k = 5;
    else if (n < 100) k = (int)(5 + 5 * std::ceil((double)((n - 50) / 50)));
    else if (n < 500) k = (int)std::ceil(10 + 15 * std::ceil((double)((n - 100) / 400)));
    else k = (int)(25 + std::ceil((n - 500) * 0.02));
    return k < n ? k : n;
}

to_status build(to_ctx ctx, int n, int d, const double* pred, const double* const* ys,
                int n_y, int clip0, int R, int k, int normalize, int sem,
                double* const* outs) {
    long Ql = 1;
    for (int j = 0; j < d; ++j) Ql *= R;
    if (Ql > (1 << 22) || d > TO_LSM_MAXD)
        return to_set_error(ctx, TO_ERR_UNSUPPORTED, "grid %d^%d", R, d);
    const int Q = (int)Ql;
    const int kk = k > 0 ? k : 1;
    // predictors and responses, one copy to the device
    const size_t nx = (size_t)d * n, one = (size_t)R * d + Q;
    std::vector<float> in(nx + (size_t)n_y * n);
    for (size_t i = 0; i < nx; ++i) {
        if (!std::isfinite(pred[i])) return to_set_error(ctx, TO_ERR_NONFINITE, "predictor %zu", i);
        in[i] = (float)pred[i];
    }
    for (int v = 0; v < n_y; ++v)
        for (int i = 0; i < n; ++i) {
            if (!std::isfinite(ys[v][i])) return to_set_error(ctx, TO_ERR_NONFINITE, "value %d", i);
            in[nx + (size_t)v * n + i] = (float)ys[v][i];
        }
    size_t bytes = to_align256(in.size() * 4) + to_align256(nx * 4) +
                   2 * to_align256((size_t)d * Q * 4) + 2 * to_align256((size_t)kk * Q * 4) +
                   to_align256(n_y * one * 4);
    TO_TRY(to_arena_reserve(ctx, bytes + 4096));
    SurrArgs a;
    memset(&a, 0, sizeof(a));
    a.n = n; a.d = d; a.R = R; a.Q = Q; a.k = k; a.normalize = normalize; a.sem = sem;
    a.n_y = n_y; a.clip0 = clip0;
    float* d_in = to_arena_take<float>(ctx, in.size());
    a.raw = d_in; a.y = d_in + nx;
    a.pn = to_arena_take<float>(ctx, nx);
    a.qn = to_arena_take<float>(ctx, (size_t)d * Q);
    a.xq = to_arena_take<float>(ctx, (size_t)d * Q);
    a.dist = to_arena_take<float>(ctx, (size_t)kk * Q);
    a.ind = to_arena_take<int>(ctx, (size_t)kk * Q);
    a.out = to_arena_take<float>(ctx, n_y * one);
    TO_CUDA(ctx, cudaMemcpyAsync(d_in, in.data(), in.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
    const int ctas = (Q + 1023) / 1024;
    k_surr_prepare<<<ctas < ctx->sm_count ? ctas : ctx->sm_count, 1024, 0, ctx->stream>>>(a);
    TO_LAUNCHED(ctx);
    if (n >= 3 && k > 0) TO_TRY(to_k::knn(ctx, a.pn, n, a.qn, Q, d, k, a.dist, a.ind));
    const auto regress = d == 1 ? k_surr_regress<1> : d == 2 ? k_surr_regress<2>
                       : d == 3 ? k_surr_regress<3> : d == 4 ? k_surr_regress<4>
                                                             : k_surr_regress<0>;
    to_prof_begin(ctx, "surrogate_regress");
    regress<<<dim3((Q + 63) / 64, n_y), 64, 0, ctx->stream>>>(a);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    std::vector<float> of(n_y * one);
    TO_CUDA(ctx, cudaMemcpyAsync(of.data(), a.out, of.size() * 4, cudaMemcpyDeviceToHost, ctx->stream));
    TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int v = 0; v < n_y; ++v)
        if (outs[v])
            for (size_t i = 0; i < one; ++i) outs[v][i] = (double)of[v * one + i];
    return TO_OK;
}

}  // namespace

extern "C" {

to_status to_build_surrogate_mte(to_ctx ctx, int samples, const double* iars,
                                 const double* pops_mean, const double* pops_sd, int dim_res,
                                 double* out_mean, double* out_sd) {
    if (!ctx || samples <= 0 || !iars || !pops_mean || dim_res < 2) return TO_ERR_INVALID;
    cudaSetDevice(ctx->device);
    const double* ys[2] = {pops_mean, pops_sd};
    double* outs[2] = {out_mean, out_sd};
    return build(ctx, samples, 1, iars, ys, pops_sd ? 2 : 1, 0, dim_res, k_mte(samples),
                 0, 0, outs);
}

to_status to_build_surrogate_rov(to_ctx ctx, int samples, int n_dims, const double* predictors,
                                 const double* values, const double* values_sd, int dim_res,
                                 int sem, double* out_mean, double* out_sd) {
    if (!ctx || samples <= 0 || n_dims <= 0 || !predictors || !values || dim_res < 2)
        return TO_ERR_INVALID;
    cudaSetDevice(ctx->device);
    const double* ys[2] = {values, values_sd};
    double* outs[2] = {out_mean, out_sd};
    return build(ctx, samples, n_dims, predictors, ys, values_sd ? 2 : 1, 1, dim_res,
                 k_rov(samples), 1, sem, outs);
}

}  // extern "C"
