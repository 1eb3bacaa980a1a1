// mlp.cu - learned surrogate of the road-evaluation outputs: an MLP
// 16 -> 128 -> 128 -> 3 (ReLU), trained and evaluated with this library's
// own kernels.  The reference has no learned surrogate (its GA fitness uses
// the local-linear grid surrogates, SimulateGPU.cu:5533-5917); this is the
// learned alternative used for GA screening, with the plain Monte Carlo as
// the fallback and the measure of its error.
//
// A CTA of 16 warps owns a tile of 128 rows (TMEM lane = row, a warp a
// quarter of its 32 rows' columns) and runs the whole forward and, for
// training, the whole backward pass on it:
//   F1  H1 = X W1^T            tcgen05 kind::f16, M=128 N=128 K=16
//   F2  H2 = H1 W2^T           M=128 N=128 K=128
//   L3  Y = H2 W3^T + b3       SIMT (3 outputs)
//   B2  dH1 = dH2 W2           M=128 (rows) N=128 K=128
//   G2  dW2 = dH2^T H1         M=128 (units) N=128 K=128 (rows)
//   G1  dW1 = dH1^T X          M=128 N=16 K=128
// Operands are BF16 in shared memory (K-major core-matrix tiles written by
// the threads; where a GEMM contracts over rows, a tile's core matrices are
// transposed by ldmatrix / stmatrix), accumulators FP32 in TMEM.  Rounding
// points (every value that feeds an MMA is rounded to BF16 once; biases,
// ReLU, layer 3 and all reductions in FP32) are restated by the oracle.
// Each tile writes its gradient partial; the partials are summed in tile
// order (deterministic) and Adam is applied to the FP32 master parameters.
//
// Training is a chain of small steps (512 rows are four tiles), bound by the
// latency of what follows what within a step: the FP32 sums over 128 units or
// rows keep their order, so that a parameter's trajectory does not depend on
// the thread count, and are a thread each; an epoch is one launch whose CTAs
// meet twice a step.  20,000 rows, batches of 512, four epochs: 10.2 -> 4.2 ms,
// 65 -> 25 us a step (three launches a step and four warps a tile before).
#include <cuda_bf16.h>

#include <cmath>
#include <vector>

#include "to_internal.cuh"
#include "to_tc.cuh"

namespace {

constexpr int IN = TO_MLP_IN, HID = TO_MLP_HID, OUT = TO_MLP_OUT;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + HID * IN, OFF_W2 = OFF_B1 + HID,
              OFF_B2 = OFF_W2 + HID * HID, OFF_W3 = OFF_B2 + HID, OFF_B3 = OFF_W3 + OUT * HID,
              NPARAM = OFF_B3 + OUT;
static_assert(NPARAM == TO_MLP_NPARAM, "parameter layout");
constexpr int PSTRIDE = (NPARAM + 3) & ~3;           // per-tile partial stride (16-byte rows)

// shared memory map (bytes)
constexpr int KB_IN = IN * 2, KB_HID = HID * 2;      // K bytes per row of the bf16 tiles
constexpr int S_X = 0;                               // X   [128 rows][16]
constexpr int S_W1 = S_X + 128 * KB_IN;              // W1  [128 units][16]
constexpr int S_XT = S_W1 + 128 * KB_IN;             // X^T [16][128 rows]
constexpr int S_A = S_XT + IN * KB_HID;              // H1 [row][unit] -> dH2 -> dH1
constexpr int S_B = S_A + 128 * KB_HID;              // W2 [out][in]
constexpr int S_W2T = S_B + 128 * KB_HID;            // W2^T [in][out]
constexpr int S_H1T = S_W2T + 128 * KB_HID;          // H1^T [unit][row]
constexpr int S_D2T = S_H1T + 128 * KB_HID;          // dH2^T [unit][row] -> dH1^T
constexpr int H2_ROW = HID / 2 + 1;                  // words of a row of H2: no bank conflicts
constexpr int S_H2 = S_D2T + 128 * KB_HID;           // H2 bf16 [row][H2_ROW words]
constexpr int S_F = S_H2 + 128 * H2_ROW * 4;         // fp32: W3, b1, b2, b3, dY, squared errors
constexpr int F_W3 = 0, F_B1 = F_W3 + OUT * HID, F_B2 = F_B1 + HID, F_B3 = F_B2 + HID,
              F_DY = F_B3 + 4, F_L = F_DY + 128 * OUT, F_END = F_L + 128 * OUT;
constexpr int SMEM_BYTES = S_F + F_END * 4;
constexpr int NT = 512;                              // threads of a tile

constexpr uint32_t SBO_IN = KB_IN * 8, SBO_HID = KB_HID * 8, LBO = 128;

__device__ __forceinline__ float bf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ unsigned short bfbits(float x) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}
__device__ __forceinline__ void st_bf16(unsigned char* base, uint32_t off, float x) {
    *reinterpret_cast<unsigned short*>(base + off) = bfbits(x);
}
// 8 consecutive K elements of one row as one 16-byte store
__device__ __forceinline__ void st_bf16x8(unsigned char* base, uint32_t off, const float* v) {
    uint4 q;
    q.x = bfbits(v[0]) | ((uint32_t)bfbits(v[1]) << 16);
    q.y = bfbits(v[2]) | ((uint32_t)bfbits(v[3]) << 16);
    q.z = bfbits(v[4]) | ((uint32_t)bfbits(v[5]) << 16);
    q.w = bfbits(v[6]) | ((uint32_t)bfbits(v[7]) << 16);
    *reinterpret_cast<uint4*>(base + off) = q;
}

// issue a K = 16*steps chain of MMAs into tmem_d (one elected thread)
__device__ __forceinline__ void mma_chain(uint32_t tmem_d, const unsigned char* a, uint32_t sbo_a,
                                          const unsigned char* b, uint32_t sbo_b, uint32_t id,
                                          int steps) {
    for (int s = 0; s < steps; ++s)
        to_tc::mma_bf16(tmem_d, to_tc::sdesc(to_tc::smem_u32(a + 256 * s), LBO, sbo_a),
                        to_tc::sdesc(to_tc::smem_u32(b + 256 * s), LBO, sbo_b), id, s > 0);
}

// CTA-wide wait on the MMA barrier; false (all threads) if any timed out
__device__ __forceinline__ bool wait_mma(uint64_t* mbar, uint32_t& phase) {
    bool ok = to_tc::mbar_wait(mbar, phase);
    phase ^= 1u;
    ok = !__syncthreads_or(!ok);
    to_tc::fence_after_sync();
    return ok;
}

__device__ __forceinline__ void publish_smem() {
    to_tc::fence_async_smem();
    to_tc::fence_before_sync();
    __syncthreads();
    to_tc::fence_after_sync();
}

// the 32 x 32 block at (r0, c0) of a 128 x 128 tile, transposed into dst: a
// core matrix at a time, four per instruction; the warp wrote it itself
__device__ __forceinline__ void transpose_block(const unsigned char* src, unsigned char* dst, int r0,
                                                int c0) {
    const int lane = threadIdx.x & 31, cg = (c0 >> 3) + (lane >> 3), in = (lane & 7) * 16;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int rg = (r0 >> 3) + i;
        uint32_t m[4];
        to_tc::ldsm_x4_t(src + rg * (KB_HID * 8) + cg * 128 + in, m);
        to_tc::stsm_x4(dst + cg * (KB_HID * 8) + rg * 128 + in, m);
    }
}

// sum of row u of a [128][128] bf16 tile, K ascending
__device__ __forceinline__ float row_sum(const unsigned char* tile, int u) {
    const unsigned char* row = tile + (u >> 3) * (KB_HID * 8) + (u & 7) * 16;
    float s = 0.0f;
#pragma unroll 4
    for (int c = 0; c < 16; ++c) {
        const uint4 q = *reinterpret_cast<const uint4*>(row + c * 128);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            s = s + __uint_as_float(w[j] << 16);
            s = s + __uint_as_float(w[j] & 0xFFFF0000u);
        }
    }
    return s;
}

// a thread's share of a tile's inputs: half a row of x, one target
struct MlpRows {
    float x[8], t;
};
__device__ __forceinline__ MlpRows load_rows(int r0, int n, const int* __restrict__ rows,
                                             const float* __restrict__ x,
                                             const float* __restrict__ t) {
    const int row = threadIdx.x & 127, which = threadIdx.x >> 7, gr = r0 + row;
    const bool valid = gr < n;
    const size_t src = valid ? (rows ? rows[gr] : gr) : 0;
    MlpRows r;
#pragma unroll
    for (int k = 0; k < 8; ++k) r.x[k] = valid && which < 2 ? x[src * IN + which * 8 + k] : 0.0f;
    r.t = valid && t && which < OUT ? t[src * OUT + which] : 0.0f;
    return r;
}

// What a CTA keeps across its tiles.
struct MlpCta {
    unsigned char* sm;
    uint64_t* mbar;
    uint32_t tmem, phase;
    bool ok;                                   // no MMA wait has expired
};

// One tile: rows r0 .. r0 + 127 of n.  Parameters are read past L1 (another
// CTA may have written them).  gp, loss only when BWD.
template <bool BWD>
__device__ __forceinline__ void mlp_tile(MlpCta& k, const float* params, int r0, int n,
                                         const MlpRows& in, float inv_count, float* y_out, float* gp,
                                         double* loss) {
    unsigned char* sm = k.sm;
    float* f = reinterpret_cast<float*>(sm + S_F);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp & 3, cq = (warp >> 2) * 32;         // 32 rows and 32 columns of the warp
    const int row = wr * 32 + lane;
    const int j128 = tid & 127, which = tid >> 7;           // one of 128, and of four
    bool ok = k.ok;

    // ---- stage parameters (bf16 operand tiles, fp32 for the SIMT parts)
    if (tid < 256) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __ldcg(params + OFF_W1 + j128 * IN + which * 8 + j);
        st_bf16x8(sm + S_W1, to_tc::kmaj_off(j128, which * 8, KB_IN, 2), v);
    }
#pragma unroll
    for (int i = 0; i < 2048 / NT; ++i) {
        const int e = tid + i * NT, o = (e & 7) | ((e >> 7) << 3), c = ((e >> 3) & 15) * 8;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __ldcg(params + OFF_W2 + o * HID + c + j);
        st_bf16x8(sm + S_B, to_tc::kmaj_off(o, c, KB_HID, 2), v);
    }
    if (BWD)
#pragma unroll
        for (int i = 0; i < 2048 / NT; ++i) {
            const int o = (which + i * (NT / 128)) * 8;
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __ldcg(params + OFF_W2 + (o + j) * HID + j128);
            st_bf16x8(sm + S_W2T, to_tc::kmaj_off(j128, o, KB_HID, 2), v);
        }
    if (tid < OUT * HID) f[F_W3 + tid] = bf(__ldcg(params + OFF_W3 + tid));
    else f[F_B1 + j128] = __ldcg(params + OFF_B1 + j128);
    if (tid < HID) f[F_B2 + tid] = __ldcg(params + OFF_B2 + tid);
    else if (tid < HID + OUT) f[F_B3 + tid - HID] = __ldcg(params + OFF_B3 + tid - HID);
    if (tid < 256) {
        st_bf16x8(sm + S_X, to_tc::kmaj_off(j128, which * 8, KB_IN, 2), in.x);
        if (BWD)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                st_bf16(sm + S_XT, to_tc::kmaj_off(which * 8 + j, j128, KB_HID, 2), in.x[j]);
    }
    publish_smem();
    const uint32_t T0 = k.tmem, T1 = k.tmem + 128;          // two 128-column accumulators

    // ---- F1
    if (ok && tid == 0) {
        mma_chain(T0, sm + S_X, SBO_IN, sm + S_W1, SBO_IN, to_tc::idesc(1, 128, HID), 1);
        to_tc::commit(k.mbar);
    }
    if (ok) ok = wait_mma(k.mbar, k.phase);
    uint32_t mask1 = 0, mask2 = 0;
    if (ok) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c0 = cq + h * 16;
            float v[16];
            to_tc::tmem_ld16(to_tc::lane_addr(T0, wr, c0), v);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float a = v[j] + f[F_B1 + c0 + j];
                if (a > 0.0f) mask1 |= 1u << (h * 16 + j);
                v[j] = a > 0.0f ? a : 0.0f;
            }
            st_bf16x8(sm + S_A, to_tc::kmaj_off(row, c0, KB_HID, 2), v);
            st_bf16x8(sm + S_A, to_tc::kmaj_off(row, c0 + 8, KB_HID, 2), v + 8);
        }
        if (BWD) transpose_block(sm + S_A, sm + S_H1T, wr * 32, cq);
    }
    publish_smem();

    // ---- F2
    if (ok && tid == 0) {
        mma_chain(T1, sm + S_A, SBO_HID, sm + S_B, SBO_HID, to_tc::idesc(1, 128, HID), HID / 16);
        to_tc::commit(k.mbar);
    }
    if (ok) ok = wait_mma(k.mbar, k.phase);
    uint32_t* h2 = reinterpret_cast<uint32_t*>(sm + S_H2);
    if (ok) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c0 = cq + h * 16;
            float v[16];
            to_tc::tmem_ld16(to_tc::lane_addr(T1, wr, c0), v);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float a = v[j] + f[F_B2 + c0 + j];
                if (a > 0.0f) mask2 |= 1u << (h * 16 + j);
                v[j] = a > 0.0f ? a : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 16; j += 2)
                h2[row * H2_ROW + ((c0 + j) >> 1)] = bfbits(v[j]) | ((uint32_t)bfbits(v[j + 1]) << 16);
        }
    }
    __syncthreads();

    // ---- layer 3 (SIMT) on bf16 H2: a thread a (row, output)
    if (tid < 128 * OUT) {
        float y = 0.0f;
        if (ok) {
            const float* w = f + F_W3 + which * HID;
#pragma unroll 8
            for (int o = 0; o < HID / 2; ++o) {
                const uint32_t u = h2[j128 * H2_ROW + o];
                y = y + __uint_as_float(u << 16) * w[2 * o];
                y = y + __uint_as_float(u & 0xFFFF0000u) * w[2 * o + 1];
            }
            y = y + f[F_B3 + which];
        }
        const bool valid = r0 + j128 < n;
        if (!BWD) {
            if (ok && valid) y_out[(size_t)(r0 + j128) * OUT + which] = y;
        } else {
            const float d = valid ? y - in.t : 0.0f;
            f[F_L + which * 128 + j128] = d * d;
            f[F_DY + j128 * OUT + which] = 2.0f * d * inv_count;
        }
    }
    if (!BWD) {
        k.ok = ok;
        return;
    }
    __syncthreads();
    // ---- dH2 = (dY W3) * relu'(a2)
    if (ok) {
        const float dy0 = f[F_DY + row * OUT + 0], dy1 = f[F_DY + row * OUT + 1],
                    dy2 = f[F_DY + row * OUT + 2];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int c0 = cq + h * 8;
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int o = c0 + j;
                const float g = (dy0 * f[F_W3 + o] + dy1 * f[F_W3 + HID + o]) + dy2 * f[F_W3 + 2 * HID + o];
                v[j] = (mask2 >> (h * 8 + j)) & 1u ? g : 0.0f;
            }
            st_bf16x8(sm + S_A, to_tc::kmaj_off(row, c0, KB_HID, 2), v);
        }
        transpose_block(sm + S_A, sm + S_D2T, wr * 32, cq);
    }
    publish_smem();
    // ---- B2 (dH1 pre-mask) into T0, G2 (dW2) into T1
    if (ok && tid == 0) {
        mma_chain(T0, sm + S_A, SBO_HID, sm + S_W2T, SBO_HID, to_tc::idesc(1, 128, HID), HID / 16);
        mma_chain(T1, sm + S_D2T, SBO_HID, sm + S_H1T, SBO_HID, to_tc::idesc(1, 128, HID), HID / 16);
        to_tc::commit(k.mbar);
    }
    // meanwhile: dW3, db2 (rows summed in order, a thread a sum), the loss
    if (which < OUT) {
        const uint32_t* hc = h2 + (j128 >> 1);
        const int sh = (j128 & 1) ? 0 : 16;
        float g = 0.0f;
#pragma unroll 8
        for (int r = 0; r < 128; ++r)
            g = g + f[F_DY + r * OUT + which] * __uint_as_float((hc[r * H2_ROW] << sh) & 0xFFFF0000u);
        gp[OFF_W3 + which * HID + j128] = g;
    } else {
        gp[OFF_B2 + j128] = row_sum(sm + S_D2T, j128);
    }
    if (warp == NT / 32 - 1) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* q = f + F_L + lane + 32 * i;
            s += (double)((q[0] + q[128]) + q[256]);
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) *loss = s;
    }
    if (ok) ok = wait_mma(k.mbar, k.phase);
    if (ok) {
        // dH1 = B2 * relu'(a1), transposed for G1; dW2 rows out
        float4* dst = reinterpret_cast<float4*>(gp + OFF_W2 + (size_t)row * HID + cq);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c0 = cq + h * 16;
            float v[16];
            to_tc::tmem_ld16(to_tc::lane_addr(T0, wr, c0), v);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = (mask1 >> (h * 16 + j)) & 1u ? v[j] : 0.0f;
            st_bf16x8(sm + S_A, to_tc::kmaj_off(row, c0, KB_HID, 2), v);
            st_bf16x8(sm + S_A, to_tc::kmaj_off(row, c0 + 8, KB_HID, 2), v + 8);
        }
        transpose_block(sm + S_A, sm + S_D2T, wr * 32, cq);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float v[16];
            to_tc::tmem_ld16(to_tc::lane_addr(T1, wr, cq + h * 16), v);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                dst[h * 4 + j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
    }
    publish_smem();
    // ---- G1 (dW1) into T0
    if (ok && tid == 0) {
        mma_chain(T0, sm + S_D2T, SBO_HID, sm + S_XT, SBO_HID, to_tc::idesc(1, 128, IN), HID / 16);
        to_tc::commit(k.mbar);
    }
    if (which == 0) {
        gp[OFF_B1 + j128] = row_sum(sm + S_D2T, j128);
    } else if (tid >= 128 && tid < 128 + OUT) {
        float s = 0.0f;
#pragma unroll 8
        for (int r = 0; r < 128; ++r) s = s + f[F_DY + r * OUT + (tid - 128)];
        gp[OFF_B3 + tid - 128] = s;
    }
    if (ok) ok = wait_mma(k.mbar, k.phase);
    if (ok && warp < 4) {
        float v[16];
        to_tc::tmem_ld16(to_tc::lane_addr(T0, warp, 0), v);
        float4* dst = reinterpret_cast<float4*>(gp + OFF_W1 + (size_t)row * IN);
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    k.ok = ok;
}

__device__ __forceinline__ MlpCta mlp_enter(unsigned char* sm, uint64_t* mbar, uint32_t* tslot) {
    if (threadIdx.x == 0) to_tc::mbar_init(mbar, 1);
    if (threadIdx.x < 32) to_tc::tmem_alloc<256>(tslot);
    publish_smem();
    MlpCta k;
    k.sm = sm; k.mbar = mbar; k.tmem = *tslot; k.phase = 0; k.ok = true;
    return k;
}
__device__ __forceinline__ void mlp_leave(const MlpCta& k, int* err) {
    if (!k.ok && threadIdx.x == 0) atomicExch(err, TO_DEVERR_SPIN);
    to_tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) to_tc::tmem_free<256>(k.tmem);
}

// rows: optional row index list (training order); t/part/loss only when BWD
template <bool BWD>
__global__ void __launch_bounds__(NT, 1)
k_mlp(const float* params, int n, const int* __restrict__ rows, const float* __restrict__ x,
      const float* __restrict__ t, float inv_count, float* __restrict__ y_out,
      float* __restrict__ part, double* __restrict__ loss_part, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char sm_mlp[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tslot;
    const int r0 = blockIdx.x * 128;
    const MlpRows in = load_rows(r0, n, rows, x, BWD ? t : nullptr);
    MlpCta k = mlp_enter(sm_mlp, &mbar, &tslot);
    mlp_tile<BWD>(k, params, r0, n, in, inv_count, y_out,
                  BWD ? part + (size_t)blockIdx.x * PSTRIDE : nullptr,
                  BWD ? loss_part + blockIdx.x : nullptr);
    mlp_leave(k, err);
}

// All CTAs of a cooperative launch: their writes before are seen after.
// False (everywhere) when the others do not come within a second.
__device__ __forceinline__ bool grid_meet(unsigned* counter, unsigned& target) {
    target += gridDim.x;
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(counter, 1u);
        uint64_t t0 = to_tc::now_ns();
        while ((int)(to_tc::ld_acquire(counter) - target) < 0)
            if (to_tc::now_ns() - t0 > 1000000000ull) { ok = false; break; }
        __threadfence();
    }
    return !__syncthreads_or(!ok);
}

// Adam's state and constants
struct MlpAdam {
    float *params, *m, *v;                     // [PSTRIDE]
    const float2* corr;                        // bias corrections of each step
    float lr, b1, b2, eps;
};
__device__ __forceinline__ void adam_update(const MlpAdam& a, float g, float& m, float& v, float& p,
                                            float c1, float c2) {
    m = a.b1 * m + (1.0f - a.b1) * g;
    v = a.b2 * v + (1.0f - a.b2) * g * g;
    p = p - a.lr * (m / c1) / (sqrtf(v / c2) + a.eps);
}

// One epoch in one cooperative launch: a step's tiles a CTA each, then the
// gradient sums and Adam spread over all CTAs.  The next step's rows are
// fetched before the CTAs meet.
__global__ void __launch_bounds__(NT, 1)
k_mlp_epoch(MlpAdam ad, int n, int batch, const int* __restrict__ rows, const float* __restrict__ x,
            const float* __restrict__ t, float* part, double* loss_part, double* loss,
            unsigned* counter, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char sm_mlp[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tslot;
    const int r0 = blockIdx.x * 128, tid = threadIdx.x;
    MlpRows in = load_rows(r0, min(batch, n), rows, x, t);
    MlpCta k = mlp_enter(sm_mlp, &mbar, &tslot);
    unsigned target = 0;
    int step = 0;
    for (int s0 = 0; s0 < n; s0 += batch, ++step) {
        const int bs = min(batch, n - s0), tiles = (bs + 127) / 128;
        if ((int)blockIdx.x < tiles)
            mlp_tile<true>(k, ad.params, r0, bs, in, 1.0f / (3.0f * (float)bs), nullptr,
                           part + (size_t)blockIdx.x * PSTRIDE, loss_part + blockIdx.x);
        if (s0 + batch < n) in = load_rows(r0, min(batch, n - s0 - batch), rows + s0 + batch, x, t);
        to_tc::fence_before_sync();
        if (!grid_meet(counter, target)) { k.ok = false; break; }
        to_tc::fence_after_sync();
        const float2 c = ad.corr[step];
        for (int q = blockIdx.x * NT + tid; q < PSTRIDE / 4; q += gridDim.x * NT) {
            float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            float4 m = __ldcg(reinterpret_cast<const float4*>(ad.m) + q);
            float4 v = __ldcg(reinterpret_cast<const float4*>(ad.v) + q);
            float4 p = __ldcg(reinterpret_cast<const float4*>(ad.params) + q);
#pragma unroll 4
            for (int i = 0; i < tiles; ++i) {
                const float4 d = __ldcg(reinterpret_cast<const float4*>(part + (size_t)i * PSTRIDE) + q);
                g.x = g.x + d.x; g.y = g.y + d.y; g.z = g.z + d.z; g.w = g.w + d.w;
            }
            adam_update(ad, g.x, m.x, v.x, p.x, c.x, c.y);
            adam_update(ad, g.y, m.y, v.y, p.y, c.x, c.y);
            adam_update(ad, g.z, m.z, v.z, p.z, c.x, c.y);
            adam_update(ad, g.w, m.w, v.w, p.w, c.x, c.y);
            reinterpret_cast<float4*>(ad.m)[q] = m;
            reinterpret_cast<float4*>(ad.v)[q] = v;
            reinterpret_cast<float4*>(ad.params)[q] = p;
        }
        if (blockIdx.x == 0 && tid == 0) {
            double s = 0.0;
            for (int i = 0; i < tiles; ++i) s += __ldcg(loss_part + i);
            *loss += s;
        }
        if (!grid_meet(counter, target)) { k.ok = false; break; }
    }
    mlp_leave(k, err);
}

// grad = sum of tile partials (tile order); optional Adam update
__global__ void k_mlp_adam(int tiles, const float* __restrict__ part, float* __restrict__ grad,
                           float* __restrict__ params, float* __restrict__ m,
                           float* __restrict__ v, float lr, float b1, float b2, float eps,
                           float c1, float c2) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= NPARAM) return;
    float g = 0.0f;
    for (int i = 0; i < tiles; ++i) g = g + part[(size_t)i * PSTRIDE + p];
    if (grad) grad[p] = g;
    if (params) {
        float mm = b1 * m[p] + (1.0f - b1) * g;
        float vv = b2 * v[p] + (1.0f - b2) * g * g;
        m[p] = mm;
        v[p] = vv;
        params[p] = params[p] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    }
}

__global__ void k_sum_loss(int tiles, const double* __restrict__ lp, double* __restrict__ out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < tiles; ++i) s += lp[i];
        *out += s;
    }
}

template <bool BWD>
to_status launch_mlp(to_ctx ctx, const float* params, int n, const int* rows, const float* x,
                     const float* t, float inv_count, float* y, float* part, double* lp) {
    static bool attr[2] = {false, false};
    if (!attr[BWD]) {
        TO_CUDA(ctx, cudaFuncSetAttribute(k_mlp<BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          SMEM_BYTES));
        attr[BWD] = true;
    }
    const int tiles = (n + 127) / 128;
    to_prof_begin(ctx, BWD ? "mlp_fwd_bwd" : "mlp_fwd");
    k_mlp<BWD><<<tiles, NT, SMEM_BYTES, ctx->stream>>>(params, n, rows, x, t, inv_count, y, part,
                                                         lp, ctx->d_flags);
    to_prof_end(ctx);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

}  // namespace

namespace to_k {

to_status mlp_forward(to_ctx ctx, const float* d_params, int n, const float* d_x, float* d_y) {
    if (n <= 0) return TO_OK;
    return launch_mlp<false>(ctx, d_params, n, nullptr, d_x, nullptr, 0.0f, d_y, nullptr, nullptr);
}

// one epoch over n rows in the order d_rows; false in *done (and nothing
// launched) when the CTAs of a step's tiles cannot all be resident
to_status mlp_epoch(to_ctx ctx, const MlpAdam& ad, int n, int batch, const int* d_rows,
                    const float* d_x, const float* d_t, float* d_part, double* d_lp, double* d_loss,
                    unsigned* d_counter, bool* done) {
    *done = false;
    const int tiles = (batch + 127) / 128, sms = ctx->sm_count > 0 ? ctx->sm_count : TO_SM_TARGET;
    if (tiles > sms) return TO_OK;
    int grid = (PSTRIDE / 4 + NT - 1) / NT;    // Adam: four parameters a thread
    if (grid > sms) grid = sms;
    if (grid < tiles) grid = tiles;
    TO_CUDA(ctx, cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      SMEM_BYTES));
    TO_CUDA(ctx, cudaMemsetAsync(d_counter, 0, sizeof(unsigned), ctx->stream));
    to_prof_begin(ctx, "mlp_fwd_bwd");
    MlpAdam a = ad;
    int* err = ctx->d_flags;
    void* args[] = {&a, &n, &batch, &d_rows, &d_x, &d_t, &d_part, &d_lp, &d_loss, &d_counter, &err};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_mlp_epoch, dim3(grid), dim3(NT),
                                                      args, SMEM_BYTES, ctx->stream);
    to_prof_end(ctx);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return TO_OK;
    }
    TO_CUDA(ctx, e);
    TO_LAUNCHED(ctx);
    *done = true;
    return TO_OK;
}

size_t mlp_part_floats(int n) { return (size_t)((n + 127) / 128) * PSTRIDE; }

// gradient of mean((y - t)^2) over the n selected rows; d_part: mlp_part_floats(n)
to_status mlp_grad(to_ctx ctx, const float* d_params, int n, const int* d_rows, const float* d_x,
                   const float* d_t, float* d_part, double* d_lp, float* d_grad, float* d_params_upd,
                   float* d_m, float* d_v, float lr, int step) {
    const int tiles = (n + 127) / 128;
    TO_TRY(launch_mlp<true>(ctx, d_params, n, d_rows, d_x, d_t, 1.0f / (3.0f * (float)n), nullptr,
                            d_part, d_lp));
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    k_mlp_adam<<<(NPARAM + 255) / 256, 256, 0, ctx->stream>>>(tiles, d_part, d_grad, d_params_upd,
                                                              d_m, d_v, lr, b1, b2, 1e-8f, c1, c2);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

to_status mlp_sum_loss(to_ctx ctx, int tiles, const double* d_lp, double* d_out) {
    k_sum_loss<<<1, 32, 0, ctx->stream>>>(tiles, d_lp, d_out);
    TO_LAUNCHED(ctx);
    return TO_OK;
}

}  // namespace to_k

// ---- C ABI ------------------------------------------------------------------
namespace {

to_status mlp_check_flags(to_ctx ctx) {
    int f = 0;
    TO_TRY(to_read_device_flags(ctx, &f));
    if (f != TO_DEVERR_NONE) {
        int z = 0;
        TO_CUDA(ctx, cudaMemcpy(ctx->d_flags, &z, sizeof(int), cudaMemcpyHostToDevice));
        return to_set_error(ctx, TO_ERR_TIMEOUT, "tensor-core wait expired in the MLP kernel");
    }
    return TO_OK;
}

// seeded Fisher-Yates shuffle (splitmix64 stream)
void shuffle_rows(int* r, int n, uint64_t& state) {
    for (int i = 0; i < n; ++i) r[i] = i;
    for (int i = n - 1; i > 0; --i) {
        state += 0x9E3779B97F4A7C15ull;
        uint64_t z = state;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        int j = (int)(z % (uint64_t)(i + 1));
        int t = r[i]; r[i] = r[j]; r[j] = t;
    }
}

bool finite_all(const float* v, size_t n) {
    for (size_t i = 0; i < n; ++i)
        if (!std::isfinite(v[i])) return false;
    return true;
}

}  // namespace

extern "C" {

to_status to_mlp_predict_d(to_ctx ctx, const float* d_params, int n, const float* d_x, float* d_y) {
    if (!ctx || n < 0 || (n > 0 && (!d_params || !d_x || !d_y))) return TO_ERR_INVALID;
    cudaSetDevice(ctx->device);
    return to_k::mlp_forward(ctx, d_params, n, d_x, d_y);
}

to_status to_mlp_predict(to_ctx ctx, const float* params, int n, const float* x, float* y) {
    if (!ctx || !params || n < 0 || (n > 0 && (!x || !y))) return TO_ERR_INVALID;
    if (n == 0) return TO_OK;
    cudaSetDevice(ctx->device);
    const size_t bytes = to_align256((size_t)NPARAM * 4) + to_align256((size_t)n * IN * 4) +
                         to_align256((size_t)n * OUT * 4);
    TO_TRY(to_arena_reserve(ctx, bytes + 1024));
    float* d_p = to_arena_take<float>(ctx, NPARAM);
    float* d_x = to_arena_take<float>(ctx, (size_t)n * IN);
    float* d_y = to_arena_take<float>(ctx, (size_t)n * OUT);
    TO_CUDA(ctx, cudaMemcpyAsync(d_p, params, (size_t)NPARAM * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(d_x, x, (size_t)n * IN * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_TRY(to_k::mlp_forward(ctx, d_p, n, d_x, d_y));
    TO_CUDA(ctx, cudaMemcpyAsync(y, d_y, (size_t)n * OUT * 4, cudaMemcpyDeviceToHost, ctx->stream));
    TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return mlp_check_flags(ctx);
}

to_status to_mlp_grad(to_ctx ctx, const float* params, int n, const float* x, const float* t,
                      float* grad, double* loss) {
    if (!ctx || !params || n <= 0 || !x || !t || !grad) return TO_ERR_INVALID;
    cudaSetDevice(ctx->device);
    const int tiles = (n + 127) / 128;
    const size_t bytes = to_align256((size_t)NPARAM * 4) * 2 + to_align256((size_t)n * IN * 4) +
                         to_align256((size_t)n * OUT * 4) + to_align256(to_k::mlp_part_floats(n) * 4) +
                         to_align256((size_t)tiles * 8) + 256;
    TO_TRY(to_arena_reserve(ctx, bytes + 1024));
    float* d_p = to_arena_take<float>(ctx, NPARAM);
    float* d_g = to_arena_take<float>(ctx, NPARAM);
    float* d_x = to_arena_take<float>(ctx, (size_t)n * IN);
    float* d_t = to_arena_take<float>(ctx, (size_t)n * OUT);
    float* d_part = to_arena_take<float>(ctx, to_k::mlp_part_floats(n));
    double* d_lp = to_arena_take<double>(ctx, tiles);
    double* d_l = to_arena_take<double>(ctx, 1);
    TO_CUDA(ctx, cudaMemcpyAsync(d_p, params, (size_t)NPARAM * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(d_x, x, (size_t)n * IN * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(d_t, t, (size_t)n * OUT * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemsetAsync(d_l, 0, 8, ctx->stream));
    TO_TRY(to_k::mlp_grad(ctx, d_p, n, nullptr, d_x, d_t, d_part, d_lp, d_g, nullptr, nullptr,
                          nullptr, 0.0f, 1));
    TO_TRY(to_k::mlp_sum_loss(ctx, tiles, d_lp, d_l));
    double l = 0.0;
    TO_CUDA(ctx, cudaMemcpyAsync(grad, d_g, (size_t)NPARAM * 4, cudaMemcpyDeviceToHost, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(&l, d_l, 8, cudaMemcpyDeviceToHost, ctx->stream));
    TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (loss) *loss = l / (3.0 * n);
    return mlp_check_flags(ctx);
}

to_status to_mlp_train(to_ctx ctx, float* params, int n, const float* x, const float* t,
                       int epochs, int batch, float lr, uint64_t seed, double* loss_curve) {
    if (!ctx || !params || n <= 0 || !x || !t || epochs < 0 || batch <= 0 || !(lr > 0.0f))
        return TO_ERR_INVALID;
    if (!finite_all(x, (size_t)n * IN) || !finite_all(t, (size_t)n * OUT) ||
        !finite_all(params, NPARAM))
        return to_set_error(ctx, TO_ERR_NONFINITE, "non-finite MLP training input");
    cudaSetDevice(ctx->device);
    if (batch > n) batch = n;
    const int tiles = (batch + 127) / 128;
    const size_t ep = epochs > 0 ? epochs : 1;
    const size_t spe = ((size_t)n + batch - 1) / batch;        // steps an epoch
    const size_t bytes = to_align256((size_t)PSTRIDE * 4) * 3 + to_align256((size_t)n * IN * 4) +
                         to_align256((size_t)n * OUT * 4) + to_align256(ep * n * 4) +
                         to_align256(to_k::mlp_part_floats(batch) * 4) + to_align256((size_t)tiles * 8) +
                         to_align256(ep * 8) + to_align256(ep * spe * 8) + 256;
    TO_TRY(to_arena_reserve(ctx, bytes + 2048));
    MlpAdam ad;
    float* d_p = ad.params = to_arena_take<float>(ctx, PSTRIDE);
    float* d_m = ad.m = to_arena_take<float>(ctx, PSTRIDE);
    float* d_v = ad.v = to_arena_take<float>(ctx, PSTRIDE);
    float* d_x = to_arena_take<float>(ctx, (size_t)n * IN);
    float* d_t = to_arena_take<float>(ctx, (size_t)n * OUT);
    int* d_rows = to_arena_take<int>(ctx, ep * n);
    float* d_part = to_arena_take<float>(ctx, to_k::mlp_part_floats(batch));
    double* d_lp = to_arena_take<double>(ctx, tiles);
    double* d_loss = to_arena_take<double>(ctx, ep);
    float2* d_corr = to_arena_take<float2>(ctx, ep * spe);
    unsigned* d_counter = to_arena_take<unsigned>(ctx, 1);
    if (!d_counter) return to_set_error(ctx, TO_ERR_ALLOC, "arena sizing");
    ad.lr = lr; ad.b1 = 0.9f; ad.b2 = 0.999f; ad.eps = 1e-8f;
    std::vector<int> rows((size_t)n);
    std::vector<float2> corr(ep * spe);
    for (size_t i = 0; i < corr.size(); ++i)
        corr[i] = make_float2(1.0f - powf(ad.b1, (float)(i + 1)), 1.0f - powf(ad.b2, (float)(i + 1)));
    uint64_t st = seed;
    TO_CUDA(ctx, cudaMemcpyAsync(d_p, params, (size_t)NPARAM * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemsetAsync(d_m, 0, (size_t)PSTRIDE * 4, ctx->stream));
    TO_CUDA(ctx, cudaMemsetAsync(d_v, 0, (size_t)PSTRIDE * 4, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(d_x, x, (size_t)n * IN * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(d_t, t, (size_t)n * OUT * 4, cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(d_corr, corr.data(), corr.size() * sizeof(float2),
                                 cudaMemcpyHostToDevice, ctx->stream));
    TO_CUDA(ctx, cudaMemsetAsync(d_loss, 0, ep * 8, ctx->stream));
    int step = 0;
    for (int e = 0; e < epochs; ++e) {
        // an epoch's order is drawn while the GPU works on the one before
        int* d_order = d_rows + (size_t)e * n;
        shuffle_rows(rows.data(), n, st);
        TO_CUDA(ctx, cudaMemcpyAsync(d_order, rows.data(), (size_t)n * 4, cudaMemcpyHostToDevice,
                                     ctx->stream));
        ad.corr = d_corr + (size_t)e * spe;
        bool done = false;
        TO_TRY(to_k::mlp_epoch(ctx, ad, n, batch, d_order, d_x, d_t, d_part, d_lp, d_loss + e,
                               d_counter, &done));
        if (done) continue;
        step = (int)(e * spe);
        for (int s0 = 0; s0 < n; s0 += batch) {
            const int bs = n - s0 < batch ? n - s0 : batch;
            ++step;
            TO_TRY(to_k::mlp_grad(ctx, d_p, bs, d_order + s0, d_x, d_t, d_part, d_lp, nullptr, d_p,
                                  d_m, d_v, lr, step));
            TO_TRY(to_k::mlp_sum_loss(ctx, (bs + 127) / 128, d_lp, d_loss + e));
        }
    }
    std::vector<double> lc(ep);
    TO_CUDA(ctx, cudaMemcpyAsync(params, d_p, (size_t)NPARAM * 4, cudaMemcpyDeviceToHost, ctx->stream));
    TO_CUDA(ctx, cudaMemcpyAsync(lc.data(), d_loss, ep * 8, cudaMemcpyDeviceToHost, ctx->stream));
    TO_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (loss_curve)
        for (int e = 0; e < epochs; ++e) loss_curve[e] = lc[e] / (3.0 * n);
    return mlp_check_flags(ctx);
}

}  // extern "C"
