// to_f2.cuh - two floats in one 64-bit register pair (low half first): the
// packed FP32 instructions of sm_100+ (add / mul / fma.rn.f32x2), each half
// rounded exactly as the scalar operation - and the growth normals of two
// paths at a time in that form.
#pragma once
#include <cuda_runtime.h>

#include "to_math.h"

typedef unsigned long long f2;

__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void bits2(f2 v, unsigned& a, unsigned& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
}
__device__ __forceinline__ void unpack2(f2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 both2(float a) { return pack2(a, a); }
__device__ __forceinline__ f2 neg2(f2 v) { return v ^ 0x8000000080000000ull; }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// both words of a 32 x 32 product from one instruction
__device__ __forceinline__ void to_mul_wide(uint32_t a, uint32_t b, uint32_t& hi, uint32_t& lo) {
    const unsigned long long p = (unsigned long long)a * b;
    hi = (uint32_t)(p >> 32);
    lo = (uint32_t)p;
}

// Philox round keys of a seed (20 words: kernel arguments, so that the
// rounds read them from the constant bank instead of adding them up)
struct to_round_keys {
    uint32_t k[20];
};
static inline to_round_keys to_make_round_keys(uint64_t seed) {
    to_round_keys r;
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
    for (int i = 0; i < 10; ++i) {
        r.k[2 * i] = k0;
        r.k[2 * i + 1] = k1;
        k0 += TO_PHILOX_W0;
        k1 += TO_PHILOX_W1;
    }
    return r;
}

// The stream block of to_stream_block(seed, stream, road, path, year, group)
// taken apart by what changes: the products of round 0 and half of round 1
// depend on the path and year only, the others on the group only (one for
// all lanes and paths), so a group costs eight rounds a path.
struct to_path_stream {
    uint32_t h1, l1;       // M1 * path
    uint32_t H0, L0;       // M0 * (round 0's first word)
};
__device__ __forceinline__ void to_stream_path(to_path_stream& s, uint32_t path) {
    to_mul_wide(TO_PHILOX_M1, path, s.h1, s.l1);
}
__device__ __forceinline__ void to_stream_year(to_path_stream& s, uint32_t year,
                                               const to_round_keys& rk) {
    to_mul_wide(TO_PHILOX_M0, s.h1 ^ year ^ rk.k[0], s.H0, s.L0);
}
struct to_group_stream {
    uint32_t l0, H1, L1;
};
__device__ __forceinline__ to_group_stream to_stream_group(uint32_t group, uint32_t stream_road,
                                                           const to_round_keys& rk) {
    to_group_stream g;
    uint32_t h0;
    to_mul_wide(TO_PHILOX_M0, group, h0, g.l0);
    to_mul_wide(TO_PHILOX_M1, h0 ^ stream_road ^ rk.k[1], g.H1, g.L1);
    return g;
}
__device__ __forceinline__ to_u32x4 to_stream_words(const to_path_stream& s,
                                                    const to_group_stream& g,
                                                    const to_round_keys& rk) {
    uint32_t c0 = g.H1 ^ s.l1 ^ rk.k[2], c1 = g.L1, c2 = s.H0 ^ g.l0 ^ rk.k[3], c3 = s.L0;
#pragma unroll
    for (int r = 2; r < 10; ++r) {
        uint32_t hi0, lo0, hi1, lo1;
        to_mul_wide(TO_PHILOX_M0, c0, hi0, lo0);
        to_mul_wide(TO_PHILOX_M1, c2, hi1, lo1);
        c0 = hi1 ^ c1 ^ rk.k[2 * r];
        c1 = lo1;
        c2 = hi0 ^ c3 ^ rk.k[2 * r + 1];
        c3 = lo0;
    }
    to_u32x4 o;
    o.v[0] = c0; o.v[1] = c1; o.v[2] = c2; o.v[3] = c3;
    return o;
}

// the log and sine tables, 128 entries each, as a CTA keeps them in shared
// memory
struct to_bm_tables {
    to_f2 log[128], sc[128];
};
__device__ __forceinline__ void to_bm_load(to_bm_tables& t) {
    for (int i = threadIdx.x; i < 128; i += blockDim.x) {
        t.log[i] = to_log_entry(i);
        t.sc[i] = to_sincos_entry(i);
    }
}

// The rounded square roots of two values -2 log(u) of the 24-bit uniforms:
// one Newton step on the reciprocal square root's estimate, its residual in
// one FMA (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990).  For arguments of 0, of which it makes 0, and
// from 1e-30 to 35 (the smallest here but 0 is 2.4e-7): on all of them, every
// one of the 2^24 values of u, it equals sqrtf (tests/test_gpu_f2_math.py).
// The forward pass of 256 roads, 768 paths, 3 species: 39.1 -> 38.1 ms.
__device__ __forceinline__ f2 to_sqrt2(f2 x) {
    float x0, x1, y0, y1;
    unpack2(x, x0, x1);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(fmaxf(x0, 1e-30f)));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(fmaxf(x1, 1e-30f)));
    const f2 y = pack2(y0, y1), g = mul2(x, y);
    return fma2(fma2(neg2(g), g, x), mul2(y, both2(0.5f)), g);
}

// to_box_muller of two paths' words: the same operations, packed
__device__ __forceinline__ void to_box_muller2(uint32_t a0, uint32_t b0, uint32_t a1, uint32_t b1,
                                               const to_bm_tables& tab, f2& z0, f2& z1) {
    // to_log_u01
    const f2 u = mul2(add2(pack2((float)(a0 >> 8), (float)(a1 >> 8)), both2(0.5f)),
                      both2(0x1p-24f));
    uint32_t x0, x1;
    bits2(u, x0, x1);
    const int i0 = (int)((x0 >> 16) & 127u), i1 = (int)((x1 >> 16) & 127u);
    const to_f2 g0 = tab.log[i0], g1 = tab.log[i1];
    // the exponent, one more from entry TO_LOG_SPLIT on: by a carry
    constexpr uint32_t up = ((128u - TO_LOG_SPLIT) << 16) - (127u << 23);
    const int e0 = (int)(x0 + up) >> 23, e1 = (int)(x1 + up) >> 23;
    const f2 m = pack2(to_u2f((x0 & 0x007FFFFFu) | 0x3F800000u),
                       to_u2f((x1 & 0x007FFFFFu) | 0x3F800000u));
    const f2 t = fma2(m, pack2(g0.a, g1.a), both2(-1.0f));
    f2 q = fma2(t, both2(-0.25f), both2(0x1.555556p-2f));
    q = mul2(fma2(t, q, both2(-0.5f)), t);
    const f2 lg = add2(pack2(g0.b, g1.b), fma2(q, t, t));
    const f2 fe = pack2((float)e0, (float)e1);
    const f2 lu = fma2(fe, both2(0x1.62e430p-1f), fma2(fe, both2(-0x1.05c610p-29f), lg));
    const f2 rad = to_sqrt2(mul2(both2(-2.0f), lu));
    // to_sincos2pi_u01
    const f2 r = mul2(pack2((float)((b0 >> 8) & 0x1FFFFu), (float)((b1 >> 8) & 0x1FFFFu)),
                      both2(0x1.921fb6p-22f));
    const f2 r2 = mul2(r, r);
    f2 s = fma2(r2, both2(0x1.111112p-7f), both2(-0x1.555556p-3f));
    s = fma2(mul2(r2, r), s, r);
    f2 c = fma2(r2, both2(0x1.555556p-5f), both2(-0.5f));
    c = fma2(r2, c, both2(1.0f));
    const to_f2 s0 = tab.sc[b0 >> 25], s1 = tab.sc[b1 >> 25];
    const f2 sa = pack2(s0.a, s1.a), sb = pack2(s0.b, s1.b);
    const f2 sn = fma2(sa, c, mul2(sb, s));
    const f2 cs = fma2(sb, c, neg2(mul2(sa, s)));
    z0 = mul2(rad, cs);
    z1 = mul2(rad, sn);
}

// to_normal4 of two paths
__device__ __forceinline__ void to_normal4x2(const to_path_stream& p0, const to_path_stream& p1,
                                             const to_group_stream& g, const to_round_keys& rk,
                                             const to_bm_tables& tab, f2 (&z)[4]) {
    const to_u32x4 a = to_stream_words(p0, g, rk), b = to_stream_words(p1, g, rk);
    to_box_muller2(a.v[0], a.v[1], b.v[0], b.v[1], tab, z[0], z[1]);
    to_box_muller2(a.v[2], a.v[3], b.v[2], b.v[3], tab, z[2], z[3]);
}
