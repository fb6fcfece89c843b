// silu_row.cuh -- SiLU*up and the int8 form of one pair's 512 values (maple.c:825-832) by one warp: lane l holds columns 128 i + 4 l .. + 3
// for i = 0..3 (every access of the warp to the row covers one contiguous run).
//
// The int8 row, its scale and its sum are the reference's bits.  act ~ g / (1 + 2^(-g log2 e)) u is evaluated with the hardware's
// approximate exponential and reciprocal (relative error below SQ_EPS for every g <= 7 that does not underflow) and again exactly
// (dev_math.cuh) only where the approximation could change a result:
//   * the row maximum: every element within 2 SQ_EPS of the approximate maximum is evaluated exactly, the exact maximum is among them;
//   * a rounded value: t = act * inv lands within |t| (2 SQ_EPS + 2^-22) of a rounding boundary (about one element in two thousand).
#pragma once
#include "dev_math.cuh"

#define SQ_EPS 1.2e-5f
__device__ __forceinline__ float silu_mul_approx(float g, float u) {
    g = g < 7.0f ? g : 7.0f;
    u = u < -7.0f ? -7.0f : (u > 7.0f ? 7.0f : u);
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return g * r * u;
}
// g4, u4: this lane's part of the row (values 128 i + 4 l .. of gate and up); gate, up: the row in global memory, from which the few
// elements that need it are read again: the exact evaluation is a hundred instructions, and thirty-two inlined copies of it (one per
// element and use) cost more in instruction fetches than the arithmetic (16,384 rows 24.3 -> 22.5 us).
// pk[i]: the four int8 values of columns 128 i + 4 l ..; s: the row's scale, tot: the row's sum (both on every lane)
__device__ __forceinline__ void silu_quant_row(const float4 (&g4)[4], const float4 (&u4)[4], const float *gate, const float *up, const unsigned long long *tab,
                                               const int lane, uint32_t (&pk)[4], float &s, int &tot) {
    float v[16], mxa = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        v[4 * i] = silu_mul_approx(g4[i].x, u4[i].x); v[4 * i + 1] = silu_mul_approx(g4[i].y, u4[i].y);
        v[4 * i + 2] = silu_mul_approx(g4[i].z, u4[i].z); v[4 * i + 3] = silu_mul_approx(g4[i].w, u4[i].w);
    }
#pragma unroll
    for (int i = 0; i < 16; i++) mxa = fmaxf(mxa, fabsf(v[i]));
    mxa = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mxa)));        // >= 0: the bits order like the values
    const float thr = mxa * (1.0f - 2.5f * SQ_EPS) - 1e-30f;          // every element that can be the exact maximum
    unsigned todo = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) todo |= !(fabsf(v[i]) < thr) ? 1u << i : 0u;
    auto exact = [&](const int i) { const int c = 128 * (i >> 2) + 4 * lane + (i & 3); return dev_silu_mul_tab(__ldcg(gate + c), __ldcg(up + c), tab); };
    float mx = 0.0f;
#pragma unroll 1
    for (; __any_sync(0xffffffffu, todo != 0u); todo &= todo - 1u) if (todo) mx = fmaxf(mx, fabsf(exact(__ffs(todo) - 1)));
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    s = mx > 0.0f ? __fdiv_rn(mx, 127.0f) : 1.0f;
    const float inv = __fdiv_rn(1.0f, s), slack = 1e-36f * inv;       // slack: elements the approximation flushed to zero
    tot = 0; todo = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) pk[i] = 0u;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const float t = __fmul_rn(v[i], inv), big = __fadd_rn(t, 12582912.0f), r = __fsub_rn(big, 12582912.0f);      // r = t rounded to an integer, half to even
        const int qi = __float_as_int(big) - 0x4B400000;
        const bool near = !(0.5f - fabsf(__fsub_rn(t, r)) > fabsf(t) * (2.0f * SQ_EPS + 2.4e-7f) + slack);
        todo |= near ? 1u << i : 0u;                                   // such an element is left zero here
        tot += near ? 0 : qi; pk[i >> 2] |= near ? 0u : (uint32_t)(qi & 0xFF) << (8 * (i & 3));
    }
#pragma unroll 1
    for (; __any_sync(0xffffffffu, todo != 0u); todo &= todo - 1u) if (todo) {
        const int i = __ffs(todo) - 1, qi = __float2int_rn(__fmul_rn(exact(i), inv));
        tot += qi;
#pragma unroll
        for (int w = 0; w < 4; w++) if (w == i >> 2) pk[w] |= (uint32_t)(qi & 0xFF) << (8 * (i & 3));
    }
    tot = __reduce_add_sync(0xffffffffu, tot);
}
