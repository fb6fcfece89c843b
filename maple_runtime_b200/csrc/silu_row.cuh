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
// gate, up: the row, of which a lane touches nothing but its own columns (so each lane may have brought them itself); the few elements that need it are read
// again from there: the exact evaluation is a hundred instructions, and inlined copies of it (one per element and use) cost more in instruction fetches than the
// arithmetic (16,384 rows 24.3 -> 22.5 us).  pk[i]: the four int8 values of columns 128 i + 4 l ..; s: the row's scale, tot: the row's sum (both on every lane)
__device__ __forceinline__ void silu_quant_row(const float *gate, const float *up, const unsigned long long *tab, const int lane, uint32_t (&pk)[4], float &s, int &tot) {
    float v[16], lm = 0.0f, mx = 0.0f;
    auto exact = [&](const int i) { const int c = 128 * (i >> 2) + 4 * lane + (i & 3); return dev_silu_mul_tab(gate[c], up[c], tab); };
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float4 g = reinterpret_cast<const float4 *>(gate)[32 * i + lane], u = reinterpret_cast<const float4 *>(up)[32 * i + lane];
        v[4 * i] = silu_mul_approx(g.x, u.x); v[4 * i + 1] = silu_mul_approx(g.y, u.y); v[4 * i + 2] = silu_mul_approx(g.z, u.z); v[4 * i + 3] = silu_mul_approx(g.w, u.w);
    }
#pragma unroll
    for (int i = 0; i < 16; i++) lm = fmaxf(lm, fabsf(v[i]));
    const float mxa = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(lm)));        // >= 0: the bits order like the values
    const float thr = mxa * (1.0f - 2.5f * SQ_EPS) - 1e-30f;           // every element that can be the exact maximum
    unsigned todo = 0;
    if (!(lm < thr)) {                                                  // one lane, nearly always
#pragma unroll
        for (int i = 0; i < 16; i++) todo |= !(fabsf(v[i]) < thr) ? 1u << i : 0u;
    }
#pragma unroll 1
    for (; __any_sync(0xffffffffu, todo != 0u); todo &= todo - 1u) if (todo) mx = fmaxf(mx, fabsf(exact(__ffs(todo) - 1)));
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    s = mx > 0.0f ? __fdiv_rn(mx, 127.0f) : 1.0f;
    const float inv = __fdiv_rn(1.0f, s), lim = 0.5f - 1e-36f * inv;   // the subtrahend: elements the approximation flushed to zero
    // t rounded to an integer (half to even) is the low bits of t + 1.5 * 2^23.  How near any of the lane's elements comes to a rounding boundary is one maximum (over
    // the bits, which are those of a value >= 0 or of a NaN, and a NaN counts as near)
    auto near_of = [&](const float t, const float bf) { return __fmaf_rn(fabsf(t), 2.0f * SQ_EPS + 2.4e-7f, fabsf(__fsub_rn(t, __fsub_rn(bf, 12582912.0f)))); };
    unsigned nearest = 0u; tot = 0;
#pragma unroll
    for (int w = 0; w < 4; w++) {
        uint32_t big[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float t = __fmul_rn(v[4 * w + k], inv), bf = __fadd_rn(t, 12582912.0f);
            big[k] = __float_as_uint(bf);
            nearest = max(nearest, __float_as_uint(near_of(t, bf)));
        }
        pk[w] = __byte_perm(__byte_perm(big[0], big[1], 0x0040), __byte_perm(big[2], big[3], 0x0040), 0x5410);
        tot = __dp4a((int)pk[w], 0x01010101, tot);
    }
    todo = 0;
    if (!(__uint_as_float(nearest) < lim)) {
#pragma unroll
        for (int i = 0; i < 16; i++) { const float t = __fmul_rn(v[i], inv); todo |= !(near_of(t, __fadd_rn(t, 12582912.0f)) < lim) ? 1u << i : 0u; }
    }
#pragma unroll 1
    for (; __any_sync(0xffffffffu, todo != 0u); todo &= todo - 1u) if (todo) {
        const int i = __ffs(todo) - 1, sh = 8 * (i & 3), wi = i >> 2, qi = __float2int_rn(__fmul_rn(exact(i), inv));
        const uint32_t old = wi & 2 ? (wi & 1 ? pk[3] : pk[2]) : (wi & 1 ? pk[1] : pk[0]), change = ((uint32_t)(qi & 0xFF) << sh) ^ (old & (0xFFu << sh));
        tot += qi - (int)(int8_t)(old >> sh);
        pk[0] ^= wi == 0 ? change : 0u; pk[1] ^= wi == 1 ? change : 0u; pk[2] ^= wi == 2 ? change : 0u; pk[3] ^= wi == 3 ? change : 0u;
    }
    tot = __reduce_add_sync(0xffffffffu, tot);
}
