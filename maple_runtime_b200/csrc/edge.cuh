// edge.cuh -- the joint of two layers for one token and 256 threads: the combine of the one (maple.c:834, as combine_kernel) and the RMSNorm + int8 of the next
// (as norm_prep_kernel, its sums in the same order).  Thread tid holds float4 tid and tid + 256 of the row.  The row x of token c goes to xo, hn, q, qs and
// qsum (all with the token's index) unless store is off, and always, in the decode router's layout, to hS (token 0's place there is hS itself).
// pre: edge_pre (not WIRE).  WIRE: the pairs' rows are the tensor-core path's compact ones, as combine_wire_kernel reads them; s_dsp: the experts' down scales in shared memory.
#pragma once
#include <stdint.h>
#include "launch.cuh"
#include "wire.cuh"

struct EdgeWire { uint8_t *wire; int np_cap; const float *const *dsp; };
// What the joint reads that is older than the kernel before it (the grouping's tables; the row x, which the joint before this one wrote): read before the wait for
// that kernel, past L1: 1 token 15.85 -> 15.6 us per layer, 7 26.5 -> 26.05, 13 32.65 -> 32.2, 64 56.7 -> 56.3.  ONE: a single token, whose pairs are 0..7 in order.
// (The joint on compact rows reads them with the rest: the registers they would hold cost it 0.3 to 0.7 us.)
struct EdgePre { int slot[8]; float uv[8]; float4 x[2]; };
template <bool ONE>
__device__ __forceinline__ EdgePre edge_pre(const int c, const float *uw, const int *tp, const float *x) {
    EdgePre e;
#pragma unroll
    for (int k = 0; k < 8; k++) e.slot[k] = ONE ? k : __ldcg(tp + c * 8 + k);
#pragma unroll
    for (int k = 0; k < 8; k++) e.uv[k] = __ldcg(uw + e.slot[k]);
#pragma unroll
    for (int k = 0; k < 2; k++) e.x[k] = __ldcg(reinterpret_cast<const float4 *>(x) + (size_t)c * 512 + threadIdx.x + 256 * k);
    return e;
}
template <bool WIRE>
__device__ __forceinline__ void edge_token(const int c, const float *down, const EdgeWire ew, const float *const *s_dsp, const EdgePre &pre, const float *uw, const int *tp, const float *x, float *xo,
                                           const uint2 (&ln)[2], float *hn, int8_t *q, float *qs, int *qsum, float *hS, const bool store) {
    constexpr int HID = 2048, TOPK = 8;
    __shared__ double s_term[16 * 32];
    __shared__ float s_k, s_mx[8]; __shared__ int s_sum[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int slot[TOPK]; float uv[TOPK];
#pragma unroll
    for (int k = 0; k < TOPK; k++) slot[k] = WIRE ? tp[c * TOPK + k] : pre.slot[k];
#pragma unroll
    for (int k = 0; k < TOPK; k++) uv[k] = WIRE ? uw[slot[k]] : pre.uv[k];
    int4 rec[WIRE ? TOPK : 1];                                          // {scale of the pair's int8 row, expert, escape bits}
    if (WIRE) {
#pragma unroll
        for (int k = 0; k < TOPK; k++) rec[k] = __ldcg(reinterpret_cast<const int4 *>(ew.wire + (size_t)ew.np_cap * WIRE_PITCH + (size_t)slot[k] * WIRE_REC));
    }
    float4 v[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = tid + 256 * k;
        float4 d[TOPK];                                                 // WIRE: the scales
        v[k] = WIRE ? __ldcg(reinterpret_cast<const float4 *>(x) + (size_t)c * 512 + i) : pre.x[k];
        if (WIRE) {
            uint2 raw[TOPK];
#pragma unroll
            for (int t = 0; t < TOPK; t++) raw[t] = __ldcg(reinterpret_cast<const uint2 *>(ew.wire + (size_t)slot[t] * WIRE_PITCH) + i);
#pragma unroll
            for (int t = 0; t < TOPK; t++) { const float *p = s_dsp[rec[t].y & 0xFF]; d[t] = p ? reinterpret_cast<const float4 *>(p)[i] : make_float4(0.f, 0.f, 0.f, 0.f); }
#pragma unroll
            for (int t = 0; t < TOPK; t++) wire_add(v[k], raw[t], uv[t], __int_as_float(rec[t].x), d[t], rec[t].z, warp + 8 * k, lane, ew.wire, ew.np_cap, slot[t]);
        } else {
#pragma unroll
            for (int t = 0; t < TOPK; t++) d[t] = __ldcg(reinterpret_cast<const float4 *>(down) + (size_t)slot[t] * 512 + i);
#pragma unroll
            for (int t = 0; t < TOPK; t++) {
                v[k].x = __fmaf_rn(uv[t], d[t].x, v[k].x); v[k].y = __fmaf_rn(uv[t], d[t].y, v[k].y);
                v[k].z = __fmaf_rn(uv[t], d[t].z, v[k].z); v[k].w = __fmaf_rn(uv[t], d[t].w, v[k].w);
            }
        }
        if (store) reinterpret_cast<float4 *>(xo)[(size_t)c * 512 + i] = v[k];
        s_term[(warp + 8 * k) * 32 + lane] = ((double)v[k].x * (double)v[k].x + (double)v[k].y * (double)v[k].y) + ((double)v[k].z * (double)v[k].z + (double)v[k].w * (double)v[k].w);
    }
    __syncthreads();
    if (WIRE) l2_discard(ew.wire + (size_t)tp[c * TOPK + warp] * WIRE_PITCH + lane * 128);      // the row of pair `warp`: 32 lines, all read (not its escape plane)
    if (warp == 0) {
        double ss = 0.0;
#pragma unroll
        for (int i = 0; i < 16; i++) ss += s_term[i * 32 + lane];
#pragma unroll
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) s_k = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn((float)(ss / (double)HID), 1e-6f)));
    }
    __syncthreads();
    const float kk = s_k;
    float mx = 0.0f;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = tid + 256 * k, col = 4 * i;
        v[k].x = __fmul_rn(__fmul_rn(v[k].x, kk), __uint_as_float(ln[k].x << 16)); v[k].y = __fmul_rn(__fmul_rn(v[k].y, kk), __uint_as_float(ln[k].x & 0xFFFF0000u));
        v[k].z = __fmul_rn(__fmul_rn(v[k].z, kk), __uint_as_float(ln[k].y << 16)); v[k].w = __fmul_rn(__fmul_rn(v[k].w, kk), __uint_as_float(ln[k].y & 0xFFFF0000u));
        mx = fmaxf(fmaxf(mx, fmaxf(fabsf(v[k].x), fabsf(v[k].y))), fmaxf(fabsf(v[k].z), fabsf(v[k].w)));
        if (store) reinterpret_cast<float4 *>(hn)[(size_t)c * 512 + i] = v[k];
        float *p = hS + (col >> 5) * 32 + (col & 7) * 4 + ((col >> 3) & 3);
        p[0] = v[k].x; p[4] = v[k].y; p[8] = v[k].z; p[12] = v[k].w;
    }
    if (!store) return;
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));      // >= 0: the bits order like the values
    if (lane == 0) s_mx[warp] = mx;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++) mx = fmaxf(mx, s_mx[k]);
    const float s = mx > 0.0f ? __fdiv_rn(mx, 127.0f) : 1.0f, inv = __fdiv_rn(1.0f, s);
    int tot = 0;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int q0 = __float2int_rn(__fmul_rn(v[k].x, inv)), q1 = __float2int_rn(__fmul_rn(v[k].y, inv)), q2 = __float2int_rn(__fmul_rn(v[k].z, inv)), q3 = __float2int_rn(__fmul_rn(v[k].w, inv));
        tot += (q0 + q1) + (q2 + q3);
        reinterpret_cast<uint32_t *>(q)[(size_t)c * 512 + tid + 256 * k] = (uint32_t)(q0 & 0xFF) | ((uint32_t)(q1 & 0xFF) << 8) | ((uint32_t)(q2 & 0xFF) << 16) | ((uint32_t)(q3 & 0xFF) << 24);
    }
    tot = __reduce_add_sync(0xffffffffu, tot);
    if (lane == 0) s_sum[warp] = tot;
    __syncthreads();
    if (tid == 0) {
        int t = 0;
        for (int k = 0; k < 8; k++) t += s_sum[k];
        qs[c] = s; qsum[c] = t;
    }
}
