// topk.cuh -- the reference's softmax + top-8 of one token (maple.c:910-923) as a warp-level routine: lane l holds the logits of experts
// 8l..8l+7.  p = expf(l - max); the sum runs over the experts in index order (a chain through the lanes); p /= sum; eight rounds of
// "first strict maximum" (lowest index wins a tie).  Lanes 0..7 return the k-th selected expert and its probability, every lane the sum
// of the eight in selection order: weight_k = wsel / (tsum + 1e-20f).  tab: the expf table of dev_math.cuh (or a shared-memory copy).
// row: 256 floats of shared memory of this warp, 16-byte aligned: every lane walks the chain of additions over all experts from there (a chain
// handed from lane to lane pays a shuffle per eight additions: 1 us instead of 0.6).
#pragma once
#include "dev_math.cuh"

// exponentials of the logits over their maximum
template <typename TabT>
__device__ __forceinline__ void exact_exp_warp(float (&p)[8], const int lane, const TabT *tab) {
    float mx = -1e30f;
#pragma unroll
    for (int i = 0; i < 8; i++) mx = p[i] > mx ? p[i] : mx;
    // (not a NaN) one integer maximum over the warp: the bits of a float order like it once those of the negative ones are turned over
    const int mb = __reduce_max_sync(0xffffffffu, __float_as_int(mx) ^ (__float_as_int(mx) >> 31 & 0x7FFFFFFF));
    mx = __int_as_float(mb ^ (mb >> 31 & 0x7FFFFFFF));
#pragma unroll
    for (int i = 0; i < 8; i++) p[i] = dev_expf_tab(__fsub_rn(p[i], mx), tab);
}
__device__ __forceinline__ float exact_sum_row(const float *row) {
    float run = 0.0f;
#pragma unroll 8
    for (int i = 0; i < 64; i++) {
        const float4 v = reinterpret_cast<const float4 *>(row)[i];
        run = __fadd_rn(run, v.x); run = __fadd_rn(run, v.y); run = __fadd_rn(run, v.z); run = __fadd_rn(run, v.w);
    }
    return run;
}
// N rounds of "first strict maximum" (maple.c:917-921).  Probabilities are >= +0, so their bit patterns order like the
// values: key = bits + 1, a taken entry becomes 0.  One redux.sync gives the warp's maximum, the lowest lane holding it (and
// the lowest of its eight entries) is the first maximum in expert order.  Lane k < N returns the k-th, every lane the sum of all in that order.
template <int N>
__device__ __forceinline__ void top_select_warp(const float (&p)[8], const int lane, int &isel, float &wsel, float &tsum) {
    unsigned key[8];
#pragma unroll
    for (int i = 0; i < 8; i++) key[i] = __float_as_uint(p[i]) + 1u;
    wsel = 0.0f; isel = 0; tsum = 0.0f;
    for (int k = 0; k < N; k++) {
        unsigned lk = key[0];
#pragma unroll
        for (int i = 1; i < 8; i++) lk = max(lk, key[i]);
        const unsigned m = __reduce_max_sync(0xffffffffu, lk);
        const int src = __ffs(__ballot_sync(0xffffffffu, lk == m)) - 1;
        int bi = 7;
#pragma unroll
        for (int i = 6; i >= 0; i--) if (key[i] == m) bi = i;
        const int be = __shfl_sync(0xffffffffu, lane * 8 + bi, src);
        const float bv = __uint_as_float(m - 1u);
#pragma unroll
        for (int i = 0; i < 8; i++) if (lane == src && i == bi) key[i] = 0u;
        tsum = __fadd_rn(tsum, bv);
        if (lane == k) { wsel = bv; isel = be; }
    }
}
// from the exponentials p and their sum
__device__ __forceinline__ void exact_topk_warp_from(float (&p)[8], const int lane, const float run, int &isel, float &wsel, float &tsum) {
#pragma unroll
    for (int i = 0; i < 8; i++) p[i] = __fdiv_rn(p[i], run);
    top_select_warp<8>(p, lane, isel, wsel, tsum);
}
template <typename TabT>
__device__ __forceinline__ void exact_topk_warp(float (&p)[8], const int lane, const TabT *tab, float *row, int &isel, float &wsel, float &tsum) {
    exact_exp_warp(p, lane, tab);
    __syncwarp();
    reinterpret_cast<float4 *>(row)[2 * lane] = make_float4(p[0], p[1], p[2], p[3]);
    reinterpret_cast<float4 *>(row)[2 * lane + 1] = make_float4(p[4], p[5], p[6], p[7]);
    __syncwarp();
    exact_topk_warp_from(p, lane, exact_sum_row(row), isel, wsel, tsum);
}
// The same by two warps that hold the same logits: warp 1 adds the exponentials in the reference's order (256 dependent additions) while warp 0 selects by them;
// warp 0 returns the result.  row, run: shared memory; the two meet at the named barrier `bar`.
template <typename TabT>
__device__ __forceinline__ void exact_topk_pair(float (&p)[8], const int lane, const int sum_warp, const TabT *tab, float *row, float *run_at, const int bar, int &isel, float &wsel, float &tsum) {
    exact_exp_warp(p, lane, tab);
    isel = 0; wsel = tsum = 0.0f;
    if (sum_warp) {
        reinterpret_cast<float4 *>(row)[2 * lane] = make_float4(p[0], p[1], p[2], p[3]); reinterpret_cast<float4 *>(row)[2 * lane + 1] = make_float4(p[4], p[5], p[6], p[7]);
        __syncwarp();
        const float run = exact_sum_row(row);
        if (lane == 0) *run_at = run;
        asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
        return;
    }
    float psel;                                                          // lane k < 9: the k-th largest
    top_select_warp<9>(p, lane, isel, psel, tsum);
    asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
    const float run = *run_at;
    wsel = __fdiv_rn(psel, run);
    // The reference selects by the quotients, which fall with the exponentials: another order only where unequal exponentials have equal quotients (or are not numbers).
    // Among the first nine that shows between neighbours.  Beyond the ninth it needs the ninth's own quotient above it, so the eighth has to be larger than the ninth: where
    // the two are the same exponential, a smaller one with a lower index may have the same quotient.
    const float pn = __shfl_down_sync(0xffffffffu, psel, 1), wn = __shfl_down_sync(0xffffffffu, wsel, 1);
    if (__any_sync(0xffffffffu, lane < 8 && !(wsel > wn || (psel == pn && lane < 7)))) exact_topk_warp_from(p, lane, run, isel, wsel, tsum);
    else {
        tsum = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++) tsum = __fadd_rn(tsum, __shfl_sync(0xffffffffu, wsel, k));
    }
}
