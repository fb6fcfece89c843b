// k_router_umma.cu -- router logits on the tensor cores for prefill-sized batches (maple.c:870-889 computes them with AVX2
// multiply-adds), plus the selection that makes the result safe to use: sm_100a, tcgen05.mma kind::f16.
//
// logit[b][e] = sum_c W[e][c] hn[b][c], W bf16, hn fp32.  The tensor cores take fp16 operands with fp32 accumulation, so
//   * hn is split into two fp16 terms, hi = fp16(hn), lo = fp16(hn - hi) (the norm kernel writes them, k_route.cu): 22 bits of hn;
//   * W goes to fp16 once per layer: exact for every bf16 value of magnitude >= 2^-17, below that to within 2^-25;
//   * a CTA owns 128 tokens x 256 experts x one eighth of the columns (K = 2 x 256 fp16 values): 32 MMAs of 128 x 256 x 16 into one
//     accumulator of 256 tensor-memory columns.  Short accumulation chains keep the accumulator's own rounding small; the eight
//     partial sums of a token are added in a fixed order by the selection kernel.
// The logits differ from the reference's (its particular order of fp32 roundings) by a few 1e-7 of |W||hn|.  The reference's
// top-8 is reproduced all the same:
//   * router_select_kernel (one warp per token) takes the nine largest logits; if every gap between consecutive ones exceeds
//     ROUTER_GAP * |hn_b| * max_e |W_e| (a bound on both computations' error, with margin), the order of the top nine is the order the
//     reference finds, the eight indices are final and the weights are exp(l_k - l_1) / sum over the eight (equal to the reference's
//     p_k / (sum p + 1e-20) up to rounding: the softmax denominator cancels);
//   * otherwise the token is flagged: router_fix_kernel recomputes its 256 logits in the reference's exact order (eight strided
//     multiply-add chains, then the pairwise adds of maple.c:117-121) and redoes its selection with the exact softmax + top-8
//     (topk.cuh).  Ties, near-ties and all-equal rows therefore take the reference's path bit for bit.
// Indices are the reference's for every token; weights of unflagged tokens agree to ~1e-6 relative.
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include "kernels.h"
#include "launch.cuh"
#include "umma.cuh"
#include "topk.cuh"

extern "C" void k_count_add(long n);

#define HID 2048
#define NEXP 256
#define TOPK 8
#define RU_KS 8                          /* column splits */
#define RU_KCOLS (HID / RU_KS)           /* 256 columns of hn per CTA */
#define RU_KBLK (RU_KCOLS / 64)          /* 4 blocks of 64 columns (128 bytes of fp16) */
#define RU_STAGES 3
#define RU_ABYTES (128 * 128)            /* 128 tokens x 64 fp16 */
#define RU_BBYTES (256 * 128)            /* 256 experts x 64 fp16 */
#define RU_STAGE_BYTES (2 * RU_ABYTES + RU_BBYTES)
#define RU_ROW (NEXP * 4 + 16)
static_assert(128 * RU_ROW <= RU_STAGES * RU_STAGE_BYTES, "the sums of a tile fit the ring");
#define ROUTER_GAP 3.814697265625e-6f     /* 2^-18: the difference between the two computations stayed below 2^-23 |hn| max|W_e| over a million tokens */

// kind::f16: D fp32, A and B fp16, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t idesc_f16(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// router rows bf16 [256][2048] -> fp16 [256][2048]; wnorm[0] = max over experts of the row's Euclidean norm (float bits, atomicMax)
__global__ void __launch_bounds__(256) router_w16_kernel(const uint16_t *__restrict__ W, __half *__restrict__ W16, float *__restrict__ wnorm) {
    __shared__ float sn[8];
    const int e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint4 v = reinterpret_cast<const uint4 *>(W + (size_t)e * HID)[tid];
    const uint32_t ww[4] = {v.x, v.y, v.z, v.w};
    __align__(16) __half o[8]; float n2 = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float f = __uint_as_float((i & 1) ? (ww[i >> 1] & 0xFFFF0000u) : (ww[i >> 1] << 16));
        o[i] = __float2half_rn(f); n2 = fmaf(f, f, n2);
    }
    reinterpret_cast<uint4 *>(W16 + (size_t)e * HID)[tid] = *reinterpret_cast<const uint4 *>(o);
#pragma unroll
    for (int s = 16; s; s >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, s);
    if (lane == 0) sn[wid] = n2;
    __syncthreads();
    if (tid == 0) {
        float t = 0.0f;
        for (int i = 0; i < 8; i++) t += sn[i];
        atomicMax(reinterpret_cast<int *>(wnorm), __float_as_int(sqrtf(t)));      // norms are >= 0: their bit patterns order like the values
    }
}
extern "C" void k_router_w16(cudaStream_t st, const uint16_t *router, void *w16, float *wnorm) {
    cudaMemsetAsync(wnorm, 0, 4, st);
    router_w16_kernel<<<NEXP, 256, 0, st>>>(router, (__half *)w16, wnorm);
    k_count_add(1);
}

struct RuBars { uint64_t full[RU_STAGES], empty[RU_STAGES], acc; uint32_t tmem_base; int abort_flag; };

// grid (RU_KS, token tiles of 128).  Warp 0: TMA (one lane), warp 1: tensor-memory allocation and MMA issue, warps 2-5: epilogue.
// part [RU_KS][ntok_cap][256] fp32 receives the partial sums.
__global__ void __launch_bounds__(192, 1) router_umma_kernel(const __grid_constant__ TMap amap, const __grid_constant__ TMap wmap,
                                                             float *__restrict__ part, int nb, int ntok_cap, int *err, int *__restrict__ nflagged,
                                                             unsigned *__restrict__ mask, int mask_n) {
    extern __shared__ __align__(1024) uint8_t ru_raw[];
    uint8_t *ring = (uint8_t *)(((uintptr_t)ru_raw + 1023) & ~(uintptr_t)1023);
    __shared__ RuBars sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int ks = blockIdx.x, tile = blockIdx.y;
    volatile int *abortp = &sh.abort_flag;
    if (tid == 0) {
        for (int s = 0; s < RU_STAGES; s++) { mbar_init(&sh.full[s], 1); mbar_init(&sh.empty[s], 1); }
        mbar_init(&sh.acc, 1); sh.abort_flag = 0; mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(&sh.tmem_base, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tb = sh.tmem_base;
    pdl_wait(); pdl_trigger();
    if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) *nflagged = 0;      // the selection kernel counts its flagged tokens from zero
    if (mask) {     // and sets the grouping's bits and counters: cleared here, one word per thread
        const int w = (blockIdx.y * gridDim.x + blockIdx.x) * 192 + tid;
        for (int i = w; i < mask_n; i += gridDim.x * gridDim.y * 192) mask[i] = 0u;
    }
    if (warp == 0) {
        if (lane == 0) {
            for (int kb = 0; kb < RU_KBLK; kb++) {
                const int s = kb % RU_STAGES;
                if (!mbar_wait(&sh.empty[s], ((kb / RU_STAGES) & 1) ^ 1, abortp)) break;
                const uint32_t dst = smem_u32(ring + s * RU_STAGE_BYTES);
                const int col = ks * RU_KCOLS + kb * 64;
                mbar_expect_tx(&sh.full[s], RU_STAGE_BYTES);
                tma_load_2d(dst, &amap, col, tile * 128, &sh.full[s]);                       // hi terms of 128 tokens
                tma_load_2d(dst + RU_ABYTES, &amap, HID + col, tile * 128, &sh.full[s]);      // lo terms
                tma_load_2d(dst + 2 * RU_ABYTES, &wmap, col, 0, &sh.full[s]);                 // 256 experts
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc = idesc_f16(NEXP);
        const uint32_t ring0 = __shfl_sync(0xffffffffu, smem_u32(ring), 0);
        bool live = true;
#pragma unroll 1
        for (int kb = 0; kb < RU_KBLK && live; kb++) {
            const int s = kb % RU_STAGES;
            if (!mbar_wait(&sh.full[s], (kb / RU_STAGES) & 1, abortp)) { live = false; break; }
            tc_fence_after();
            const uint64_t ahi = smem_desc_k128(ring0 + s * RU_STAGE_BYTES, 0), alo = smem_desc_k128(ring0 + s * RU_STAGE_BYTES + RU_ABYTES, 0);
            const uint64_t bd = smem_desc_k128(ring0 + s * RU_STAGE_BYTES + 2 * RU_ABYTES, 0);
#pragma unroll
            for (int k = 0; k < 4; k++) {       // 16 fp16 values = 32 bytes per MMA
                if (elect_one()) umma_f16_ss(tb, ahi + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
                if (elect_one()) umma_f16_ss(tb, alo + 2 * k, bd + 2 * k, idesc, 1);
            }
            if (elect_one()) umma_commit(&sh.empty[s]);
        }
        if (live && elect_one()) umma_commit(&sh.acc);
        __syncwarp();
    } else {
        // a warp reaches the tensor-memory lanes 32 (warp % 4) ..: lane = token of the tile, columns = experts
        const int q4 = warp & 3, tok = tile * 128 + q4 * 32 + lane;
        if (mbar_wait(&sh.acc, 0, abortp)) {
            tc_fence_after();
            // Through the ring, which nothing reads any more: a lane puts its token's sums into a row of shared memory (rows 16 bytes apart in their banks) and sends the
            // row off as one copy.  Stored from the registers, 16 bytes to each of 32 rows an
            // instruction, it took 2 us longer (a layer of 512 / 843 / 2048 tokens 95.5 / 105.8 / 156.1 -> 93.8 / 103.9 / 153.5).
            uint8_t *row = ring + (q4 * 32 + lane) * RU_ROW;
#pragma unroll 1
            for (int c = 0; c < NEXP; c += 32) {
                uint32_t v[32];
                tmem_ld32(tb + ((uint32_t)(q4 * 32) << 16) + c, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4 *>(row + (c + j) * 4) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            }
            proxy_fence_async_smem();
            if (tok < nb) bulk_store(part + ((size_t)ks * ntok_cap + tok) * NEXP, smem_u32(row), NEXP * 4);
            bulk_store_wait();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tb, 256);
        if (lane == 0 && sh.abort_flag) *(volatile int *)err = 31;
    }
}

// One warp and CTA per token (2048 tokens 148.9 us per layer; with eight warps per CTA 150.8): lane l holds experts 8l..8l+7.  Adds the eight partial sums (fixed order) and the bias, stores the logits, takes the
// nine largest (lowest index first among equals), decides whether their order is safe, and writes top-8 / weights or flags the token.
__global__ void __launch_bounds__(32) router_select_kernel(const float *__restrict__ part, int ntok_cap, const float *__restrict__ bias,
                                                            const float *__restrict__ hnorm, const float *__restrict__ wnorm,
                                                            float *__restrict__ logits, int *__restrict__ top, float *__restrict__ topw,
                                                            int *__restrict__ flagged, int *__restrict__ nflagged,
                                                            unsigned *__restrict__ mask, int mask_words, int nb) {
    const int lane = threadIdx.x & 31, b = blockIdx.x;
    pdl_wait(); pdl_trigger();
    if (b >= nb) return;
    float l[8];
    {
        float4 p[RU_KS][2];
#pragma unroll
        for (int s = 0; s < RU_KS; s++) {
            const float4 *r = reinterpret_cast<const float4 *>(part + ((size_t)s * ntok_cap + b) * NEXP + lane * 8);
            p[s][0] = r[0]; p[s][1] = r[1];
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float4 a01, a23, a45, a67;
            a01.x = p[0][h].x + p[1][h].x; a01.y = p[0][h].y + p[1][h].y; a01.z = p[0][h].z + p[1][h].z; a01.w = p[0][h].w + p[1][h].w;
            a23.x = p[2][h].x + p[3][h].x; a23.y = p[2][h].y + p[3][h].y; a23.z = p[2][h].z + p[3][h].z; a23.w = p[2][h].w + p[3][h].w;
            a45.x = p[4][h].x + p[5][h].x; a45.y = p[4][h].y + p[5][h].y; a45.z = p[4][h].z + p[5][h].z; a45.w = p[4][h].w + p[5][h].w;
            a67.x = p[6][h].x + p[7][h].x; a67.y = p[6][h].y + p[7][h].y; a67.z = p[6][h].z + p[7][h].z; a67.w = p[6][h].w + p[7][h].w;
            l[4 * h + 0] = (a01.x + a23.x) + (a45.x + a67.x); l[4 * h + 1] = (a01.y + a23.y) + (a45.y + a67.y);
            l[4 * h + 2] = (a01.z + a23.z) + (a45.z + a67.z); l[4 * h + 3] = (a01.w + a23.w) + (a45.w + a67.w);
        }
    }
    if (bias) {
        const float4 b0 = reinterpret_cast<const float4 *>(bias + lane * 8)[0], b1 = reinterpret_cast<const float4 *>(bias + lane * 8)[1];
        l[0] += b0.x; l[1] += b0.y; l[2] += b0.z; l[3] += b0.w; l[4] += b1.x; l[5] += b1.y; l[6] += b1.z; l[7] += b1.w;
    }
    {
        float4 *o = reinterpret_cast<float4 *>(logits + (size_t)b * NEXP + lane * 8);
        o[0] = make_float4(l[0], l[1], l[2], l[3]); o[1] = make_float4(l[4], l[5], l[6], l[7]);
    }
    // order-preserving keys: larger float <-> larger unsigned; 0 marks a taken entry (no finite float maps to 0)
    unsigned key[8];
#pragma unroll
    for (int i = 0; i < 8; i++) { const unsigned u = __float_as_uint(l[i]); key[i] = (u & 0x80000000u) ? ~u : (u | 0x80000000u); if (key[i] == 0u) key[i] = 1u; }
    float sel = 0.0f, gapmin = 3.0e38f, prev = 0.0f; int isel = 0;
#pragma unroll 1
    for (int k = 0; k < TOPK + 1; k++) {
        unsigned lk = key[0];
#pragma unroll
        for (int i = 1; i < 8; i++) lk = max(lk, key[i]);
        const unsigned m = __reduce_max_sync(0xffffffffu, lk);
        const int src = __ffs(__ballot_sync(0xffffffffu, lk == m)) - 1;
        int bi = 7;
#pragma unroll
        for (int i = 6; i >= 0; i--) if (key[i] == m) bi = i;
        const int be = __shfl_sync(0xffffffffu, lane * 8 + bi, src);
#pragma unroll
        for (int i = 0; i < 8; i++) if (lane == src && i == bi) key[i] = 0u;
        const float bv = __uint_as_float((m & 0x80000000u) ? (m & 0x7FFFFFFFu) : ~m);
        if (k > 0) gapmin = fminf(gapmin, prev - bv);
        prev = bv;
        if (lane == k) { sel = bv; isel = be; }
    }
    const float lmax = __shfl_sync(0xffffffffu, sel, 0);
    const float bound = ROUTER_GAP * hnorm[b] * wnorm[0];
    if (!(gapmin > bound)) {                                  // also catches NaN
        if (lane == 0) flagged[atomicAdd(nflagged, 1)] = b;
        return;
    }
    // weights in selection order: e_k / (sum_k e_k + 1e-20), e_k = exp(l_k - l_1)
    const float ek = lane < TOPK ? expf(sel - lmax) : 0.0f;
    float tsum = 0.0f;
#pragma unroll
    for (int k = 0; k < TOPK; k++) tsum += __shfl_sync(0xffffffffu, ek, k);
    if (lane < TOPK) {
        top[b * TOPK + lane] = isel; topw[b * TOPK + lane] = ek / (tsum + 1e-20f);
        if (mask) { atomicOr(&mask[(size_t)(b >> 5) * NEXP + isel], 1u << (b & 31)); atomicAdd(&mask[(size_t)NEXP * mask_words + isel], 1u); }
    }
}

// The flagged tokens over again as the reference computes them (maple.c:870-889, 117-121, 910-923).  grid (8 expert eighths, RF_GROUPS): CTA
// (x, y) walks flagged tokens y, y + RF_GROUPS, ... four at a time and computes 32 experts of each: 256 threads = 8 lanes x 32 experts, the
// eight strided multiply-add chains per expert and their pairwise adds.  A group's eight CTAs are a cluster: CTA t gets the logits of the group's
// token t through distributed shared memory and runs the exact softmax + top-8 on them.
// Bound by latency: list -> token -> hidden row -> 256 chained multiply-adds -> cluster barrier -> softmax + top-8.  So the CTA's 32 router rows come
// into shared memory before it waits for the selection, four tokens' chains run side by side in a thread, and as many clusters as the GPU holds at once (15) cover
// 60 tokens (2% of 2048 are flagged: 45) in one round.  Through memory (rows, fence, a counter that the last CTA finds full) the exchange took 0.8 us more, the softmax's sum in
// front of the selection instead of beside it (two warps) 0.5: 512 / 843 / 2048 tokens 85.7 / 95.8 / 145.4 -> 84.4 / 94.6 / 144.1 us per layer.  All 18 clusters, three of them
// in a second wave: 85.1 / 96.0 / 148.5.  The token numbers asked for beside their count: 0.4 us slower.  A group's chains are as many as it has tokens (one up to 15 flagged, three at 45): every chain costs 1 us of
// shared-memory reads, and all four were always read.  512 tokens 89.1 -> 85.9 us per layer, 843 99.0 -> 95.8, 2048 147.3 -> 145.7.
// WS: the router rows re-laid as [expert][column / 32][lane j][4 steps] bf16 (k_router_pack_small, k_router_tile.cu).
#define RF_GROUPS 18                     /* at most; as many as the GPU holds at once */
#define RF_TOK 4
#define RF_WPITCH (HID * 2 + 64)         /* rows 16 banks apart: the experts of a warp meet no bank twice */
#define RF_SMEM (32 * RF_WPITCH + RF_TOK * HID * 4)
__device__ __forceinline__ void rf_bulk(uint32_t dst_smem, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst_smem), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// the chains of N tokens: hidden rows and weights from shared memory
template <int N>
__device__ __forceinline__ void rf_chains(const uint8_t *wp, const float *hj, float (&acc)[RF_TOK]) {
#pragma unroll 8
    for (int i4 = 0; i4 < 64; i4++) {
        const uint2 a = *reinterpret_cast<const uint2 *>(wp + i4 * 64);
        const float w0 = __uint_as_float(a.x << 16), w1 = __uint_as_float(a.x & 0xFFFF0000u), w2 = __uint_as_float(a.y << 16), w3 = __uint_as_float(a.y & 0xFFFF0000u);
#pragma unroll
        for (int t = 0; t < N; t++) {
            const float *h = hj + t * HID + 32 * i4;
            acc[t] = __fmaf_rn(w0, h[0], acc[t]); acc[t] = __fmaf_rn(w1, h[8], acc[t]); acc[t] = __fmaf_rn(w2, h[16], acc[t]); acc[t] = __fmaf_rn(w3, h[24], acc[t]);
        }
    }
}
__global__ void __launch_bounds__(256) router_fix_kernel(const uint8_t *__restrict__ WS, const float *__restrict__ hn, const float *__restrict__ bias,
                                                         float *__restrict__ logits, int *__restrict__ top, float *__restrict__ topw,
                                                         const int *__restrict__ flagged, const int *__restrict__ nflagged,
                                                         unsigned *__restrict__ mask, int mask_words, int nb, int *err) {
    extern __shared__ __align__(128) uint8_t rf_sm[];
    float *hrow = reinterpret_cast<float *>(rf_sm + 32 * RF_WPITCH);       // [RF_TOK][HID]
    __shared__ unsigned long long tab[32];
    __shared__ __align__(16) float lrow[2][NEXP];                           // logits of the group's token (blockIdx.x), from all eight CTAs; even and odd groups
    __shared__ __align__(16) float erow[NEXP]; __shared__ float s_run;
    __shared__ uint64_t bar; __shared__ int abort_flag;
    const int tid = threadIdx.x, j = tid & 7, pos = tid >> 3, lane = tid & 31, warp = tid >> 5, e = blockIdx.x * 32 + pos;
    if (tid < 32) tab[tid] = DEV_EXP_TAB[tid];
    if (tid == 0) {
        mbar_init(&bar, 1); abort_flag = 0; mbar_init_fence();
        mbar_expect_tx(&bar, 32 * HID * 2);
        for (int r = 0; r < 32; r++) rf_bulk(smem_u32(rf_sm) + r * RF_WPITCH, WS + (size_t)(blockIdx.x * 32 + r) * (HID * 2), HID * 2, &bar);
    }
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const float be = bias ? bias[e] : 0.0f;
    __syncthreads();
    if (!mbar_wait(&bar, 0, &abort_flag) && tid == 0) *(volatile int *)err = 31;
    __syncwarp();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");            // all eight CTAs run
    pdl_wait(); pdl_trigger();
    const int groups = gridDim.y;
    const int total = min(*nflagged, nb);
    int buf = 0;
    for (int f0 = blockIdx.y; f0 < total; f0 += groups * RF_TOK, buf ^= 1) {
        int b[RF_TOK];                                                      // the group's tokens; past the end the first one again, not used
#pragma unroll
        for (int t = 0; t < RF_TOK; t++) { const int f = f0 + t * groups; b[t] = flagged[f < total ? f : f0]; }
        const int n = min((total - f0 + groups - 1) / groups, RF_TOK);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < RF_TOK; t++)
            if (t < n) {
#pragma unroll
                for (int i = 0; i < 2; i++) reinterpret_cast<float4 *>(hrow)[t * (HID / 4) + tid + 256 * i] = reinterpret_cast<const float4 *>(hn + (size_t)b[t] * HID)[tid + 256 * i];
            }
        __syncthreads();
        const uint8_t *wp = rf_sm + pos * RF_WPITCH + j * 8;
        float acc[RF_TOK] = {};
        if (n == 1) rf_chains<1>(wp, hrow + j, acc);
        else if (n == 2) rf_chains<2>(wp, hrow + j, acc);
        else if (n == 3) rf_chains<3>(wp, hrow + j, acc);
        else rf_chains<4>(wp, hrow + j, acc);
#pragma unroll
        for (int t = 0; t < RF_TOK; t++) {
            float l = acc[t];      // (l0+l4)+(l1+l5) then +((l2+l6)+(l3+l7)): the same on every lane of the expert
            l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 4));
            l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 1));
            l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, 2));
            if (j == 0 && t < n) {
                const float lb = bias ? __fadd_rn(l, be) : l;
                logits[(size_t)b[t] * NEXP + e] = lb;
                uint32_t at;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(&lrow[buf][e])), "r"(t));
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(lb) : "memory");
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if ((int)blockIdx.x < n && warp < 2) {
            int bt = b[0];
#pragma unroll
            for (int t = 1; t < RF_TOK; t++) if ((int)blockIdx.x == t) bt = b[t];
            const float4 *lr = reinterpret_cast<const float4 *>(lrow[buf]) + lane * 2;
            const float4 v0 = lr[0], v1 = lr[1];
            float p[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
            int isel; float wsel, tsum;
            exact_topk_pair(p, lane, warp, tab, erow, &s_run, 1, isel, wsel, tsum);
            if (warp == 0 && lane < TOPK) {
                top[bt * TOPK + lane] = isel; topw[bt * TOPK + lane] = __fdiv_rn(wsel, __fadd_rn(tsum, 1e-20f));
                if (mask) { atomicOr(&mask[(size_t)(bt >> 5) * NEXP + isel], 1u << (bt & 31)); atomicAdd(&mask[(size_t)NEXP * mask_words + isel], 1u); }
            }
        }
    }
}

extern "C" void k_router_tensor(cudaStream_t st, const RouterTensorArgs *r) {
    if (r->nb <= 0) return;
    static bool attr_done = false;
    const int smem = RU_STAGES * RU_STAGE_BYTES + 1024;
    static int groups = 0;
    if (!attr_done) {
        cudaFuncSetAttribute(router_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); cudaFuncSetAttribute(router_fix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RF_SMEM);
        groups = clusters_at_once(router_fix_kernel, 8, 256, RF_SMEM, RF_GROUPS); attr_done = true;
    }
    launch_pdl(router_umma_kernel, dim3(RU_KS, (r->nb + 127) / 128), 192, smem, st, r->amap, r->wmap, r->part, r->nb, r->ntok_cap, r->err, r->nflagged, r->mask, NEXP * r->mask_words + NEXP);
    launch_pdl(router_select_kernel, r->nb, 32, 0, st, r->part, r->ntok_cap, r->bias, r->hnorm, r->wnorm, r->logits, r->top, r->topw, r->flagged, r->nflagged, r->mask, r->mask_words, r->nb);
    launch_clusters(router_fix_kernel, dim3(8, groups), 8, 256, RF_SMEM, st, (const uint8_t *)r->router_s, r->hn, r->bias, r->logits, r->top, r->topw, r->flagged, r->nflagged, r->mask, r->mask_words, r->nb, r->err);
    k_count_add(3);
}
