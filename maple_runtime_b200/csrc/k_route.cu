// k_route.cu -- everything of the MoE half that is not a grouped GEMM or the router: RMSNorm + per-token int8,
// softmax + top-8, grouping of pairs by expert, SiLU-output int8, weighted combine.  sm_100a.
//
// Every kernel reproduces the reference's arithmetic operation by operation (order of additions, fused
// multiply-adds where the reference fuses, IEEE division and round-half-even), so its integer outputs are equal
// and its fp32 outputs are the same bits as maple.c's CPU path.  File:line citations are into maple.c.
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include "kernels.h"
#include "launch.cuh"
#include "dev_math.cuh"
#include "topk.cuh"
#include "silu_row.cuh"
#include "wire.cuh"
#include "edge.cuh"

static long g_launches = 0;
extern "C" void k_count_reset(void) { g_launches = 0; }
extern "C" long k_count(void) { return g_launches; }
extern "C" void k_count_add(long n) { g_launches += n; }

#define HID 2048
#define NEXP 256
#define TOPK 8
#define FFN 512

// ------------------------------------------------------------------------------------------------------------
// RMSNorm (maple.c:398-402) + prep (maple.c:184-194), one warp per token: lane l holds columns 128 i + 4 l .. + 3 for i = 0..15 (every
// load and store instruction of the warp covers one contiguous run of the row, all sixteen loads are in flight together, and the three
// reductions are shuffles: no block-wide barrier).  CTAs of one warp spread evenly over the SMs at every size (eight per CTA before: 512 tokens 93.8 -> 92.7 us per layer,
// 843 103.7 -> 103.2, 1300 123.3 -> 121.4, 2048 153.8 -> 153.4; launched programmatically 512 tokens take 96.2).
// w == NULL: x is already normalised (hn = x, not rewritten when hn == x).
// The sum of squares is accumulated in double like the reference; the tree order differs from its left-to-right
// order only below double precision, which the conversion to float absorbs.
// ------------------------------------------------------------------------------------------------------------
// hS != NULL: the normalised row is also stored as the decode router wants it, [column / 32][lane j][4 steps] (k_router_tile.cu).
// hA != NULL: the normalised row is also stored as two fp16 terms, hi = fp16(h) in columns 0..2047 and lo = fp16(h - hi) in columns
// 2048..4095 of a 4096-column row (the tensor-core router's A operand, k_router_umma.cu), and its Euclidean norm goes to hnorm.
__global__ void __launch_bounds__(32) norm_prep_kernel(const float *__restrict__ x, const uint16_t *__restrict__ w,
                                                             float *__restrict__ hn, int8_t *__restrict__ q,
                                                             float *__restrict__ qs, int *__restrict__ qsum, float *__restrict__ hS,
                                                             __half *__restrict__ hA, float *__restrict__ hnorm, int nb,
                                                             const float *__restrict__ bias_src, float *__restrict__ bias) {
    const int lane = threadIdx.x, b = blockIdx.x;
    pdl_wait(); pdl_trigger();
    if (b >= nb) {
        if (bias_src) {
            const float4 *s = reinterpret_cast<const float4 *>(bias_src) + lane; float4 *d = reinterpret_cast<float4 *>(bias) + lane;
            const float4 u = s[0], v = s[32];
            d[0] = u; d[32] = v;
        }
        return;
    }
    const float4 *xr = reinterpret_cast<const float4 *>(x + (size_t)b * HID) + lane;
    float4 v[16];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = xr[32 * i];
    if (w) {
        uint2 wr[16];                                            // 4 bf16 each
#pragma unroll
        for (int i = 0; i < 16; i++) wr[i] = reinterpret_cast<const uint2 *>(w)[32 * i + lane];
        double ss = 0.0;
#pragma unroll
        for (int i = 0; i < 16; i++) ss += (double)v[i].x * (double)v[i].x + (double)v[i].y * (double)v[i].y + ((double)v[i].z * (double)v[i].z + (double)v[i].w * (double)v[i].w);
#pragma unroll
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float k = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn((float)(ss / (double)HID), 1e-6f)));
        float4 *hr = reinterpret_cast<float4 *>(hn + (size_t)b * HID) + lane;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            v[i].x = __fmul_rn(__fmul_rn(v[i].x, k), __uint_as_float(wr[i].x << 16)); v[i].y = __fmul_rn(__fmul_rn(v[i].y, k), __uint_as_float(wr[i].x & 0xFFFF0000u));
            v[i].z = __fmul_rn(__fmul_rn(v[i].z, k), __uint_as_float(wr[i].y << 16)); v[i].w = __fmul_rn(__fmul_rn(v[i].w, k), __uint_as_float(wr[i].y & 0xFFFF0000u));
            hr[32 * i] = v[i];
        }
    } else if (hn != x) {
        float4 *hr = reinterpret_cast<float4 *>(hn + (size_t)b * HID) + lane;
#pragma unroll
        for (int i = 0; i < 16; i++) hr[32 * i] = v[i];
    }
    if (hS) {      // column c goes to (c / 32) * 32 + (c % 8) * 4 + (c / 8) % 4: granule (step / 4, lane j), slot step % 4
        float *d = hS + (size_t)b * HID;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int c = 128 * i + 4 * lane;                    // c % 8 is 0 or 4
            float *p = d + (c >> 5) * 32 + (c & 7) * 4 + ((c >> 3) & 3);
            p[0] = v[i].x; p[4] = v[i].y; p[8] = v[i].z; p[12] = v[i].w;
        }
    }
    float mx = 0.0f, n2 = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; i++) mx = fmaxf(fmaxf(mx, fmaxf(fabsf(v[i].x), fabsf(v[i].y))), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
    if (hA) {
        uint2 *hi_row = reinterpret_cast<uint2 *>(hA + (size_t)b * (2 * HID)) + lane, *lo_row = hi_row + HID / 4;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float f[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            __align__(8) __half hi[4], lo[4];
#pragma unroll
            for (int k = 0; k < 4; k++) { hi[k] = __float2half_rn(f[k]); lo[k] = __float2half_rn(f[k] - __half2float(hi[k])); n2 = fmaf(f[k], f[k], n2); }
            hi_row[32 * i] = *reinterpret_cast<const uint2 *>(hi); lo_row[32 * i] = *reinterpret_cast<const uint2 *>(lo);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, o);
        if (lane == 0) hnorm[b] = sqrtf(n2);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float s = mx > 0.0f ? __fdiv_rn(mx, 127.0f) : 1.0f, inv = __fdiv_rn(1.0f, s);
    int tot = 0;
    uint32_t *qr = reinterpret_cast<uint32_t *>(q + (size_t)b * HID) + lane;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const int q0 = __float2int_rn(__fmul_rn(v[i].x, inv)), q1 = __float2int_rn(__fmul_rn(v[i].y, inv)), q2 = __float2int_rn(__fmul_rn(v[i].z, inv)), q3 = __float2int_rn(__fmul_rn(v[i].w, inv));
        tot += (q0 + q1) + (q2 + q3);
        qr[32 * i] = (uint32_t)(q0 & 0xFF) | ((uint32_t)(q1 & 0xFF) << 8) | ((uint32_t)(q2 & 0xFF) << 16) | ((uint32_t)(q3 & 0xFF) << 24);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0) { qs[b] = s; qsum[b] = tot; }
}
static void norm_launch(cudaStream_t st, const float *x, const uint16_t *w, float *hn, int8_t *q, float *qs, int *qsum, float *hS, __half *hA, float *hnorm, int nb) {
    if (nb <= 0) return;
    if (nb > 256) launch_k(norm_prep_kernel, nb, 32, 0, st, x, w, hn, q, qs, qsum, hS, hA, hnorm, nb, (const float *)NULL, (float *)NULL);
    else launch_pdl(norm_prep_kernel, nb, 32, 0, st, x, w, hn, q, qs, qsum, hS, hA, hnorm, nb, (const float *)NULL, (float *)NULL);
    g_launches++;
}
extern "C" void k_norm_prep(cudaStream_t st, const float *x, const uint16_t *w, float *hn, int8_t *q, float *qs, int *qsum, int nb) {
    norm_launch(st, x, w, hn, q, qs, qsum, (float *)NULL, (__half *)NULL, (float *)NULL, nb);
}
extern "C" void k_norm_prep_relaid(cudaStream_t st, const float *x, const uint16_t *w, float *hn, int8_t *q, float *qs, int *qsum, float *hS, int nb) {
    norm_launch(st, x, w, hn, q, qs, qsum, hS, (__half *)NULL, (float *)NULL, nb);
}
// One more CTA brings the call's bias from the host's page-locked memory: no pageable copy in front of the kernels (24 calls of 1 token 1182 -> 1113 us, 7 1502 -> 1464).
extern "C" void k_norm_prep_call(cudaStream_t st, const float *x, float *hn, int8_t *q, float *qs, int *qsum, float *hS, int nb, const float *bias_src, float *bias) {
    launch_pdl(norm_prep_kernel, nb + (bias_src != NULL), 32, 0, st, x, (const uint16_t *)NULL, hn, q, qs, qsum, hS, (__half *)NULL, (float *)NULL, nb, bias_src, bias);
    g_launches++;
}
extern "C" void k_norm_prep_split(cudaStream_t st, const float *x, const uint16_t *w, float *hn, int8_t *q, float *qs, int *qsum, void *hA, float *hnorm, int nb) {
    norm_launch(st, x, w, hn, q, qs, qsum, (float *)NULL, (__half *)hA, hnorm, nb);
}

// (Router logits live in k_router_tile.cu.)

// ------------------------------------------------------------------------------------------------------------
// Softmax + top-8 (maple.c:910-923): two warps per token (topk.cuh), lane l holds experts 8l..8l+7.
// p = expf(l - max); the sum runs over experts in index order (a chain through the lanes); p /= sum; eight rounds
// of "first strict maximum" (lowest index wins a tie); weights divided by (their sum in selection order + 1e-20f).
// Bound by latency.  Two tokens per CTA while that is one CTA per SM, four above: 65 / 211 / 301 / 400 tokens 58.0 / 76.5 / 80.5 / 83.7 us per layer with a warp per token
// (four per CTA) -> 57.6 / 74.8 / 80.5 / 83.1 with two warps and four tokens, 56.0 / 74.7 / 80.8 / 83.1 with two.
// ------------------------------------------------------------------------------------------------------------
template <int TOKENS>
__global__ void __launch_bounds__(64 * TOKENS, 1) topk_kernel(const float *__restrict__ logits, int *__restrict__ top, float *__restrict__ topw, int nb) {
    __shared__ unsigned long long tab[32];                  // the expf table beside the arithmetic (lane-varying index)
    __shared__ __align__(16) float s_row[TOKENS][NEXP]; __shared__ float s_run[TOKENS];
    if (threadIdx.x < 32) tab[threadIdx.x] = DEV_EXP_TAB[threadIdx.x];
    __syncthreads();
    pdl_wait(); pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int pair = threadIdx.x >> 6, sum_warp = threadIdx.x >> 5 & 1, b = blockIdx.x * TOKENS + pair;
    if (b >= nb) return;
    const float4 *lr = reinterpret_cast<const float4 *>(logits + (size_t)b * NEXP + lane * 8);
    float4 v0 = lr[0], v1 = lr[1];
    float p[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    int isel; float wsel, tsum;
    exact_topk_pair(p, lane, sum_warp, tab, s_row[pair], &s_run[pair], 1 + pair, isel, wsel, tsum);
    if (!sum_warp && lane < TOPK) {
        top[b * TOPK + lane] = isel;
        topw[b * TOPK + lane] = __fdiv_rn(wsel, __fadd_rn(tsum, 1e-20f));
    }
}
extern "C" void k_topk(cudaStream_t st, const float *logits, int *top, float *topw, int nb) {
    if (nb <= 0) return;
    static int sms = 0;
    if (!sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); if (sms < 1) sms = 148; }
    if (nb <= 2 * sms) launch_pdl(topk_kernel<2>, (nb + 1) / 2, 128, 0, st, logits, top, topw, nb);
    else launch_pdl(topk_kernel<4>, (nb + 3) / 4, 256, 0, st, logits, top, topw, nb);
    g_launches++;
}

// ------------------------------------------------------------------------------------------------------------
// Grouping (maple.c:924-938) and tp (maple.c:1018-1019), deterministic without ordered atomics:
//   1. mark:  bit (b % 32) of mask[b / 32][e] is set when token b chose expert e (atomicOr: the result does not depend on order),
//             and the pairs of every expert are counted (integer adds: any order, same sum)
//   2. place: a CTA owns 128 tokens (four mask words).  Thread e scans the counts into the experts' starts (used experts numbered in
//             ascending order: NU, UE, USTART; CTA 0 writes them and the tile lists of the grouped GEMMs) and counts expert e's
//             tokens in front of the CTA's words; then one thread per token: pair slot = start + tokens in front + rank inside the
//             word; UTOK, UW, the slot of every (token, choice), and tp = the token's eight slots sorted ascending (pair index
//             order = expert order)
// ------------------------------------------------------------------------------------------------------------
__global__ void zero_words_kernel(unsigned *__restrict__ p, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = 0u;
}
__global__ void group_mark_kernel(const int *__restrict__ top, unsigned *__restrict__ mask, int mask_words, int np) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    int b = i >> 3, e = top[i];
    atomicOr(&mask[(size_t)(b >> 5) * NEXP + e], 1u << (b & 31));
    atomicAdd(&mask[(size_t)NEXP * mask_words + e], 1u);        // pairs per expert, kept behind the bit words
}
__global__ void __launch_bounds__(NEXP) group_place_kernel(const unsigned *__restrict__ mask, int mask_words, const int *__restrict__ top,
                                                          const float *__restrict__ topw, int *__restrict__ nu_out, int *__restrict__ ue,
                                                          int *__restrict__ estart, int *__restrict__ ustart, int *__restrict__ ecnt,
                                                          MoeTile *__restrict__ ta, int *__restrict__ nta, int tna, MoeTile *__restrict__ tb, int *__restrict__ ntb, int tnb,
                                                          int *__restrict__ utok, float *__restrict__ uw, int *__restrict__ slot, int *__restrict__ uexp,
                                                          int *__restrict__ tp, int nb) {
    __shared__ int w_cnt[8], w_used[8], w_ta[8], w_tb[8];
    __shared__ int s_pre[4][NEXP]; __shared__ unsigned s_word[4][NEXP];
    const int e = threadIdx.x, lane = e & 31, wid = e >> 5;
    const int cnt = (int)mask[(size_t)NEXP * mask_words + e];
    const int used = cnt > 0, na = (cnt + tna - 1) / tna, nb_ = (cnt + tnb - 1) / tnb;
    int c = cnt, u = used, a = na, b = nb_;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int tc = __shfl_up_sync(0xffffffffu, c, o), tu = __shfl_up_sync(0xffffffffu, u, o);
        int t1 = __shfl_up_sync(0xffffffffu, a, o), t2 = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) { c += tc; u += tu; a += t1; b += t2; }
    }
    if (lane == 31) { w_cnt[wid] = c; w_used[wid] = u; w_ta[wid] = a; w_tb[wid] = b; }
    __syncthreads();
    int oc = 0, ou = 0, oa = 0, ob = 0;
    for (int w = 0; w < wid; w++) { oc += w_cnt[w]; ou += w_used[w]; oa += w_ta[w]; ob += w_tb[w]; }
    const int start = oc + c - cnt, uidx = ou + u - used, ta0 = oa + a - na, tb0 = ob + b - nb_;
    if (blockIdx.x == 0) {
        if (ecnt) ecnt[e] = cnt;
        estart[e] = used ? start : -1;
        if (used) {
            ue[uidx] = e; ustart[uidx] = start;
            for (int t = 0; t < na; t++) { MoeTile m = {uidx, start + t * tna, min(tna, cnt - t * tna), e}; ta[ta0 + t] = m; }
            for (int t = 0; t < nb_; t++) { MoeTile m = {uidx, start + t * tnb, min(tnb, cnt - t * tnb), e}; tb[tb0 + t] = m; }
        }
        if (e == NEXP - 1) { const int nu = uidx + used; *nu_out = nu; ustart[nu] = start + cnt; *nta = ta0 + na; *ntb = tb0 + nb_; }
    }
    // expert e's tokens in front of this CTA's four words (coalesced: consecutive threads read consecutive experts of a word)
    const int w0 = blockIdx.x * 4;
    int pre = start;
    for (int w = 0; w < w0; w++) pre += __popc(mask[(size_t)w * NEXP + e]);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const unsigned word = w0 + k < mask_words ? mask[(size_t)(w0 + k) * NEXP + e] : 0u;
        s_pre[k][e] = pre; s_word[k][e] = word; pre += __popc(word);
    }
    __syncthreads();
    if (e >= 128) return;
    const int tok = blockIdx.x * 128 + e;
    if (tok >= nb) return;
    const int wk = e >> 5; const unsigned below = (1u << (e & 31)) - 1u;
    int sl[TOPK];
#pragma unroll
    for (int k = 0; k < TOPK; k++) {
        const int x = top[tok * TOPK + k];
        const int r = s_pre[wk][x] + __popc(s_word[wk][x] & below);
        sl[k] = r; slot[tok * TOPK + k] = r; utok[r] = tok; uw[r] = topw[tok * TOPK + k]; if (uexp) uexp[r] = x;
    }
#pragma unroll
    for (int i = 1; i < TOPK; i++)
#pragma unroll
        for (int k = TOPK - 1; k >= 1; k--) if (k >= i && sl[k] < sl[k - 1]) { int x = sl[k]; sl[k] = sl[k - 1]; sl[k - 1] = x; }
#pragma unroll
    for (int k = 0; k < TOPK; k++) tp[tok * TOPK + k] = sl[k];
}
// Up to 32 tokens: the whole grouping in one CTA, so that the step costs one launch instead of five, and without a
// serial walk: every pair sets its token's bit in its expert's word of a shared-memory table; an expert's
// count is the population of its word, a pair's place inside its expert the population below its token's bit, which is the
// reference's order (pairs of an expert in token order).  The scan over experts and the per-token sort of the eight pair slots
// follow in the same CTA.  (With more words per expert it also took 256 tokens, 7 us longer than the cluster below.)
// TOPK_IN (two to eight tokens): the softmax and top-8 of token w by warp w come first, which saves their kernel.
#define GS_MAXTOK 32
#define GS_TOPK 8
// inclusive sums over the warp's lanes
__device__ __forceinline__ int2 group_scan(int2 v, const int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v.x, o), y = __shfl_up_sync(0xffffffffu, v.y, o);
        if (lane >= o) { v.x += x; v.y += y; }
    }
    return v;
}
// One token: softmax, top-8 and grouping by one warp, beside which a second one adds up the softmax's sum.  A pair's place is its expert's rank among the eight: no scan
// over the experts.  24 layers of one token 17.25 -> 16.35 us each, and with the sum beside the selection 16.1; as a branch of the kernel below it cost that one 0.15 us.
__global__ void __launch_bounds__(64, 1) group_one_kernel(GroupArgs g) {
    __shared__ __align__(16) float s_row[NEXP], s_run;
    __shared__ unsigned long long tab[32];
    const int lane = threadIdx.x & 31, sum_warp = threadIdx.x >> 5;
    if (threadIdx.x < 32) tab[lane] = DEV_EXP_TAB[lane];
    __syncthreads();
    pdl_wait(); pdl_trigger();
    const float4 v0 = __ldcg(reinterpret_cast<const float4 *>(g.logits) + 2 * lane), v1 = __ldcg(reinterpret_cast<const float4 *>(g.logits) + 2 * lane + 1);
    float p[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    int isel; float wsel, tsum;
    exact_topk_pair(p, lane, sum_warp, tab, s_row, &s_run, 1, isel, wsel, tsum);
    if (sum_warp) return;
    const float w = __fdiv_rn(wsel, __fadd_rn(tsum, 1e-20f));          // lane k < 8: the k-th selected expert
    int r = 0, st[8] = {-1, -1, -1, -1, -1, -1, -1, -1};                // st: where the pairs of experts 8 lane .. + 7 start
#pragma unroll
    for (int k = 0; k < TOPK; k++) r += __shfl_sync(0xffffffffu, isel, k) < isel;
    if (lane < TOPK) {
        const MoeTile m = {r, r, 1, isel};
        g.tiles_a[r] = m; g.tiles_b[r] = m; g.ue[r] = isel; g.ustart[r] = r; g.utok[r] = 0; g.uw[r] = w; if (g.uexp) g.uexp[r] = isel;
        g.slot[lane] = r; g.tp[lane] = lane; g.top_out[lane] = isel; g.topw_out[lane] = w;
    }
    if (lane == 0) { *g.nu = TOPK; g.ustart[TOPK] = TOPK; *g.ntiles_a = TOPK; *g.ntiles_b = TOPK; }
#pragma unroll
    for (int k = 0; k < TOPK; k++) {
        const int e = __shfl_sync(0xffffffffu, isel, k), re = __shfl_sync(0xffffffffu, r, k);
#pragma unroll
        for (int i = 0; i < 8; i++) if (e == 8 * lane + i) st[i] = re;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) { g.estart[8 * lane + i] = st[i]; if (g.ecnt) g.ecnt[8 * lane + i] = st[i] >= 0; }
}
template <bool TOPK_IN>
__global__ void __launch_bounds__(NEXP, 1) group_cta_kernel(GroupArgs g) {
    constexpr int NT = NEXP;
    __shared__ unsigned s_mask[NEXP];
    __shared__ int s_slot[GS_MAXTOK * TOPK];
    __shared__ int s_start[NEXP];
    __shared__ int2 w_tot[8];
    __shared__ int s_top[TOPK_IN ? GS_TOPK * TOPK : 1]; __shared__ float s_topw[TOPK_IN ? GS_TOPK * TOPK : 1];
    __shared__ __align__(16) float s_row[TOPK_IN ? 8 : 1][NEXP];
    __shared__ unsigned long long tab[TOPK_IN ? 32 : 1];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nb = g.nb, np = nb * TOPK;
    if (TOPK_IN && tid < 32) tab[tid] = DEV_EXP_TAB[tid];
    s_mask[tid] = 0u;
    __syncthreads();
    pdl_wait(); pdl_trigger();
    if (TOPK_IN) {
        if (wid < nb) {
            const int t = wid;
            const float4 *lr = reinterpret_cast<const float4 *>(g.logits + (size_t)t * NEXP + lane * 8);
            const float4 v0 = __ldcg(lr), v1 = __ldcg(lr + 1);
            float p[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
            int isel; float wsel, tsum;
            exact_topk_warp(p, lane, tab, s_row[wid], isel, wsel, tsum);
            if (lane < TOPK) {
                const float w = __fdiv_rn(wsel, __fadd_rn(tsum, 1e-20f));
                s_top[t * TOPK + lane] = isel; s_topw[t * TOPK + lane] = w;
                g.top_out[t * TOPK + lane] = isel; g.topw_out[t * TOPK + lane] = w;
            }
        }
        __syncthreads();
    }
    auto expert = [&](const int i) { return TOPK_IN ? s_top[i] : g.top[i]; };
    for (int i = tid; i < np; i += NT) { const int t = i >> 3; atomicOr(&s_mask[expert(i)], 1u << t); }
    __syncthreads();
    {
        const int e = tid, cnt = __popc(s_mask[e]);
        const int used = cnt > 0, na = (cnt + g.tn_a - 1) / g.tn_a, nb_ = (cnt + g.tn_b - 1) / g.tn_b;
        int2 v = make_int2(cnt | used << 16, na | nb_ << 16);             // two sums in a word: at most 256 pairs, experts and tiles
        v = group_scan(v, lane);
        if (lane == 31) w_tot[wid] = v;
        __syncthreads();
        for (int w = 0; w < wid; w++) { v.x += w_tot[w].x; v.y += w_tot[w].y; }
        const int start = (v.x & 0xFFFF) - cnt, uidx = (v.x >> 16) - used, ta0 = (v.y & 0xFFFF) - na, tb0 = (v.y >> 16) - nb_;
        s_start[e] = start;
        if (g.ecnt) g.ecnt[e] = cnt;
        g.estart[e] = used ? start : -1;
        if (used) {
            g.ue[uidx] = e; g.ustart[uidx] = start;
            for (int t = 0; t < na; t++) { MoeTile m = {uidx, start + t * g.tn_a, min(g.tn_a, cnt - t * g.tn_a), e}; g.tiles_a[ta0 + t] = m; }
            for (int t = 0; t < nb_; t++) { MoeTile m = {uidx, start + t * g.tn_b, min(g.tn_b, cnt - t * g.tn_b), e}; g.tiles_b[tb0 + t] = m; }
        }
        if (e == NEXP - 1) { const int nu = uidx + used; *g.nu = nu; g.ustart[nu] = start + cnt; *g.ntiles_a = ta0 + na; *g.ntiles_b = tb0 + nb_; }
    }
    __syncthreads();
    for (int i = tid; i < np; i += NT) {                             // every pair finds its place
        const int x = expert(i), t = i >> 3, r = s_start[x] + __popc(s_mask[x] & ((1u << t) - 1u));
        s_slot[i] = r;
        g.utok[r] = t; g.uw[r] = TOPK_IN ? s_topw[i] : g.topw[i]; if (g.uexp) g.uexp[r] = x;
    }
    __syncthreads();
    for (int t = tid; t < nb; t += NT) {                         // tp: the token's eight slots ascending
        int sl[TOPK];
#pragma unroll
        for (int k = 0; k < TOPK; k++) { sl[k] = s_slot[t * TOPK + k]; g.slot[t * TOPK + k] = sl[k]; }
#pragma unroll
        for (int i = 1; i < TOPK; i++)
#pragma unroll
            for (int k = TOPK - 1; k >= 1; k--) if (k >= i && sl[k] < sl[k - 1]) { int x = sl[k]; sl[k] = sl[k - 1]; sl[k - 1] = x; }
#pragma unroll
        for (int k = 0; k < TOPK; k++) g.tp[t * TOPK + k] = sl[k];
    }
}
// Up to GROUP_CLUSTER_MAX tokens: one launch of one cluster of CTAS CTAs.  CTA r owns its share of the tokens (in whole
// words of 32) and keeps their bits in its shared memory; the counts are exchanged through distributed shared memory, after which every CTA
// scans the experts for itself and its threads place one token each.  Bound by latency: what counts is the number of launches (a launch costs
// the host 3.9 us; clearing, marking and placing as three kernels took 16.4 us per call at 1000 tokens, 10.2 us like this) and of trips through
// global memory (inside a layer of 2048 tokens, against the router setting the bits and the place kernel reading them: 4 us less).  Eight
// CTAs are what every GPU has to allow; from 513 tokens on sixteen share the scattered stores (2048 tokens: 14.4 -> 11.9 us).
// Against one CTA for up to 256 tokens, a layer of the stack: 96 tokens 70.8 -> 70.0 us, 128 77.7 -> 75.9, 256 106.1 -> 100.7.
// (One CTA per SM in the launch bounds of the grouping kernels: registers instead of reloads, 0.1 us.)
// TOPK_IN (9 to TOPK_IN_MAX tokens): the softmax and top-8 come first, two warps per token (20 tokens 41.8 -> 41.3 us; with two warps instead of one 9 / 13 / 32 tokens
// 28.4 / 32.4 / 44.45 -> 28.0 / 32.0 / 44.25).  Above, with one warp per token here or two in a kernel of their own: 33 / 40 / 48 / 64 tokens 47.3 / 50.2 / 52.15 / 56.1 and
// 46.8 / 49.6 / 52.2 / 55.5; from nine tokens on in their own: 9 / 13 28.9 / 32.1.
// GC_CARVE: the split of the SM's memory, in percent of the shared memory it can have: 132 KB, the smallest that holds a CTA of the router in front of it (RS_ALONE, k_router_tile.cu).  Left
// to the driver (or asked for 32, 64 or 100 KB) 9 / 11 tokens take 28.65 / 30.3 us per layer, with 132 KB 27.85 / 30.05, with all of it 28.2 / 30.1 but 16 / 20 34.8 / 40.9 instead of
// 33.6 / 37.5.
#define GC_CARVE 57
#define GC_WORDS 8
template <int GC_CTAS, bool TOPK_IN>
__global__ void __launch_bounds__(NEXP, 1) group_cluster_kernel(GroupArgs g) {
    __shared__ unsigned s_mask[NEXP][GC_WORDS + 1];           // + 1: a warp's 32 experts of one word lie in 32 banks
    __shared__ unsigned short s_pre[NEXP][GC_WORDS + 1];      // the pairs of the CTA's expert in front of word w
    __shared__ int s_cnt[NEXP], s_start[NEXP];
    __shared__ int2 w_tot[8];
    const int e = threadIdx.x, lane = e & 31, wid = e >> 5, nb = g.nb;
    const int per = TOPK_IN ? (nb + GC_CTAS - 1) / GC_CTAS : (((nb + 31) / 32 + GC_CTAS - 1) / GC_CTAS) * 32, tok = blockIdx.x * per + e;      // per <= 32 GC_WORDS = one token per thread
    const bool mine = e < per && tok < nb;
    constexpr int TT = TOPK_IN ? TOPK_IN_MAX / GC_CTAS : 1;
    static_assert(2 * TT <= 8, "two warps per token");
    __shared__ __align__(16) int s_top[TT * TOPK]; __shared__ __align__(16) float s_topw[TT * TOPK];
    __shared__ __align__(16) float s_row[TT][NEXP]; __shared__ float s_run[TT];
    __shared__ unsigned long long tab[TOPK_IN ? 32 : 1];
    if (TOPK_IN && e < 32) tab[e] = DEV_EXP_TAB[e];
    if (TOPK_IN) __syncthreads();
    pdl_wait(); pdl_trigger();
    if (TOPK_IN) {
        const int i = wid >> 1, t = blockIdx.x * per + i;
        if (i < per && t < nb) {
            const float4 *lr = reinterpret_cast<const float4 *>(g.logits + (size_t)t * NEXP + lane * 8);
            const float4 v0 = __ldcg(lr), v1 = __ldcg(lr + 1);
            float p[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
            int isel; float wsel, tsum;
            exact_topk_pair(p, lane, wid & 1, tab, s_row[i], &s_run[i], 1 + i, isel, wsel, tsum);
            if (!(wid & 1) && lane < TOPK) {
                const float tw = __fdiv_rn(wsel, __fadd_rn(tsum, 1e-20f));
                s_top[i * TOPK + lane] = isel; s_topw[i * TOPK + lane] = tw;
                g.top_out[t * TOPK + lane] = isel; g.topw_out[t * TOPK + lane] = tw;
            }
        }
        __syncthreads();
    }
    const bool wide = (((uintptr_t)g.top | (uintptr_t)g.topw | (uintptr_t)g.tp | (uintptr_t)g.slot) & 15) == 0;      // the caller's arrays may lie anywhere
    int x[TOPK]; float w[TOPK];
    if (mine) {
        const int *tr = TOPK_IN ? s_top + e * TOPK : g.top + (size_t)tok * TOPK; const float *wr = TOPK_IN ? s_topw + e * TOPK : g.topw + (size_t)tok * TOPK;
        if (TOPK_IN || wide) {
            const int4 a = reinterpret_cast<const int4 *>(tr)[0], b = reinterpret_cast<const int4 *>(tr)[1];
            const float4 c = reinterpret_cast<const float4 *>(wr)[0], d = reinterpret_cast<const float4 *>(wr)[1];
            x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
            w[0] = c.x; w[1] = c.y; w[2] = c.z; w[3] = c.w; w[4] = d.x; w[5] = d.y; w[6] = d.z; w[7] = d.w;
        } else {
#pragma unroll
            for (int k = 0; k < TOPK; k++) { x[k] = tr[k]; w[k] = wr[k]; }
        }
    }
#pragma unroll
    for (int k = 0; k <= GC_WORDS; k++) (&s_mask[0][0])[e + k * NEXP] = 0u;
    __syncthreads();
    if (mine)
#pragma unroll
        for (int k = 0; k < TOPK; k++) atomicOr(&s_mask[x[k]][wid], 1u << lane);
    __syncthreads();
    int own = 0;
#pragma unroll
    for (int k = 0; k < GC_WORDS; k++) { s_pre[e][k] = (unsigned short)own; own += __popc(s_mask[e][k]); }
    s_cnt[e] = own;
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    int cnt = 0, before = 0;
#pragma unroll
    for (int r = 0; r < GC_CTAS; r++) {
        uint32_t at; int v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&s_cnt[e])), "r"(r));
        asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
        cnt += v; if (r < (int)blockIdx.x) before += v;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // this CTA has read the others' counts
    const int used = cnt > 0, na = (cnt + g.tn_a - 1) / g.tn_a, nt = (cnt + g.tn_b - 1) / g.tn_b;
    int2 v = make_int2(cnt | used << 16, na | nt << 16);                  // two sums in a word: at most 32,768 pairs and tiles
    v = group_scan(v, lane);
    if (lane == 31) w_tot[wid] = v;
    __syncthreads();
    for (int k = 0; k < wid; k++) { v.x += w_tot[k].x; v.y += w_tot[k].y; }
    const int start = (v.x & 0xFFFF) - cnt, uidx = (v.x >> 16) - used, ta0 = (v.y & 0xFFFF) - na, tb0 = (v.y >> 16) - nt;
    s_start[e] = start + before;
    if (!TOPK_IN && g.place_base) {                            // the pairs are placed by the kernel that moves the rows: it gets, for every word, where the experts' pairs of it start
        const int w0 = blockIdx.x * (per >> 5);
#pragma unroll
        for (int k = 0; k < GC_WORDS; k++) if (k < per >> 5 && (w0 + k) * 32 < nb) { g.place_base[(w0 + k) * NEXP + e] = start + before + s_pre[e][k]; g.place_bits[(w0 + k) * NEXP + e] = s_mask[e][k]; }
    }
    __syncthreads();
    if (mine && (TOPK_IN || !g.place_base)) {
        int sl[TOPK];
#pragma unroll
        for (int k = 0; k < TOPK; k++) sl[k] = s_start[x[k]] + s_pre[x[k]][wid] + __popc(s_mask[x[k]][wid] & ((1u << lane) - 1u));
#pragma unroll
        for (int k = 0; k < TOPK; k++) { g.utok[sl[k]] = tok; g.uw[sl[k]] = w[k]; if (g.uexp) g.uexp[sl[k]] = x[k]; }
        int *sp = g.slot + (size_t)tok * TOPK, *tq = g.tp + (size_t)tok * TOPK;
        if (wide) { reinterpret_cast<int4 *>(sp)[0] = make_int4(sl[0], sl[1], sl[2], sl[3]); reinterpret_cast<int4 *>(sp)[1] = make_int4(sl[4], sl[5], sl[6], sl[7]); }
        else {
#pragma unroll
            for (int k = 0; k < TOPK; k++) sp[k] = sl[k];
        }
#pragma unroll
        for (int i = 1; i < TOPK; i++)
#pragma unroll
            for (int k = TOPK - 1; k >= 1; k--) if (k >= i && sl[k] < sl[k - 1]) { const int t = sl[k]; sl[k] = sl[k - 1]; sl[k - 1] = t; }
        if (wide) { reinterpret_cast<int4 *>(tq)[0] = make_int4(sl[0], sl[1], sl[2], sl[3]); reinterpret_cast<int4 *>(tq)[1] = make_int4(sl[4], sl[5], sl[6], sl[7]); }
        else {
#pragma unroll
            for (int k = 0; k < TOPK; k++) tq[k] = sl[k];
        }
    }
    if (blockIdx.x == GC_CTAS - 1) {                           // the CTA with the fewest tokens writes the experts' tables
        if (g.ecnt) g.ecnt[e] = cnt;
        g.estart[e] = used ? start : -1;
        if (used) {
            g.ue[uidx] = e; g.ustart[uidx] = start;
            for (int t = 0; t < na; t++) { const MoeTile m = {uidx, start + t * g.tn_a, min(g.tn_a, cnt - t * g.tn_a), e}; g.tiles_a[ta0 + t] = m; }
            for (int t = 0; t < nt; t++) { const MoeTile m = {uidx, start + t * g.tn_b, min(g.tn_b, cnt - t * g.tn_b), e}; g.tiles_b[tb0 + t] = m; }
        }
        if (e == NEXP - 1) { const int nu = uidx + used; *g.nu = nu; g.ustart[nu] = start + cnt; *g.ntiles_a = ta0 + na; *g.ntiles_b = tb0 + nt; }
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");        // the others have read this CTA's counts: it may go
}
extern "C" void k_group(cudaStream_t st, const GroupArgs *g) {
    if (g->nb <= 0) return;
    if (g->nb <= (g->logits ? GS_TOPK : GS_MAXTOK)) {
        if (g->logits && g->nb == 1) launch_pdl(group_one_kernel, 1, 64, 0, st, *g);
        else if (g->logits) launch_pdl(group_cta_kernel<true>, 1, NEXP, 0, st, *g); else launch_pdl(group_cta_kernel<false>, 1, NEXP, 0, st, *g);
        g_launches++; return;
    }
    const int np = g->nb * TOPK;
    if (g->nb <= GROUP_CLUSTER_MAX) {
        if (g->logits) {
            static bool split_done = false;
            if (!split_done) { cudaFuncSetAttribute(group_cluster_kernel<8, true>, cudaFuncAttributePreferredSharedMemoryCarveout, GC_CARVE); split_done = true; }
            launch_cluster(group_cluster_kernel<8, true>, 8, NEXP, st, *g);
        } else if (g->nb <= 512) launch_cluster(group_cluster_kernel<8, false>, 8, NEXP, st, *g);
        else {
            static bool attr_done = false;
            if (!attr_done) { cudaFuncSetAttribute(group_cluster_kernel<16, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1); attr_done = true; }
            launch_cluster(group_cluster_kernel<16, false>, 16, NEXP, st, *g);
        }
        g_launches++; return;
    }
    if (!g->marked) {
        const int zw = NEXP * g->mask_words + NEXP;                                           // bit words + the 256 counters behind them
        launch_k(zero_words_kernel, (zw + 1023) / 1024, 1024, 0, st, g->mask, zw);
        launch_k(group_mark_kernel, (np + 255) / 256, 256, 0, st, g->top, g->mask, g->mask_words, np);
        g_launches += 2;
    }
    launch_k(group_place_kernel, (g->nb + 127) / 128, NEXP, 0, st, g->mask, g->mask_words, g->top, g->topw, g->nu, g->ue, g->estart, g->ustart, g->ecnt,
                                                            g->tiles_a, g->ntiles_a, g->tn_a, g->tiles_b, g->ntiles_b, g->tn_b,
                                                            g->utok, g->uw, g->slot, g->uexp, g->tp, g->nb);
    g_launches += 1;
}

// ------------------------------------------------------------------------------------------------------------
// SiLU-output int8 (the prep call of maple.c:831 on 512 values): one warp per pair, 16 values per lane.
// ------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) actq_kernel(const float *__restrict__ act, int8_t *__restrict__ aq, float *__restrict__ aqs,
                                                   int *__restrict__ aqsum, int np, const int *__restrict__ np_dev) {
    if (np_dev) np = min(np, *np_dev);
    const int lane = threadIdx.x & 31, a = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (a >= np) return;
    const float4 *r = reinterpret_cast<const float4 *>(act + (size_t)a * FFN) + lane * 4;
    float v[16];
#pragma unroll
    for (int i = 0; i < 4; i++) { float4 t = r[i]; v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w; }
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; i++) mx = fmaxf(mx, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float s = mx > 0.0f ? __fdiv_rn(mx, 127.0f) : 1.0f, inv = __fdiv_rn(1.0f, s);
    int tot = 0; uint32_t pk[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 16; i++) { int qi = __float2int_rn(__fmul_rn(v[i], inv)); tot += qi; pk[i >> 2] |= (uint32_t)(qi & 0xFF) << (8 * (i & 3)); }
    reinterpret_cast<uint4 *>(aq + (size_t)a * FFN)[lane] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
#pragma unroll
    for (int o = 16; o; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0) { aqs[a] = s; aqsum[a] = tot; }
}
extern "C" void k_actq(cudaStream_t st, const float *act, int8_t *aq, float *aqs, int *aqsum, const int *np_dev, int np_max) {
    if (np_max <= 0) return;
    launch_k(actq_kernel, (np_max + 7) / 8, 256, 0, st, act, aq, aqs, aqsum, np_max, np_dev); g_launches++;
}

// ------------------------------------------------------------------------------------------------------------
// SiLU*up + int8 in one pass (maple.c:825-832) for the tensor-core path, whose GEMM stores gate and up: one warp per pair (silu_row.cuh).  The results are
// the reference's bits, as those of the kernel below that evaluates every element exactly.
// Bound by instruction issue (800 per pair at first, 60% of the slots used) beside 75 MB per 2048 tokens: the bytes of a row are cut out of the rounding sums with
// byte permutes and added with dp4a, and the distance to a rounding boundary is one running maximum per lane that is taken apart only where it is near.  CTAs of two warps
// instead of eight, so that an SM takes new rows as each pair of warps ends: between events 22.1 -> 20.1 us at 2048 tokens, 14.3 -> 12.5 at 843.
// Launched programmatically up to 1536 tokens: 511 tokens 96.4 -> 96.0 us per layer, 843 106.3 -> 105.7, 1300 125.8 -> 125.1, 2048 the same, 3000 222.2 -> 224.7.
// (Two rows per warp, whose exact evaluations share a pass, at 122 registers: 24.6.  Rows brought ahead into shared memory by resident warps, 24 per SM: 21.3.)
// ------------------------------------------------------------------------------------------------------------
#define SQ_EARLY (1536 * TOPK)
__global__ void __launch_bounds__(64, 16) silu_quant_kernel(const float *__restrict__ gate, const float *__restrict__ up,
                                                         int8_t *__restrict__ aq, float *__restrict__ aqs, int *__restrict__ aqsum, int np, const int *__restrict__ np_dev, int drop) {
    __shared__ unsigned long long tab[32];
    if (threadIdx.x < 32) tab[threadIdx.x] = DEV_EXP_TAB[threadIdx.x];
    __syncthreads();
    pdl_wait(); pdl_trigger();
    if (np_dev) np = min(np, *np_dev);
    const int lane = threadIdx.x & 31, a = blockIdx.x * 2 + (threadIdx.x >> 5);
    if (a >= np) return;
    float s; int tot; uint32_t pk[4];
    silu_quant_row(gate + (size_t)a * FFN, up + (size_t)a * FFN, tab, lane, pk, s, tot);
#pragma unroll
    for (int i = 0; i < 4; i++) reinterpret_cast<uint32_t *>(aq + (size_t)a * FFN)[32 * i + lane] = pk[i];
    if (lane == 0) { aqs[a] = s; aqsum[a] = tot; }
    if (drop) { __syncwarp(); l2_discard((lane < 16 ? gate : up) + (size_t)a * FFN + (lane & 15) * 32); }
}
// Every element evaluated exactly with the libm-equal expf in double (dev_math.cuh), and the fp32 activations stored (stage comparisons).
__global__ void __launch_bounds__(256, 4) silu_quant_exact_kernel(const float *__restrict__ gate, const float *__restrict__ up, float *__restrict__ act,
                                                         int8_t *__restrict__ aq, float *__restrict__ aqs, int *__restrict__ aqsum, int np, const int *__restrict__ np_dev) {
    __shared__ unsigned long long tab[32];
    if (threadIdx.x < 32) tab[threadIdx.x] = DEV_EXP_TAB[threadIdx.x];
    __syncthreads();
    if (np_dev) np = min(np, *np_dev);
    const int lane = threadIdx.x & 31, a = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (a >= np) return;
    const float4 *gr = reinterpret_cast<const float4 *>(gate + (size_t)a * FFN) + lane, *ur = reinterpret_cast<const float4 *>(up + (size_t)a * FFN) + lane;
    float4 *o = reinterpret_cast<float4 *>(act + (size_t)a * FFN) + lane;
    float v[16], mx = 0.0f; int tot = 0; uint32_t pk[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float4 g = gr[32 * i], u = ur[32 * i];
        v[4 * i] = dev_silu_mul_tab(g.x, u.x, tab); v[4 * i + 1] = dev_silu_mul_tab(g.y, u.y, tab); v[4 * i + 2] = dev_silu_mul_tab(g.z, u.z, tab); v[4 * i + 3] = dev_silu_mul_tab(g.w, u.w, tab);
        o[32 * i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
#pragma unroll
    for (int i = 0; i < 16; i++) mx = fmaxf(mx, fabsf(v[i]));
#pragma unroll
    for (int i = 16; i; i >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, i));
    const float s = mx > 0.0f ? __fdiv_rn(mx, 127.0f) : 1.0f, inv = __fdiv_rn(1.0f, s);
#pragma unroll
    for (int i = 0; i < 16; i++) { const int qi = __float2int_rn(__fmul_rn(v[i], inv)); tot += qi; pk[i >> 2] |= (uint32_t)(qi & 0xFF) << (8 * (i & 3)); }
#pragma unroll
    for (int i = 16; i; i >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, i);
#pragma unroll
    for (int i = 0; i < 4; i++) reinterpret_cast<uint32_t *>(aq + (size_t)a * FFN)[32 * i + lane] = pk[i];
    if (lane == 0) { aqs[a] = s; aqsum[a] = tot; }
}
extern "C" void k_silu_quant(cudaStream_t st, const float *gate, const float *up, float *act, int8_t *aq, float *aqs, int *aqsum, int np, const int *np_dev, int drop) {
    if (np <= 0) return;
    if (act) launch_k(silu_quant_exact_kernel, (np + 7) / 8, 256, 0, st, gate, up, act, aq, aqs, aqsum, np, np_dev);
    else if (np <= SQ_EARLY) launch_pdl(silu_quant_kernel, (np + 1) / 2, 64, 0, st, gate, up, aq, aqs, aqsum, np, np_dev, drop);
    else launch_k(silu_quant_kernel, (np + 1) / 2, 64, 0, st, gate, up, aq, aqs, aqsum, np, np_dev, drop);
    g_launches++;
}

// ------------------------------------------------------------------------------------------------------------
// Decode batches, between two layers: the combine of the one (maple.c:834, as combine_kernel) and the RMSNorm + int8 of the next (as
// norm_prep_kernel, its sums in the same order) for one token per CTA: one launch and one trip of the hidden row less.  Thread tid holds float4
// tid and tid + 256 of the row.
// WIRE: the pairs' rows are the tensor-core path's compact ones, as combine_wire_kernel reads them.  The experts' scales come from L2 for every pair (12 KB a
// pair with its row) instead of once per CTA: a layer of the stack 98.9 -> 96.4 us at 301 tokens, 110.2 -> 108.0 at 511, but 123.0 -> 124.5 at 600.
// (512 threads: 99.1 at 301; launched programmatically 96.7.)
// PER_SM (WIRE): two CTAs fit an SM at 128 registers, three at 80 with a few spilled.  The latter where it saves the second wave, 297 to 444 tokens: 301 tokens
// 86.9 -> 85.6 us per layer, 400 88.8 -> 87.0; elsewhere it costs 0.8 to 1.7.
// (fp32 rows): told that one CTA per SM is enough, the compiler keeps all loads of the joint in flight: 13 tokens 35.2 -> 33.9 us per layer, 64 60.6 -> 59.2.
// ------------------------------------------------------------------------------------------------------------
template <bool WIRE, int PER_SM>
__global__ void __launch_bounds__(256, PER_SM) edge_kernel(const float *down, const EdgeWire ew, const float *uw, const int *tp, float *x, const uint16_t *__restrict__ w,
                                                   float *hn, int8_t *q, float *qs, int *qsum, float *hS) {
    __shared__ const float *s_dsp[WIRE ? NEXP : 1];
    const int tid = threadIdx.x, c = blockIdx.x;
    const uint2 ln[2] = {reinterpret_cast<const uint2 *>(w)[tid], reinterpret_cast<const uint2 *>(w)[tid + 256]};      // weights: read before the wait
    if (WIRE) { static_assert(NEXP == 256, "one entry per thread"); s_dsp[tid] = ew.dsp[tid]; __syncthreads(); }
    EdgePre pre;
    if (!WIRE) pre = edge_pre<false>(c, uw, tp, x);
    pdl_wait(); pdl_trigger();
    edge_token<WIRE>(c, down, ew, s_dsp, pre, uw, tp, x, x, ln, hn, q, qs, qsum, hS + (size_t)c * HID, true);
}
extern "C" void k_edge(cudaStream_t st, const float *down, const float *uw, const int *tp, float *x, const uint16_t *w, float *hn, int8_t *q, float *qs, int *qsum, float *hS, int nb) {
    if (nb <= 0) return;
    launch_pdl(edge_kernel<false, 1>, nb, 256, 0, st, down, EdgeWire{NULL, 0, NULL}, uw, tp, x, w, hn, q, qs, qsum, hS); g_launches++;
}
extern "C" void k_edge_wire(cudaStream_t st, uint8_t *wire, int np_cap, const float *const *dsp, const float *uw, const int *tp, float *x, const uint16_t *w, float *hn, int8_t *q, float *qs, int *qsum, float *hS, int nb) {
    if (nb <= 0) return;
    static int sms = 0;
    if (!sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
    if (nb > 2 * sms && nb <= 3 * sms) launch_k(edge_kernel<true, 3>, nb, 256, 0, st, (const float *)NULL, EdgeWire{wire, np_cap, dsp}, uw, tp, x, w, hn, q, qs, qsum, hS);
    else launch_k(edge_kernel<true, 2>, nb, 256, 0, st, (const float *)NULL, EdgeWire{wire, np_cap, dsp}, uw, tp, x, w, hn, q, qs, qsum, hS);
    g_launches++;
}

// ------------------------------------------------------------------------------------------------------------
// Combine (maple.c:834): out[b] = init[b] (or 0) then, for the token's pairs in ascending pair order,
// out = fma(w, down, out) -- the order and the fused rounding of the reference's compiled loop.
// ------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 1) combine_kernel(const float *__restrict__ down, const float *__restrict__ uw, const int *__restrict__ tp,
                                                      const float *__restrict__ init, float *__restrict__ out, int nb) {
    const int i = blockIdx.x * 256 + threadIdx.x, b = i >> 9, c = (i & 511) * 4;
    // the tables and the rows to add to are older than the down kernel: read before the wait for it, past L1
    int a[TOPK]; float w[TOPK]; float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (b < nb) {
#pragma unroll
        for (int k = 0; k < TOPK; k++) a[k] = __ldcg(tp + b * TOPK + k);
#pragma unroll
        for (int k = 0; k < TOPK; k++) w[k] = __ldcg(uw + a[k]);
        if (init) acc = __ldcg(reinterpret_cast<const float4 *>(init + (size_t)b * HID + c));
    }
    pdl_wait(); pdl_trigger();
    if (b >= nb) return;
    float4 d[TOPK];
#pragma unroll
    for (int k = 0; k < TOPK; k++) d[k] = *reinterpret_cast<const float4 *>(down + (size_t)a[k] * HID + c);
#pragma unroll
    for (int k = 0; k < TOPK; k++) {
        acc.x = __fmaf_rn(w[k], d[k].x, acc.x); acc.y = __fmaf_rn(w[k], d[k].y, acc.y); acc.z = __fmaf_rn(w[k], d[k].z, acc.z); acc.w = __fmaf_rn(w[k], d[k].w, acc.w);
    }
    *reinterpret_cast<float4 *>(out + (size_t)b * HID + c) = acc;
}
extern "C" void k_combine(cudaStream_t st, const float *down, const float *uw, const int *tp, const float *init, float *out, int nb) {
    if (nb <= 0) return;
    launch_pdl(combine_kernel, (nb * 512 + 255) / 256, 256, 0, st, down, uw, tp, init, out, nb); g_launches++;
}
