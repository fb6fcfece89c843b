// k_router_tile.cu -- router logits for prefill-sized batches (maple.c:870-889 job_route_multi), sm_100a.
//
// logit[b][e] = hsum over eight lanes of ( sum_i W[e][8i+l] * hn[b][8i+l] ), each lane one chain of fused multiply-adds in
// increasing i, the lanes added as ((l0+l4)+(l1+l5))+((l2+l6)+(l3+l7)) (maple.c:117-121): the same bits as the CPU path.
//
// A CTA owns up to 32 tokens x 128 experts.  Eight warps hold 8 lanes x 32 positions; a position is an
// 8-token (fewer when that fills the SMs better) x 16-expert register tile, so one step of a lane costs 64 bytes of shared-memory reads (eight fp32 hidden values,
// sixteen bf16 weights) for 128 multiply-adds: half a byte per multiply-add, half of what the load path delivers at the full
// multiply-add rate.  The multiply-adds are issued two at a time (fma.rn.f32x2, each half an IEEE fused multiply-add).
// Both operands come from copies laid out for exactly this access: per 128-column chunk and 8-token (16-expert) group,
// [step i][half h][lane j][4 tokens fp32 | 8 experts bf16], so that the eight lanes of a position read 128 consecutive bytes and a
// chunk of a CTA's operands is one contiguous block.  Thread 0 streams those blocks through a four-stage ring with
// cp.async.bulk and mbarriers; every wait is bounded.
#include <cuda_runtime.h>
#include <stdint.h>
#include "kernels.h"
#include "launch.cuh"
#include "umma.cuh"
#include "edge.cuh"

#define HID 2048
#define NEXP 256
#define RP_TOK 32
#define RP_EXP 128
#define RP_KI 16                          /* steps of 8 columns per chunk */
#define RP_NCH (HID / 8 / RP_KI)          /* 16 chunks */
#define RP_GRP (RP_KI * 256)              /* bytes of one group (8 tokens or 16 experts) in one chunk */
#define RP_HB ((RP_TOK / 8) * RP_GRP)     /* 16 KB */
#define RP_WB ((RP_EXP / 16) * RP_GRP)    /* 32 KB */
#define RP_STAGES 4
#define RP_SMEM (RP_STAGES * (RP_HB + RP_WB))

extern "C" void k_count_add(long n);

// router rows (bf16 [256][2048]) -> [expert block of 128][chunk][group of 16][i][h][j][8 experts]; once per layer
__global__ void __launch_bounds__(256) router_pack_w_kernel(const uint16_t *__restrict__ W, uint4 *__restrict__ WT) {
    const int o = blockIdx.x * 256 + threadIdx.x;
    const int j = o & 7, h = (o >> 3) & 1, i = (o >> 4) & 15, eg = (o >> 8) & 7, ch = (o >> 11) & 15, eb = o >> 15;
    const int e = eb * RP_EXP + eg * 16 + h * 8, col = (ch * RP_KI + i) * 8 + j;
    uint32_t v[4];
#pragma unroll
    for (int m = 0; m < 4; m++)
        v[m] = (uint32_t)W[(size_t)(e + 2 * m) * HID + col] | ((uint32_t)W[(size_t)(e + 2 * m + 1) * HID + col] << 16);
    WT[o] = make_uint4(v[0], v[1], v[2], v[3]);
}
// normalised hidden rows (fp32 [nb][2048]) -> [tile of 4*tt tokens][chunk][group of tt tokens in 8 slots][i][h][j][4 slots];
// slots past tt and rows past nb read as zero
__global__ void __launch_bounds__(256) router_pack_h_kernel(const float *__restrict__ hn, float4 *__restrict__ hT, int nb, int tt) {
    const int o = blockIdx.x * 256 + threadIdx.x;
    const int j = o & 7, h = (o >> 3) & 1, i = (o >> 4) & 15, tg = (o >> 8) & 3, ch = (o >> 10) & 15, tile = o >> 14;
    const int t0 = tile * 4 * tt + tg * tt, col = (ch * RP_KI + i) * 8 + j;
    float v[4];
#pragma unroll
    for (int m = 0; m < 4; m++) v[m] = (h * 4 + m < tt && t0 + h * 4 + m < nb) ? hn[(size_t)(t0 + h * 4 + m) * HID + col] : 0.0f;
    hT[o] = make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void bulk_load(uint32_t dst_smem, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst_smem), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint64_t pair64(uint32_t lo, uint32_t hi) {
    uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi)); return r;
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

struct RpBars { uint64_t full[RP_STAGES], empty[RP_STAGES]; int abort; };

template <int TT>
__global__ void __maxnreg__(224) router_tile_kernel(const uint8_t *__restrict__ WT, const uint8_t *__restrict__ hT,
                                                            const float *__restrict__ bias, float *__restrict__ logits, int nb, int *err) {
    extern __shared__ __align__(128) uint8_t rp_ring[];
    __shared__ RpBars sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.y, eb = blockIdx.x;
    if (tid == 0) {
        for (int s = 0; s < RP_STAGES; s++) { mbar_init(&sh.full[s], 1); mbar_init(&sh.empty[s], 8); }
        sh.abort = 0;
        mbar_init_fence();
    }
    __syncthreads();
    volatile int *abortp = &sh.abort;
    {
        // thread 0 is also the producer: it fills the ring before the arithmetic starts and, at the top of every chunk, refills
        // the stage that all eight warps released one chunk earlier
        const uint8_t *hsrc = hT + (size_t)tile * RP_NCH * RP_HB, *wsrc = WT + (size_t)eb * RP_NCH * RP_WB;
        auto issue = [&](int ch) {
            const int s = ch % RP_STAGES;
            const uint32_t dst = smem_u32(rp_ring) + s * (RP_HB + RP_WB);
            mbar_expect_tx(&sh.full[s], RP_HB + RP_WB);
            bulk_load(dst, hsrc + (size_t)ch * RP_HB, RP_HB, &sh.full[s]);
            bulk_load(dst + RP_HB, wsrc + (size_t)ch * RP_WB, RP_WB, &sh.full[s]);
        };
        if (tid == 0) for (int ch = 0; ch < RP_STAGES - 1; ch++) issue(ch);
        const int j = tid & 7, tg = (tid >> 3) & 3, eg = warp;      // the four positions of a warp share their sixteen experts
        uint64_t acc[TT][8];                                          // [token][expert pair], halves = experts 2m, 2m+1
#pragma unroll
        for (int a = 0; a < TT; a++)
#pragma unroll
            for (int m = 0; m < 8; m++) acc[a][m] = 0ull;
        bool live = true;
        for (int ch = 0; ch < RP_NCH && live; ch++) {
            const int s = ch % RP_STAGES, n = ch / RP_STAGES;
            if (tid == 0 && ch + RP_STAGES - 1 < RP_NCH) {
                // a wait that ran out has raised the abort flag: nothing is issued and every warp leaves at its next wait
                if (ch == 0 || mbar_wait(&sh.empty[(ch - 1) % RP_STAGES], ((ch - 1) / RP_STAGES) & 1, abortp)) issue(ch + RP_STAGES - 1);
            }
            if (!mbar_wait(&sh.full[s], n & 1, abortp)) { live = false; break; }
            const uint8_t *hp = rp_ring + s * (RP_HB + RP_WB) + tg * RP_GRP + j * 16;
            const uint8_t *wp = rp_ring + s * (RP_HB + RP_WB) + RP_HB + eg * RP_GRP + j * 16;
#pragma unroll 4
            for (int i = 0; i < RP_KI; i++) {
                const float4 h0 = *reinterpret_cast<const float4 *>(hp + i * 256), h1 = *reinterpret_cast<const float4 *>(hp + i * 256 + 128);
                const uint4 w0 = *reinterpret_cast<const uint4 *>(wp + i * 256), w1 = *reinterpret_cast<const uint4 *>(wp + i * 256 + 128);
                const uint32_t wu[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
                const float hv[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                uint64_t wv[8], hh[8];
#pragma unroll
                for (int m = 0; m < 8; m++) wv[m] = pair64(wu[m] << 16, wu[m] & 0xFFFF0000u);
#pragma unroll
                for (int a = 0; a < TT; a++) hh[a] = pair64(__float_as_uint(hv[a]), __float_as_uint(hv[a]));
#pragma unroll
                for (int a = 0; a < TT; a++)
#pragma unroll
                    for (int m = 0; m < 8; m++) fma2(acc[a][m], wv[m], hh[a]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.empty[s]);
        }
        if (live) {
            // every lane ends with the full sums (the additions commute pairwise); lane j stores token j's sixteen logits
            const int e0 = eb * RP_EXP + eg * 16, b0 = tile * 4 * TT + tg * TT;
            float bv[16];
#pragma unroll
            for (int c = 0; c < 16; c++) bv[c] = bias ? bias[e0 + c] : 0.0f;
#pragma unroll
            for (int a = 0; a < TT; a++) {
                float l[16];
#pragma unroll
                for (int m = 0; m < 8; m++) { l[2 * m] = __uint_as_float((uint32_t)acc[a][m]); l[2 * m + 1] = __uint_as_float((uint32_t)(acc[a][m] >> 32)); }
#pragma unroll
                for (int c = 0; c < 16; c++) {
                    float v = l[c];
                    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
                    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
                    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
                    l[c] = bias ? __fadd_rn(v, bv[c]) : v;
                }
                if (a == j && b0 + a < nb) {
                    float4 *dst = reinterpret_cast<float4 *>(logits + (size_t)(b0 + a) * NEXP + e0);
                    dst[0] = make_float4(l[0], l[1], l[2], l[3]); dst[1] = make_float4(l[4], l[5], l[6], l[7]);
                    dst[2] = make_float4(l[8], l[9], l[10], l[11]); dst[3] = make_float4(l[12], l[13], l[14], l[15]);
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0 && sh.abort) *(volatile int *)err = 31;      // a wait ran out: the host reports it and the logits are not to be used
}

extern "C" void k_router_pack(cudaStream_t st, const uint16_t *router, void *router_t) {
    router_pack_w_kernel<<<NEXP * HID / 8 / 256, 256, 0, st>>>(router, (uint4 *)router_t);
    k_count_add(1);
}
static int g_force_tt = 0;
// pins the tokens per thread (4..8; 0 = choose by batch size); include/gmoe.h
extern "C" void gmoe_router_tile_tokens(int tt) { g_force_tt = (tt >= 4 && tt <= 8) ? tt : 0; }
template <int TT>
static void launch_tile(cudaStream_t st, const void *router_t, const float *hn, void *hT, const float *bias, float *logits, int nb, int *err) {
    static bool attr_done = false;
    if (!attr_done) { cudaFuncSetAttribute(router_tile_kernel<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, RP_SMEM); attr_done = true; }
    const int tiles = (nb + 4 * TT - 1) / (4 * TT);
    launch_k(router_pack_h_kernel, tiles * 64, 256, 0, st, hn, (float4 *)hT, nb, TT);
    launch_k(router_tile_kernel<TT>, dim3(NEXP / RP_EXP, tiles), 256, RP_SMEM, st, (const uint8_t *)router_t, (const uint8_t *)hT, bias, logits, nb, err);
}
// A thread's tile is tt tokens x 16 experts, a CTA's 4*tt tokens x 128 experts; tt in 4..8 is chosen so that the CTAs fill whole
// waves of the SMs with the least arithmetic per wave (2048 tokens: tt = 7, 148 CTAs).  hT must hold ceil(nb/16) * 256 KB.
extern "C" void k_router_logits_tile(cudaStream_t st, const void *router_t, const float *hn, void *hT, const float *bias, float *logits, int nb, int *err) {
    if (nb <= 0) return;
    static int sms = 0;
    if (!sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); if (sms < 1) sms = 148; }
    int best = 8; long cost = -1;
    for (int tt = 8; tt >= 4 && !g_force_tt; tt--) {
        const long ctas = 2L * ((nb + 4 * tt - 1) / (4 * tt)), c = ((ctas + sms - 1) / sms) * (tt * 8 + 5);   /* 5: the per-step cost that does not shrink with tt */
        if (cost < 0 || c < cost) { cost = c; best = tt; }
    }
    if (g_force_tt) best = g_force_tt;
    switch (best) {
    case 4: launch_tile<4>(st, router_t, hn, hT, bias, logits, nb, err); break;
    case 5: launch_tile<5>(st, router_t, hn, hT, bias, logits, nb, err); break;
    case 6: launch_tile<6>(st, router_t, hn, hT, bias, logits, nb, err); break;
    case 7: launch_tile<7>(st, router_t, hn, hT, bias, logits, nb, err); break;
    default: launch_tile<8>(st, router_t, hn, hT, bias, logits, nb, err); break;
    }
    k_count_add(2);
}

// ---------------------------------------------------------------------------------------------------------------------
// Decode batches (up to 148 tokens on 148 SMs).  The arithmetic is a handful of microseconds of dependent multiply-adds (256 per chain), so
// the kernel is about latency: a CTA owns 8 tokens x 8 experts, fetches all 2048 columns of both in two bulk copies (64 KB of
// hidden values, 32 KB of bf16 weights, both pre-laid as [column / 32][lane j][4 steps] so that the eight lanes of a position
// read consecutive 16-byte (8-byte) pieces), waits once, and runs the 64 x 4 steps without another synchronisation.  Two CTAs
// share an SM, so the 256 CTAs of a 64-token batch are one wave.  256 threads = 8 lanes x 32 positions (8 tokens x 4 expert pairs).
// ---------------------------------------------------------------------------------------------------------------------
#define RS_TOK 8
#define RS_EXP 8
#define RS_HB (RS_TOK * HID * 4)
#define RS_WB (RS_EXP * HID * 2)
#define RS_ALONE (120 << 10)              /* shared memory that leaves no room for a second CTA on the SM */
// router rows (bf16 [256][2048]) -> [expert][i4 = column / 32][lane j][4 steps]; once per layer
__global__ void __launch_bounds__(256) router_pack_w_small_kernel(const uint16_t *__restrict__ W, uint2 *__restrict__ WS) {
    const int o = blockIdx.x * 256 + threadIdx.x, j = o & 7, i4 = (o >> 3) & 63, e = o >> 9;
    uint16_t v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = W[(size_t)e * HID + (4 * i4 + k) * 8 + j];
    WS[o] = make_uint2((uint32_t)v[0] | ((uint32_t)v[1] << 16), (uint32_t)v[2] | ((uint32_t)v[3] << 16));
}
// hidden rows (fp32 [nb][2048]) -> [token][i4][lane j][4 steps]
__global__ void __launch_bounds__(256) router_pack_h_small_kernel(const float *__restrict__ hn, float4 *__restrict__ hS, int nb) {
    const int o = blockIdx.x * 256 + threadIdx.x, j = o & 7, i4 = (o >> 3) & 63, b = o >> 9;
    if (b >= nb) return;
    const float *r = hn + (size_t)b * HID + 32 * i4 + j;
    hS[o] = make_float4(r[0], r[8], r[16], r[24]);
}
// STEP: the order of the reference's single-token decode (bf_row, maple.c:146-157, called at maple.c:609): per lane two chains, one over
// columns 16m + j and one over 16m + 8 + j, added before the lanes are; otherwise one chain per lane (job_route_small/multi).
// EDGE (one token, between layers): every CTA first does the joint of the two layers for itself (edge.cuh; 64 KB of down rows out of L2), the first one
// also stores what it gives; the row goes into shared memory.  One kernel less in the chain: 24 layers 500 -> 459 us.  From two tokens on repeating the joint in
// every CTA costs more than the launch (2: 548 -> 561, 4: 600 -> 715).
struct RouterEdge { const float *down, *uw; const int *tp; const float *x; float *xo; const uint16_t *w; float *hn; int8_t *q; float *qs; int *qsum; };
template <bool STEP, bool EDGE>
__global__ void __launch_bounds__(256, 2) router_small_kernel(const uint8_t *__restrict__ WS, const uint8_t *__restrict__ hS, const float *__restrict__ bias,
                                                             float *__restrict__ logits, int nb, int *err, const RouterEdge ed) {
    extern __shared__ __align__(128) uint8_t rs_sm[];                  // hidden 64 KB, then weights 32 KB
    __shared__ uint64_t bar; __shared__ int abort_flag;
    const int tid = threadIdx.x, j = tid & 7, pos = tid >> 3, tok = pos & 7, ep = pos >> 3;
    const int b0 = blockIdx.y * RS_TOK, e0 = blockIdx.x * RS_EXP, ntok = min(RS_TOK, nb - b0);
    if (tid == 0) { mbar_init(&bar, 1); abort_flag = 0; mbar_init_fence(); }
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(&bar, (uint32_t)((EDGE ? 0 : ntok * HID * 4) + RS_WB));
        bulk_load(smem_u32(rs_sm + RS_HB), WS + (size_t)e0 * HID * 2, RS_WB, &bar);      // the layer's weights: no kernel of the layer loop writes them
        if (!EDGE) {
            pdl_wait();
            bulk_load(smem_u32(rs_sm), hS + (size_t)b0 * HID * 4, (uint32_t)(ntok * HID * 4), &bar);
        }
    }
    if (EDGE) {
        const uint2 ln[2] = {reinterpret_cast<const uint2 *>(ed.w)[tid], reinterpret_cast<const uint2 *>(ed.w)[tid + 256]};
        const EdgePre pre = edge_pre<true>(0, ed.uw, nullptr, ed.x);
        pdl_wait(); pdl_trigger();
        edge_token<false>(0, ed.down, EdgeWire{}, nullptr, pre, ed.uw, ed.tp, ed.x, ed.xo, ln, ed.hn, ed.q, ed.qs, ed.qsum, reinterpret_cast<float *>(rs_sm), blockIdx.x == 0);
        __syncthreads();
    } else { pdl_wait(); pdl_trigger(); }
    const bool ok = mbar_wait(&bar, 0, &abort_flag);
    float acc0 = 0.0f, acc1 = 0.0f, odd0 = 0.0f, odd1 = 0.0f;       // odd0/odd1: the second chain of the step order (columns 16m + 8 + j)
    if (ok && tok < ntok) {
        const uint8_t *hp = rs_sm + tok * (HID * 4) + j * 16;
        const uint8_t *w0p = rs_sm + RS_HB + (2 * ep) * (HID * 2) + j * 8, *w1p = w0p + HID * 2;
#pragma unroll 8
        for (int i4 = 0; i4 < 64; i4++) {
            const float4 h = *reinterpret_cast<const float4 *>(hp + i4 * 128);
            const uint2 a = *reinterpret_cast<const uint2 *>(w0p + i4 * 64), b = *reinterpret_cast<const uint2 *>(w1p + i4 * 64);
            acc0 = __fmaf_rn(__uint_as_float(a.x << 16), h.x, acc0); acc1 = __fmaf_rn(__uint_as_float(b.x << 16), h.x, acc1);
            if (STEP) { odd0 = __fmaf_rn(__uint_as_float(a.x & 0xFFFF0000u), h.y, odd0); odd1 = __fmaf_rn(__uint_as_float(b.x & 0xFFFF0000u), h.y, odd1); }
            else { acc0 = __fmaf_rn(__uint_as_float(a.x & 0xFFFF0000u), h.y, acc0); acc1 = __fmaf_rn(__uint_as_float(b.x & 0xFFFF0000u), h.y, acc1); }
            acc0 = __fmaf_rn(__uint_as_float(a.y << 16), h.z, acc0); acc1 = __fmaf_rn(__uint_as_float(b.y << 16), h.z, acc1);
            if (STEP) { odd0 = __fmaf_rn(__uint_as_float(a.y & 0xFFFF0000u), h.w, odd0); odd1 = __fmaf_rn(__uint_as_float(b.y & 0xFFFF0000u), h.w, odd1); }
            else { acc0 = __fmaf_rn(__uint_as_float(a.y & 0xFFFF0000u), h.w, acc0); acc1 = __fmaf_rn(__uint_as_float(b.y & 0xFFFF0000u), h.w, acc1); }
        }
        if (STEP) { acc0 = __fadd_rn(acc0, odd0); acc1 = __fadd_rn(acc1, odd1); }
    }
    // the eight lanes of a position sit in one warp: (l0+l4)+(l1+l5) then +(l2+l6)+(l3+l7), the same on every lane
    float l0 = acc0, l1 = acc1;
    l0 = __fadd_rn(l0, __shfl_xor_sync(0xffffffffu, l0, 4)); l1 = __fadd_rn(l1, __shfl_xor_sync(0xffffffffu, l1, 4));
    l0 = __fadd_rn(l0, __shfl_xor_sync(0xffffffffu, l0, 1)); l1 = __fadd_rn(l1, __shfl_xor_sync(0xffffffffu, l1, 1));
    l0 = __fadd_rn(l0, __shfl_xor_sync(0xffffffffu, l0, 2)); l1 = __fadd_rn(l1, __shfl_xor_sync(0xffffffffu, l1, 2));
    if (ok && j == 0 && tok < ntok) {
        const int e = e0 + 2 * ep;
        float *dst = logits + (size_t)(b0 + tok) * NEXP + e;
        dst[0] = bias ? __fadd_rn(l0, bias[e]) : l0; dst[1] = bias ? __fadd_rn(l1, bias[e + 1]) : l1;
    }
    if (tid == 0 && !ok) *(volatile int *)err = 31;
}
// ---------------------------------------------------------------------------------------------------------------------
// A few hundred tokens.  The kernel above runs one wave per 74 of them (a multiply-add costs it three quarters of a shared-memory read and an unpacking);
// the prefill kernel's CTAs are too few to fill the SMs, its one warp per scheduler issues every 2.5 cycles, and it wants its rows copied once more.  Here a
// warp is 8 lanes x 4 positions of TT tokens x 8 experts, small enough for two warps per scheduler at 300 tokens; a CTA is four of them on the same 4 TT
// tokens and 32 experts, and a fifth that fills a ring of two stages of 256 columns (three: 0.4 to 0.9 us slower, 511 tokens 1.2).  Rows and weights are read as they
// lie: rows in the decode layout that the norm left, weights in the tile layout.  Kernel above -> here, per layer of the stack: 160 tokens 84.8 -> 83.1, 256 108.2 -> 105.6,
// 301 103.3 -> 98.7, 416 112.5 -> 104.9 us.  With the tokens per CTA chosen by the SMs they fill (below), 12 or 16 before: 230 tokens 82.8 -> 79.5, 296 84.8 -> 80.4,
// 301 87.5 -> 86.9, 400 92.2 -> 88.8, 511 97.6 -> 96.4.  (TT = 4 with 16 experts per position, two warps per CTA: 103 at 301, 107 at 400.  CTAs of 16 experts: 85 to 86 at 230
// to 256 with TT = 4, 83 with 3, level with 32 experts for TT = 2.)
// ---------------------------------------------------------------------------------------------------------------------
#define RM_COLS 256
#define RM_NCH (HID / RM_COLS)
#define RM_ROW (RM_COLS * 4)
#define RM_WB (2 * 2 * RP_GRP)            /* two chunks of the tile layout x two groups of 16 experts */
#define RM_STAGES 2
template <int TT>
__device__ __forceinline__ void router_mid_cta(const uint8_t *__restrict__ WT, const uint8_t *__restrict__ hS, const float *__restrict__ bias,
                                               float *__restrict__ logits, int nb, int *err, const int tok0) {
    extern __shared__ __align__(128) uint8_t rm_ring[];
    __shared__ uint64_t full[RM_STAGES], empty[RM_STAGES]; __shared__ int abort_flag, late;
    constexpr int HB = 4 * TT * RM_ROW, STAGE = HB + RM_WB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, j = lane & 7, tg = lane >> 3;
    const int g0 = blockIdx.x * 2;                                         // first group of 16 experts
    if (tid == 0) {
        for (int s = 0; s < RM_STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 4); }
        abort_flag = late = 0; mbar_init_fence();
    }
    __syncthreads();
    if (warp == 4) {                                                       // lane 0 copies the weights, lane t row t of the tile (a row past the end is the last one again)
        auto issue_w = [&](int ch) {
            const int s = ch % RM_STAGES;
            mbar_expect_tx(&full[s], STAGE);
            const uint8_t *w = WT + (size_t)(g0 / 8) * RP_NCH * RP_WB + (g0 % 8) * RP_GRP;
            for (int h = 0; h < 2; h++) bulk_load(smem_u32(rm_ring) + s * STAGE + HB + h * 2 * RP_GRP, w + (size_t)(2 * ch + h) * RP_WB, 2 * RP_GRP, &full[s]);
        };
        auto issue_h = [&](int ch) {
            const int s = ch % RM_STAGES;
            bulk_load(smem_u32(rm_ring) + s * STAGE + lane * RM_ROW, hS + (size_t)min(tok0 + lane, nb - 1) * HID * 4 + ch * RM_ROW, RM_ROW, &full[s]);
        };
        if (lane == 0) for (int ch = 0; ch < RM_STAGES; ch++) issue_w(ch);   // the layer's weights: no kernel of the layer loop writes them
        __syncwarp();
        pdl_wait(); pdl_trigger();
        if (lane < 4 * TT) for (int ch = 0; ch < RM_STAGES; ch++) issue_h(ch);
        int ch = RM_STAGES;
        for (; ch < RM_NCH; ch++) {
            const bool go = mbar_wait(&empty[ch % RM_STAGES], (ch / RM_STAGES - 1) & 1, &abort_flag);
            if (!__all_sync(0xffffffffu, go)) break;
            if (lane == 0) issue_w(ch);
            __syncwarp();
            if (lane < 4 * TT) issue_h(ch);
        }
        // after a wait that ran out the copies still in flight land first (again with a limit)
        if (ch < RM_NCH && lane == 0) for (int c = ch - RM_STAGES; c < ch; c++) mbar_wait(&full[c % RM_STAGES], (c / RM_STAGES) & 1, &late);
    } else {
        pdl_wait(); pdl_trigger();
        uint64_t acc[TT][4];                                               // [token][expert pair], halves = experts 2m, 2m+1
#pragma unroll
        for (int a = 0; a < TT; a++)
#pragma unroll
            for (int m = 0; m < 4; m++) acc[a][m] = 0ull;
        bool live = true;
        for (int ch = 0; ch < RM_NCH; ch++) {
            const int s = ch % RM_STAGES;
            if (!mbar_wait(&full[s], (ch / RM_STAGES) & 1, &abort_flag)) live = false;
            live = __all_sync(0xffffffffu, live);
            if (!live) break;
            const uint8_t *hp = rm_ring + s * STAGE + tg * TT * RM_ROW + j * 16, *wp = rm_ring + s * STAGE + HB + (warp >> 1) * RP_GRP + (warp & 1) * 128 + j * 16;
            // a step's weights are read one step ahead, its rows four (the last read of a chunk wraps to its start and goes unused)
            float4 hv[TT], hn4[TT];
#pragma unroll
            for (int a = 0; a < TT; a++) hn4[a] = *reinterpret_cast<const float4 *>(hp + a * RM_ROW);
            uint4 n0 = *reinterpret_cast<const uint4 *>(wp);
#pragma unroll 2
            for (int i4 = 0; i4 < RM_COLS / 32; i4++) {
#pragma unroll
                for (int a = 0; a < TT; a++) { hv[a] = hn4[a]; hn4[a] = *reinterpret_cast<const float4 *>(hp + a * RM_ROW + (i4 + 1) % 8 * 128); }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t wu[4] = {n0.x, n0.y, n0.z, n0.w};
                    const int t = (4 * i4 + k + 1) % 32;
                    n0 = *reinterpret_cast<const uint4 *>(wp + (t >> 4) * 2 * RP_GRP + (t & 15) * 256);
                    uint64_t wv[4];
#pragma unroll
                    for (int m = 0; m < 4; m++) wv[m] = pair64(wu[m] << 16, wu[m] & 0xFFFF0000u);
#pragma unroll
                    for (int a = 0; a < TT; a++) {
                        const float h = k == 0 ? hv[a].x : k == 1 ? hv[a].y : k == 2 ? hv[a].z : hv[a].w;
                        const uint64_t hh = pair64(__float_as_uint(h), __float_as_uint(h));
#pragma unroll
                        for (int m = 0; m < 4; m++) fma2(acc[a][m], wv[m], hh);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        }
        if (live) {
            const int e0 = (g0 + (warp >> 1)) * 16 + (warp & 1) * 8, b0 = tok0 + tg * TT;
#pragma unroll
            for (int a = 0; a < TT; a++) {
                float l[8];
#pragma unroll
                for (int m = 0; m < 4; m++) { l[2 * m] = __uint_as_float((uint32_t)acc[a][m]); l[2 * m + 1] = __uint_as_float((uint32_t)(acc[a][m] >> 32)); }
                float p = 0.0f;                                            // every lane gets all eight sums and stores that of expert j
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    l[c] = __fadd_rn(l[c], __shfl_xor_sync(0xffffffffu, l[c], 4));
                    l[c] = __fadd_rn(l[c], __shfl_xor_sync(0xffffffffu, l[c], 1));
                    l[c] = __fadd_rn(l[c], __shfl_xor_sync(0xffffffffu, l[c], 2));
                    if (j == c) p = l[c];
                }
                if (b0 + a < nb) logits[(size_t)(b0 + a) * NEXP + e0 + j] = bias ? __fadd_rn(p, bias[e0 + j]) : p;
            }
        }
    }
    __syncthreads();
    if (tid == 0 && abort_flag) *(volatile int *)err = 31;      // a wait ran out: the host reports it and the logits are not to be used
}
// The first nbig rows of the grid take 4 TB tokens each, the others 4 TS: CTAs go to the SMs one each before any gets its second, so an SM that has a big one gets a small
// one beside it (the small rows first: 301 tokens 82.3 us per layer instead of 80.3).
template <int TB, int TS>
__global__ void __launch_bounds__(160) router_mid_kernel(const uint8_t *__restrict__ WT, const uint8_t *__restrict__ hS, const float *__restrict__ bias,
                                                         float *__restrict__ logits, int nb, int nbig, int *err) {
    const int y = blockIdx.y;
    if (TB == TS || y < nbig) router_mid_cta<TB>(WT, hS, bias, logits, nb, err, y * 4 * TB);
    else if constexpr (TB != TS) router_mid_cta<TS>(WT, hS, bias, logits, nb, err, nbig * 4 * TB + (y - nbig) * 4 * TS);
}
// Launched plainly (programmatically: 301 tokens 87.0 -> 88.3 us per layer, 400 88.8 -> 92.2) and with so much shared memory that per_sm CTAs fit an SM and no more.
// Without the preference for shared memory the driver leaves room for fewer than two CTAs at some sizes (400 tokens 92.0 -> 89.3).
#define RM_ALONE (116 << 10)
#define RM_PAIR (78 << 10)
// nbig = 0: all rows of 4 TB tokens
template <int TB, int TS>
static void launch_mid(cudaStream_t st, const void *router_t, const void *hS, const float *bias, float *logits, int nb, int nbig, int *err, int per_sm) {
    static bool attr_done = false;
    if (!attr_done) {
        cudaFuncSetAttribute(router_mid_kernel<TB, TS>, cudaFuncAttributeMaxDynamicSharedMemorySize, RM_ALONE);
        cudaFuncSetAttribute(router_mid_kernel<TB, TS>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared); attr_done = true;
    }
    static_assert(RM_STAGES * (4 * TB * RM_ROW + RM_WB) <= RM_PAIR && TS <= TB, "ring");
    const int small = nb - nbig * 4 * TB, rows = nbig + (small + 4 * TS - 1) / (4 * TS);
    launch_k(router_mid_kernel<TB, TS>, dim3(NEXP / 32, rows), 160, per_sm == 1 ? RM_ALONE : RM_PAIR, st, (const uint8_t *)router_t, (const uint8_t *)hS, bias, logits, nb, nbig, err);
}
extern "C" void k_router_pack_small(cudaStream_t st, const uint16_t *router, void *router_s) {
    router_pack_w_small_kernel<<<NEXP * HID / 4 / 256, 256, 0, st>>>(router, (uint2 *)router_s);
    k_count_add(1);
}
static int g_step_order = 0;
// single-token calls compute their logits in the order of the reference's `step` (bf_row) instead of `step_batch` (gmoe_set_step_order)
extern "C" void k_router_step_order(int on) { g_step_order = on != 0; }
extern "C" void k_router_logits_small(cudaStream_t st, const void *router_s, const void *router_t, const float *hn, void *hS, int relaid, const float *bias, float *logits, int nb, int *err) {
    if (nb <= 0) return;
    static bool attr_done = false;
    if (!attr_done) {
        cudaFuncSetAttribute(router_small_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, RS_ALONE);
        cudaFuncSetAttribute(router_small_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, RS_ALONE); attr_done = true;
    }
    if (!relaid) launch_k(router_pack_h_small_kernel, nb * 2, 256, 0, st, hn, (float4 *)hS, nb);
    static int sms = 0;
    if (!sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); if (sms < 1) sms = 148; }
    if (nb > 2 * 2 * sms / (NEXP / RS_EXP) * RS_TOK) {             // past two waves of the small kernel (148 tokens)
        // tokens per CTA (8 CTAs of 32 experts cover them): the fewest CTA-times of work per SM.  One CTA of 12 on each SM is the cheapest (to 216 tokens); two of 8 take
        // 0.5 us more (to 296), two of 12 another 3.5 (to 444), two of 16 another 6 (to 592); three of 8 take 1 us more than two of 12, three of 12 1.5 more than two of 16.
        const int one = sms / (NEXP / 32), two = 2 * sms / (NEXP / 32);
        // Between two of these lie SMs with one of either kind: 301 tokens (12 + 8) 81.7 -> 80.3 us per layer, 352 82.8 -> 81.6, 445 (16 + 12) 91.7 -> 89.1, 504 92.8 -> 90.6.
        // No more big rows than the tokens ask for (301 tokens with 18 of them 80.6), and one row less than fits the SMs: a full grid puts two big CTAs on one (352 82.9, 511 93.1).
        const int big2 = (nb - 8 * (two - 1) + 3) / 4, big3 = (nb - 12 * (two - 1) + 3) / 4, half = sms / (NEXP / 32);   // rows of the bigger kind among two - 1
        if (nb <= 12 * one) launch_mid<3, 3>(st, router_t, hS, bias, logits, nb, 0, err, 1);
        else if (nb <= 8 * two) launch_mid<2, 2>(st, router_t, hS, bias, logits, nb, 0, err, 2);
        else if (big2 <= half) launch_mid<3, 2>(st, router_t, hS, bias, logits, nb, big2, err, 2);
        else if (nb <= 12 * two) launch_mid<3, 3>(st, router_t, hS, bias, logits, nb, 0, err, 2);
        else if (big3 <= half) launch_mid<4, 3>(st, router_t, hS, bias, logits, nb, big3, err, 2);
        else launch_mid<4, 4>(st, router_t, hS, bias, logits, nb, 0, err, 2);
        k_count_add(relaid ? 1 : 2);
        return;
    }
    const dim3 grid(NEXP / RS_EXP, (nb + RS_TOK - 1) / RS_TOK);
    // CTAs that are no more than the SMs get one each: placed while the kernel before them ends, they would pair up on the SMs that are free first (32 tokens, 128 CTAs:
    // 50.5 -> 48.3 us per layer; no change up to 24 tokens, whose CTAs are fewer)
    const int rsm = (int)(grid.x * grid.y) <= sms ? RS_ALONE : RS_HB + RS_WB;
    if (g_step_order && nb == 1) launch_pdl(router_small_kernel<true, false>, grid, 256, rsm, st, (const uint8_t *)router_s, (const uint8_t *)hS, bias, logits, nb, err, RouterEdge{});
    else launch_pdl(router_small_kernel<false, false>, grid, 256, rsm, st, (const uint8_t *)router_s, (const uint8_t *)hS, bias, logits, nb, err, RouterEdge{});
    k_count_add(relaid ? 1 : 2);
}
// the joint of two layers and the router of the next, for one token; x and xo are different buffers (the CTAs read x while the first writes xo)
extern "C" void k_router_edge(cudaStream_t st, const void *router_s, const float *down, const float *uw, const int *tp, const float *x, float *xo, const uint16_t *w,
                              float *hn, int8_t *q, float *qs, int *qsum, const float *bias, float *logits, int *err) {
    static bool attr_done = false;
    if (!attr_done) {
        cudaFuncSetAttribute(router_small_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RS_HB + RS_WB);
        cudaFuncSetAttribute(router_small_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RS_HB + RS_WB); attr_done = true;
    }
    const RouterEdge ed = {down, uw, tp, x, xo, w, hn, q, qs, qsum};
    if (g_step_order) launch_pdl(router_small_kernel<true, true>, dim3(NEXP / RS_EXP), 256, RS_HB + RS_WB, st, (const uint8_t *)router_s, (const uint8_t *)NULL, bias, logits, 1, err, ed);
    else launch_pdl(router_small_kernel<false, true>, dim3(NEXP / RS_EXP), 256, RS_HB + RS_WB, st, (const uint8_t *)router_s, (const uint8_t *)NULL, bias, logits, 1, err, ed);
    k_count_add(1);
}
