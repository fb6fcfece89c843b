// k_expert_mma.cu -- grouped ternary expert GEMMs, register-decode variant for sm_100a.
//
// The 2-bit codes go from HBM straight into registers (128-bit loads), are split into four byte-wide code words per
// 32-bit word with one shift and one mask, and feed mma.sync.m16n8k32 (u8 codes x s8 activations -> s32) as the A
// operand without touching shared memory.  This is the path for decode batches (a few tokens per expert, bound by
// the weight stream) and the fallback for any token count.
//
// Launched programmatically (launch.cuh): while the last gate+up CTAs run, the first down CTAs already hold their weights.
//
// Arithmetic = maple.c:425-458 (tdot_multi): tot = sum(code * q) over the row, out = (float)(tot - qsum) * qs * s[r].
// Integer sums are exact, so any summation order gives the reference's int32.
//
// Column bookkeeping.  A packed row is cols/4 bytes; each 128-column group is 32 bytes and byte j holds columns
// j, j+32, j+64, j+96 at bits 0,2,4,6 (convert.py:29-33).  A K-chunk is 256 columns = 64 packed bytes.  Thread
// (g = lane/4, t = lane%4) loads bytes [16t, 16t+16) of the chunk for rows g and g+8: group G = 2*chunk + t/2, half
// h = t%2.  Word w (0..3) of that load shifted right by 2s and masked with 0x03030303 is the four codes of columns
// G*128 + 32s + 16h + 4w + (0..3).  MMA (s, p) takes words 2p and 2p+1 as its k = 4t..4t+3 and k = 16+4t..19+4t
// slices, so the B fragment of thread (g, t) is the 16 activation bytes of token g at column G*128 + 32s + 16h:
// words 2p, 2p+1 of that 16-byte piece.  Shared memory holds the tile's activations as [chunk][s][token][t][16 B],
// which makes every B-fragment fetch one conflict-free 128-bit load.
#include <cuda_runtime.h>
#include <stdint.h>
#include "kernels.h"
#include "launch.cuh"
#include "dev_math.cuh"
#include "span.cuh"

extern "C" void k_count_add(long n);


__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ldg_stream(const uint8_t *p) {   // weights are read once: do not keep them in L1
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ MoeTile ldcg_tile(const MoeTile *t) {
    const int4 v = __ldcg(reinterpret_cast<const int4 *>(t)); return MoeTile{v.x, v.y, v.z, v.w};
}

// KCH: K-chunks of 256 columns (8 for gate/up K=2048, 2 for down K=512).  NBLK: 8-token blocks per tile.
// GATEUP: rows block A = gate rows, block B = up rows of the same index, epilogue = SiLU*up;
// otherwise A and B are two consecutive 16-row blocks of the down matrix, epilogue = scale only.
// PF: chunks of weights in flight per thread.  NW: warps per CTA.  ITER: row blocks that a CTA takes in turn (down).
template <int KCH, int NBLK, bool GATEUP, int PF, int NW, bool FULL, int ITER>
__global__ void __launch_bounds__(NW * 32) expert_mma_kernel(ExpertArgs a) {
    constexpr bool STAGED = GATEUP && PF == 8;               // gate+up: the tokens' scales come with their rows, not behind the products (one tile deep 17.4 -> 17.2 us per layer, longer lists lose)
    constexpr int TN = NBLK * 8, KB = KCH * 256;            // tokens per tile, bytes of one int8 activation vector
    extern __shared__ __align__(16) uint8_t smem[];          // [KCH][4][TN][4][16]
    const int tile_i = blockIdx.y;
    if (GATEUP) { pdl_wait(); pdl_trigger(); }       // the tiles are its predecessor's; the down kernel's are two kernels old, so that its weights come in before its wait
    constexpr bool dense = !GATEUP && KCH == 8;
    const int ntiles = dense ? gridDim.y : __ldcg(a.ntiles);
    const MoeTile tile = dense ? MoeTile{0, a.dense_p0 + tile_i * TN, min(TN, a.dense_n - tile_i * TN), 0}
                               : ldcg_tile(a.tiles + (tile_i < a.max_tiles ? tile_i : 0));      // read beside the count, not after it
    if (tile_i >= ntiles) { if (!GATEUP) { pdl_wait(); pdl_trigger(); } return; }
    const ExpertPtrs ep = a.tab[tile.ex];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;

    const int rows_per_cta = NW * (GATEUP ? 16 : 32);
    int r0 = blockIdx.x * (rows_per_cta * ITER) + warp * (GATEUP ? 16 : 32);
    static_assert(ITER == 1 || (PF == KCH && !GATEUP), "all weights of a round at once");
    const uint8_t *wa = (GATEUP ? ep.gc : ep.dc) + (size_t)(r0 + g) * (KB / 4) + t * 16;
    const uint8_t *wb = GATEUP ? ep.uc + (size_t)(r0 + g) * (KB / 4) + t * 16 : wa + 16 * (KB / 4);
    // the weight stream starts before anything else: the first PF chunks are on their way while the activations are staged
    uint4 wq[PF][4];
#pragma unroll
    for (int p = 0; p < PF; p++) if (p < KCH) {
        wq[p][0] = ldg_stream(wa + p * 64); wq[p][1] = ldg_stream(wa + 8 * (KB / 4) + p * 64);
        wq[p][2] = ldg_stream(wb + p * 64); wq[p][3] = ldg_stream(wb + 8 * (KB / 4) + p * 64);
    }

    if (!GATEUP) { pdl_wait(); pdl_trigger(); }
    if (dense && tid == 0) span_begin(a.span);
    float *const t_qs = reinterpret_cast<float *>(smem + KCH * 4 * TN * 64); int *const t_qsum = reinterpret_cast<int *>(t_qs + TN);      // the tokens' scales and code sums
    // stage the tile's activation vectors (16-byte pieces) in fragment order
    if (GATEUP || !a.act_for_down) {
        const int8_t *src = GATEUP ? a.hq : a.aq;
        for (int i = tid; i < tile.cnt * (KB / 16); i += NW * 32) {
            int n = i / (KB / 16), q = i % (KB / 16);            // piece q covers columns 16q..16q+15
            int row = (GATEUP && a.ptok) ? a.ptok[tile.p0 + n] : tile.p0 + n;
            uint4 v = *reinterpret_cast<const uint4 *>(src + (size_t)row * KB + q * 16);
            if (STAGED && q == 0) { t_qs[n] = a.hqs[row]; t_qsum[n] = a.hqsum[row]; }
            int G = q >> 3, s = (q & 7) >> 1, h = q & 1, c = G >> 1, tt = (G & 1) * 2 + h;
            *reinterpret_cast<uint4 *>(smem + ((((c * 4 + s) * TN + n) * 4 + tt) << 4)) = v;
        }
    } else {
        // down, decode path: the SiLU outputs arrive as fp32 and are quantised here (the prep of maple.c:831), one warp per pair;
        // every row-block CTA of the tile repeats this for the tile's few pairs, the first one also stores the result
        for (int n = warp; n < tile.cnt; n += NW) {
            const int pair = tile.p0 + n;
            const float4 *r = reinterpret_cast<const float4 *>(a.act_for_down + (size_t)pair * 512) + lane * 4;
            float v[16];
#pragma unroll
            for (int i = 0; i < 4; i++) { float4 x = r[i]; v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w; }
            float mx = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i++) mx = fmaxf(mx, fabsf(v[i]));
            mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));      // >= 0: the bits order like the values
            const float sc = mx > 0.0f ? __fdiv_rn(mx, 127.0f) : 1.0f, inv = __fdiv_rn(1.0f, sc);
            int tot = 0; uint32_t pk[4] = {0, 0, 0, 0};
#pragma unroll
            for (int i = 0; i < 16; i++) { int qi = __float2int_rn(__fmul_rn(v[i], inv)); tot += qi; pk[i >> 2] |= (uint32_t)(qi & 0xFF) << (8 * (i & 3)); }
            tot = __reduce_add_sync(0xffffffffu, tot);
            // lane holds columns 16 lane .. 16 lane + 15 = piece q = lane
            const int q = lane, G = q >> 3, s = (q & 7) >> 1, h = q & 1, c = G >> 1, tt = (G & 1) * 2 + h;
            *reinterpret_cast<uint4 *>(smem + ((((c * 4 + s) * TN + n) * 4 + tt) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            if (lane == 0) { t_qs[n] = sc; t_qsum[n] = tot; }
            if (blockIdx.x == 0) {
                reinterpret_cast<uint4 *>(a.aq_out + (size_t)pair * 512)[lane] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
                if (lane == 0) { a.aqs_out[pair] = sc; a.aqsum_out[pair] = tot; }
            }
        }
    }
    __syncthreads();

#pragma unroll 1
    for (int it = 0; it < ITER; it++, r0 += rows_per_cta) {
        int acc_a[NBLK][4], acc_b[NBLK][4];
#pragma unroll
        for (int j = 0; j < NBLK; j++)
#pragma unroll
            for (int k = 0; k < 4; k++) { acc_a[j][k] = 0; acc_b[j][k] = 0; }

#pragma unroll
        for (int c = 0; c < KCH; c++) {
            const uint4 wa0 = wq[c % PF][0], wa1 = wq[c % PF][1], wb0 = wq[c % PF][2], wb1 = wq[c % PF][3];
            if (c + PF < KCH) {   // PF chunks in flight while this one is multiplied
                wq[c % PF][0] = ldg_stream(wa + (c + PF) * 64); wq[c % PF][1] = ldg_stream(wa + 8 * (KB / 4) + (c + PF) * 64);
                wq[c % PF][2] = ldg_stream(wb + (c + PF) * 64); wq[c % PF][3] = ldg_stream(wb + 8 * (KB / 4) + (c + PF) * 64);
            }
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const uint32_t m = 0x03030303u;
                uint32_t ax0 = (wa0.x >> (2 * s)) & m, ay0 = (wa0.y >> (2 * s)) & m, az0 = (wa0.z >> (2 * s)) & m, aw0 = (wa0.w >> (2 * s)) & m;
                uint32_t ax1 = (wa1.x >> (2 * s)) & m, ay1 = (wa1.y >> (2 * s)) & m, az1 = (wa1.z >> (2 * s)) & m, aw1 = (wa1.w >> (2 * s)) & m;
                uint32_t bx0 = (wb0.x >> (2 * s)) & m, by0 = (wb0.y >> (2 * s)) & m, bz0 = (wb0.z >> (2 * s)) & m, bw0 = (wb0.w >> (2 * s)) & m;
                uint32_t bx1 = (wb1.x >> (2 * s)) & m, by1 = (wb1.y >> (2 * s)) & m, bz1 = (wb1.z >> (2 * s)) & m, bw1 = (wb1.w >> (2 * s)) & m;
                const uint8_t *bs = smem + ((((c * 4 + s) * TN + g) * 4 + t) << 4);
#pragma unroll
                for (int j = 0; j < NBLK; j++) {
                    uint4 q = *reinterpret_cast<const uint4 *>(bs + j * 8 * 64);
                    mma_u8s8(acc_a[j], ax0, ax1, ay0, ay1, q.x, q.y);
                    mma_u8s8(acc_a[j], az0, az1, aw0, aw1, q.z, q.w);
                    mma_u8s8(acc_b[j], bx0, bx1, by0, by1, q.x, q.y);
                    mma_u8s8(acc_b[j], bz0, bz1, bw0, bw1, q.z, q.w);
                }
            }
        }

        if (ITER > 1 && it + 1 < ITER) {                         // the next round's weights: on their way while this one's results are stored
            wa += (size_t)rows_per_cta * (KB / 4); wb += (size_t)rows_per_cta * (KB / 4);
#pragma unroll
            for (int p = 0; p < PF; p++) {
                wq[p][0] = ldg_stream(wa + p * 64); wq[p][1] = ldg_stream(wa + 8 * (KB / 4) + p * 64);
                wq[p][2] = ldg_stream(wb + p * 64); wq[p][3] = ldg_stream(wb + 8 * (KB / 4) + p * 64);
            }
        }
        // epilogue: acc[j][0..3] = (row g, token 2t), (row g, token 2t+1), (row g+8, token 2t), (row g+8, token 2t+1)
        if (GATEUP) {
            // Two tokens at a time: their 32 values lie four to a lane in the eight lanes of one t and go one to a lane, so that the SiLU (a hundred and fifty
            // instructions, part of them in double) runs once for them and not four times, and not at all for tokens that do not exist: 1 token 17.8 -> 17.2 us per layer,
            // 4 22.6 -> 22.3, 13 33.4 -> 33.1, 32 46.5 -> 45.3, 64 58.6 -> 57.9, 128 73.9 -> 73.6
            const int k = lane & 3, rr = r0 + g + (k >> 1) * 8;
            const float s_a = ep.gs[rr], s_b = ep.us[rr];
#pragma unroll
            for (int j = 0; j < NBLK; j++)
#pragma unroll 1
                for (int tt = 0; tt < 4 && j * 8 + 2 * tt < tile.cnt; tt++) {
                    const int src = (lane & ~3) | tt, n = j * 8 + 2 * tt + (k & 1), pair = tile.p0 + n;
                    int va[4], vb[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) { va[i] = __shfl_sync(0xffffffffu, acc_a[j][i], src); vb[i] = __shfl_sync(0xffffffffu, acc_b[j][i], src); }
                    if (n >= tile.cnt) continue;
                    const int tok = STAGED ? 0 : a.ptok ? a.ptok[pair] : pair, qsum = STAGED ? t_qsum[n] : a.hqsum[tok];
                    const float qs = STAGED ? t_qs[n] : a.hqs[tok];
                    const int da = (k & 2 ? (k & 1 ? va[3] : va[2]) : (k & 1 ? va[1] : va[0])) - qsum, db = (k & 2 ? (k & 1 ? vb[3] : vb[2]) : (k & 1 ? vb[1] : vb[0])) - qsum;
                    const float gv = __fmul_rn(__fmul_rn((float)da, qs), s_a), uv = __fmul_rn(__fmul_rn((float)db, qs), s_b);
                    a.act[(size_t)pair * 512 + rr] = dev_silu_mul(gv, uv);
                    if (FULL && a.gate) { a.gate[(size_t)pair * 512 + rr] = gv; a.up[(size_t)pair * 512 + rr] = uv; }
                    if (FULL && a.gu_dots) { a.gu_dots[(size_t)pair * 1024 + rr] = da; a.gu_dots[(size_t)pair * 1024 + 512 + rr] = db; }
                }
        } else if (dense && NBLK == 1) {
            // the tile's 8 x 128 results through shared memory, so that a token's 128 leave as one run of 512 bytes: the rows may be page-locked host memory
            constexpr int PITCH = NW * 32 + 4;                   // the four token pairs of a store eight banks apart
            const float sca[2] = {ep.ds[r0 + g], ep.ds[r0 + g + 8]}, scb[2] = {ep.ds[r0 + g + 16], ep.ds[r0 + g + 24]};
            float *const out = reinterpret_cast<float *>(smem);
            float qs2[2]; int qsum2[2];
#pragma unroll
            for (int i = 0; i < 2; i++) { const int pair = tile.p0 + min(2 * t + i, tile.cnt - 1); qs2[i] = a.aqs[pair]; qsum2[i] = a.aqsum[pair]; }
            __syncthreads();                                     // the activations have been read
#pragma unroll
            for (int k = 0; k < 4; k++) {
                float *o = out + (2 * t + (k & 1)) * PITCH + warp * 32 + g + (k >> 1) * 8;
                o[0] = __fmul_rn(__fmul_rn((float)(acc_a[0][k] - qsum2[k & 1]), qs2[k & 1]), sca[k >> 1]);
                o[16] = __fmul_rn(__fmul_rn((float)(acc_b[0][k] - qsum2[k & 1]), qs2[k & 1]), scb[k >> 1]);
            }
            __syncthreads();
            for (int n = warp; n < tile.cnt; n += NW)
                reinterpret_cast<float4 *>(a.down + (size_t)(tile.p0 + n) * a.down_stride + blockIdx.x * (NW * 32))[lane] = reinterpret_cast<const float4 *>(out + n * PITCH)[lane];
        } else {
            const float sca[2] = {ep.ds[r0 + g], ep.ds[r0 + g + 8]}, scb[2] = {ep.ds[r0 + g + 16], ep.ds[r0 + g + 24]};
#pragma unroll
            for (int j = 0; j < NBLK; j++)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int n = j * 8 + 2 * t + (k & 1), rr = r0 + g + (k >> 1) * 8;
                    if (n >= tile.cnt) continue;
                    const int pair = tile.p0 + n;
                    int qsum_p; float qs;
                    if (a.act_for_down) { qs = t_qs[n]; qsum_p = t_qsum[n]; }
                    else { qs = a.aqs[pair]; qsum_p = a.aqsum[pair]; }
                    const int da = acc_a[j][k] - qsum_p, db = acc_b[j][k] - qsum_p;
                    float *drow = a.down + (size_t)pair * (a.down_stride ? a.down_stride : 2048);
                    if (FULL && a.rx_src) { const int2 sp = a.rx_src[pair]; drow = a.peer_down[sp.x] + (size_t)sp.y * 2048; }   // the row goes to the token's rank
                    drow[rr] = __fmul_rn(__fmul_rn((float)da, qs), sca[k >> 1]);
                    drow[rr + 16] = __fmul_rn(__fmul_rn((float)db, qs), scb[k >> 1]);
                    if (FULL && a.dn_dots) { a.dn_dots[(size_t)pair * 2048 + rr] = da; a.dn_dots[(size_t)pair * 2048 + rr + 16] = db; }
                }
        }
    }
    if (dense && tid == 0) span_end(a.span);
}

template <int KCH, int NBLK, bool GATEUP, int PF, int NW, bool FULL, int ITER>
static void launch_as(cudaStream_t st, const ExpertArgs *a) {
    const size_t smem = (size_t)KCH * 4 * NBLK * 8 * 64 + NBLK * 8 * 8;   // + scale and code sum per token
    static bool attr_done = false;
    if (!attr_done) { cudaFuncSetAttribute(expert_mma_kernel<KCH, NBLK, GATEUP, PF, NW, FULL, ITER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); attr_done = true; }
    dim3 grid((GATEUP ? 32 : 64) / (NW * ITER), a->max_tiles);
    launch_pdl(expert_mma_kernel<KCH, NBLK, GATEUP, PF, NW, FULL, ITER>, grid, NW * 32, smem, st, *a);
    k_count_add(1);
}
// FULL: the stage outputs and the rows that go to other ranks, which the lean kernels have no code for (13 tokens 35.1 -> 34.8 us per layer, 64 60.6 -> 60.1)
template <int KCH, int NBLK, bool GATEUP, int PF, int NW, int ITER = 1>
static void launch(cudaStream_t st, const ExpertArgs *a) {
    if (GATEUP ? a->gate != NULL || a->gu_dots != NULL : a->dn_dots != NULL || a->rx_src != NULL) launch_as<KCH, NBLK, GATEUP, PF, NW, true, ITER>(st, a);
    else launch_as<KCH, NBLK, GATEUP, PF, NW, false, ITER>(st, a);
}
// Two chunks in flight leave room for six CTAs per SM, which is what a long list of tiles wants (four chunks: 64 tokens 34.5 instead of 31 us).
// Where the whole list is resident at once at one or two CTAs per SM, all eight chunks go out together: one trip to memory instead of four
// (1 token 22.1 -> 20.9 us per layer; from 4 tokens on the two are level).
#define PF8_TILES 24
// Gate+up: eight warps per CTA share a tile's staged rows once the list of tiles is long.  max_tiles is 256 + the tokens, as many tiles as there could be.  Four / eight warps on this
// path: 132 tokens 69.4 / 70.5 us per layer, 144 71.7 / 72.2, 160 73.2 / 73.3, 176 74.9 / 74.4, 192 77.0 / 76.4, 224 83.2 / 82.6, 256 89.4 / 88.9.  By size a layer has no such list
// (from 161 tokens on the tcgen05 kernels run); other ranks' tokens and gmoe_set_path(1) bring them.
#define NW8_TILES 416
// The down kernel's CTAs each quantise the tile's activations for themselves and wait for its tile and its pointers: with more tiles than CTAs fit at once they take two
// or four blocks of 128 rows in turn, the next one's codes on their way while the results of this one are stored.  Rounds 1 / 2 / 4: 32 tokens 44.2 / 44.2 / 47.9 us per layer,
// 52 53.3 / 53.2 / 55.5, 64 56.4 / 55.9 / 57.8, 96 66.8 / 64.5 / 64.9, 112 71.1 / 68.4 / 68.1, 128 73.6 / 70.4 / 69.5.
#define DOWN2_TILES 304
#define DOWN4_TILES 360
extern "C" void k_gateup_mma(cudaStream_t st, const ExpertArgs *a, int tn) {
    if (a->max_tiles <= 0) return;
    if (tn != 8) launch<8, 4, true, 2, 4>(st, a); else if (a->max_tiles <= PF8_TILES) launch<8, 1, true, 8, 4>(st, a);
    else if (a->max_tiles <= NW8_TILES) launch<8, 1, true, 2, 4>(st, a); else launch<8, 1, true, 2, 8>(st, a);
}
extern "C" void k_down_mma(cudaStream_t st, const ExpertArgs *a, int tn) {
    if (a->max_tiles <= 0) return;
    if (tn != 8) launch<2, 4, false, 2, 4>(st, a); else if (a->max_tiles <= DOWN2_TILES) launch<2, 1, false, 2, 4>(st, a);
    else if (a->max_tiles <= DOWN4_TILES) launch<2, 1, false, 2, 4, 2>(st, a); else launch<2, 1, false, 2, 4, 4>(st, a);
}

// The attention projections (gpu_pre.m:200-256 gpre_dense*): the same int8 x 2-bit product with one matrix instead of 256
// experts and every token in it: K = 2048, two 16-row blocks per warp, 128 rows per CTA, tiles of 32 tokens.
// Up to 128 tokens in tiles of 8 with all weights of a CTA in flight at once: more CTAs (64 tokens, q,k,v: 192 instead of 48) and one trip to memory
// instead of four; the codes (1.6 MB) are read again by every tile, from L2.
template <int NBLK, int PF>
static void launch_dense(cudaStream_t st, const ExpertArgs *a, int rows) {
    const size_t smem = (size_t)8 * 4 * NBLK * 8 * 64 + NBLK * 8 * 8;
    static bool attr_done = false;
    if (!attr_done) { cudaFuncSetAttribute(expert_mma_kernel<8, NBLK, false, PF, 4, false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); attr_done = true; }
    launch_pdl(expert_mma_kernel<8, NBLK, false, PF, 4, false, 1>, dim3(rows / 128, (a->dense_n + NBLK * 8 - 1) / (NBLK * 8)), 128, smem, st, *a);
    k_count_add(1);
}
extern "C" void k_dense_mma(cudaStream_t st, const ExpertArgs *a, int rows) {
    if (a->dense_n <= 0 || rows <= 0) return;
    if (a->dense_n <= 128) launch_dense<1, 8>(st, a, rows); else launch_dense<4, 2>(st, a, rows);
}
