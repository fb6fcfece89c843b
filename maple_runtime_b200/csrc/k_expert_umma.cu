// k_expert_umma.cu -- grouped ternary expert GEMMs on the 5th-generation tensor cores (tcgen05.mma kind::i8), sm_100a.
//
// Work item = one tile (a used expert and up to UMMA_TN = 96 of its pairs) x one block of 2 x 128 weight rows:
//   gate+up: 128 gate rows and the 128 up rows of the same index (the SiLU*up step finds both in one thread);
//   down:    256 consecutive down rows, the even ones in accumulator half 0 and the odd ones in half 1 (a thread of the
//            epilogue then holds two neighbouring rows and stores them as one word of the compact result row, kernels.h WIRE_*).
// D[128 rows][N tokens] (s32, tensor memory) += A[128 rows][K] (u8 codes 0,1,2) x B[N tokens][K]^T (s8 activations).
// A persistent grid (one CTA per SM) walks the items; every ring below keeps running across items, so the next item's
// weights are already on their way while the current one is multiplied.
//
// Data movement
//   weights  HBM -> shared memory, still 2-bit packed: TMA tiled copies (cp.async.bulk.tensor, one tensor map per expert
//            matrix, box = 128 bytes x 128 rows, 128-byte swizzle), 32 KB stages = 256 rows x 512 columns; the swizzle makes
//            the later row-per-thread reads free of bank conflicts;
//   decode   eight warps; a thread owns one row of each accumulator half and every second block (of 128 or 256 columns): per 128 columns it reads 32 packed
//            bytes per row, expands every 32-bit word with (w >> 2s) & 0x03030303 (the four codes of columns 32s+4j..32s+4j+3
//            of the group, in column order; convert.py:29-33) and writes the block with tcgen05.st into the tensor-memory A
//            operand: lane = row, one 32-bit cell = four consecutive K values.  Decoded weights never touch shared memory;
//   B        int8 activation rows in pair order (the tokens' rows are put into expert-grouped order first), TMA
//            tiled copies (box = 128 bytes x 32, 64 or 96 rows, whichever covers the tile's pairs; 128-byte swizzle = the
//            K-major layout the MMA descriptor names), one block per stage.
// Arithmetic = maple.c:425-458: out = (float)(sum(code*q) - qsum) * qs * s[r]; integer sums are exact.  gate+up scales here;
// down stores sum(code*q) - qsum as integers and the combine applies qs and s[r] (same two roundings, same order).
//
// Warps (640 threads): 0 weight TMA, 1 B TMA, 2 and 3 MMA issue (one per accumulator half), 4-11 decode (warp w: tensor-memory lanes 32 (w % 4).., every second block),
// 12-19 epilogue.  The issuing warps come first, so that a scheduler does not keep them behind the decode warps' long runs: 843 tokens 99.8 -> 99.4 us per layer, 1300 119.1 -> 118.7.
// An MMA is issued by one elected lane of warp-uniform code; a kind::i8 MMA with A in tensor memory executes in N/2 cycles.
// Instructions in the SM's cache bound these kernels as much as any unit: five roles run side by side on every scheduler, each in code of its own, and what does not fit the
// instruction cache is fetched again from the L2 side in every round.  The kernels were 72 to 78 KB of code (spin loops unrolled four times at every wait, the
// copying warps' loops unrolled whole, stage outputs and expert parallelism beside the lean path); they are 26 to 31 KB now, and with nothing else changed a layer of 301 / 843 /
// 2048 tokens took 93.2 / 116.3 / 163.4 us instead of 97.5 / 119.9 / 168.0.  So: loops over blocks, stages and items stay rolled, one copy of an epilogue piece, a
// predicated block of MMAs instead of a branch per MMA, and FULL = the variant with stage outputs and expert parallelism.  With the three points below: 92.4 / 114.0 / 162.2.
// One barrier pair per block (k_full: the four decode warps that wrote the A stage, and the bytes of the B stage; k_empty: both MMA warps) instead of one per
// ring: a wait that succeeds at once still costs a warp 100 to 180 cycles here.  A look at the next barrier ahead of time (test_wait) made it slower (92.9 / 114.8 / 163.1): more
// instructions.  One MMA warp for both halves: 93.2 / 115.3 / 163.5.  Sixteen decode warps, one half each: 96.9 / 121.6 / 173.9, at 72 registers a thread.
// Tensor memory: A stages for two blocks of 256 or three of 128 columns (UmShape), and the rest, which the accumulators of two items share, even items from the low end
// and odd ones from the high end, 2 N columns each: those that fit beside each other (pairs rounded up to 16s, 128 or 160 for both) let an item's epilogue run under the next
// one's MMAs; larger ones wait for each other (acc_place).  Deeper rings are not faster: B stages 3 against 4 of 256 columns 99.3 and 100.1 us at 843 tokens, weight stages 4
// against 3 83.3 and 82.5 at 301 (2: 86.2); tiles of 32 pairs in the room that leaves: level.
// The codes are read once per tile: their copies say so to the L2 (evict_first), which then still holds the rows that come in, the results and what the next kernels read
// when they are asked for: a layer of 301 / 511 / 843 / 2048 tokens 92.1 / 104.4 / 113.8 / 159.8 -> 88.1 / 99.6 / 111.0 / 157.4 us.
// An item's scales come in pair order (the kernels at the end of this file put them there): through the token index they were a second global read in front of every item.
// Every mbarrier wait is bounded (umma.cuh): on a timeout the CTA raises args.err, frees tensor memory and returns.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include "kernels.h"
#include "launch.cuh"
#include "dev_math.cuh"
#include "umma.cuh"
#include "span.cuh"

extern "C" void k_count_add(long n);

#define UM_TN UMMA_TN                /* 96 */
#define UM_NACC 2                    /* items whose accumulators are in use at a time: an item's epilogue runs under the next item's MMAs */
#define UM_WBYTES (256 * 128)        /* a weight stage: 256 rows x 512 columns */
#define UM_WSTAGES 3
#define UM_BSTAGES 8                 /* at most */
// What is handed over at a time: BW x 128 columns.  NA A stages (64 BW columns of tensor memory each: the block in both halves), the rest of tensor memory for the
// accumulators; BST stages of the tile's rows, BW sub-tiles of 128 columns each.
template <int BW> struct UmShape {
    static constexpr int NA = BW == 2 ? 2 : 3, ACC = 512 - 64 * BW * NA, BST = BW == 2 ? 3 : 8, BBYTES = UM_TN * 128 * BW, KCOLS = 128 * BW;
    static_assert(ACC >= 2 * UM_TN && NA < BST && BST <= UM_BSTAGES, "stages");
};

struct __align__(16) UmShared {
    uint64_t w_full[UM_WSTAGES], w_empty[UM_WSTAGES], k_full[UM_BSTAGES], k_empty[UM_BSTAGES], acc_full[UM_NACC], acc_empty[UM_NACC];
    uint32_t tmem_base; int abort_flag;
    __align__(16) float m_qs[8][UM_TN]; __align__(16) int m_qsum[8][UM_TN];      // per epilogue warp: scale and code-sum correction of the tile's tokens
    __align__(16) unsigned long long m_dst[8][UM_TN];                             // expert parallel, down: where each token's compact row lives (a peer's memory)
};

__device__ __forceinline__ MoeTile ldcg_tile(const MoeTile *t) {
    const int4 v = __ldcg(reinterpret_cast<const int4 *>(t)); return MoeTile{v.x, v.y, v.z, v.w};
}

template <int K, int MODE, bool FULL, int BW>
__global__ void __launch_bounds__(640, 1) expert_umma_kernel(ExpertArgs a, const __grid_constant__ TMap4 bmap) {
    extern __shared__ __align__(1024) uint8_t um_smem_raw[];
    uint8_t *base = (uint8_t *)(((uintptr_t)um_smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *wsm = base;                                              // packed weights
    using SH = UmShape<BW>;
    uint8_t *bsm = base + UM_WSTAGES * UM_WBYTES;                         // int8 activations
    __shared__ UmShared sh_static;                                    // static, so that the compiler knows these accesses are shared-memory ones
    UmShared *sh = &sh_static;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    constexpr bool GATEUP = MODE == 0, DENSE = MODE == 2, DOWN = MODE == 1;
    constexpr int NA = SH::NA, WST = UM_WSTAGES, BST = SH::BST, KB = K / SH::KCOLS, BPS = 4 / BW, TN = UM_TN;      // KB: blocks of an item, BPS: of a weight stage
    constexpr int NACC = UM_NACC;
    constexpr uint32_t ACOL = SH::ACC;                              // first A column (behind the accumulators)
    static_assert(NACC == 2 && KB % BPS == 0, "blocks");
    const int MB = GATEUP ? 4 : (DENSE ? a.dense_mblocks : 8);      // 256-row blocks of the matrix (gate+up: 128 + 128)
    constexpr int NSB = KB / BPS;
    volatile int *abortp = &sh->abort_flag;

    if (tid == 0) {
        for (int s = 0; s < WST; s++) { mbar_init(&sh->w_full[s], 1); mbar_init(&sh->w_empty[s], 8); }
        // an A stage is full when its four decode warps have stored it, a B stage when its bytes have landed; both are empty again
        // when both issuing warps' MMAs on them have completed
        for (int s = 0; s < BST; s++) { mbar_init(&sh->k_full[s], 5); mbar_init(&sh->k_empty[s], 2); }
        for (int b = 0; b < NACC; b++) { mbar_init(&sh->acc_full[b], 2); mbar_init(&sh->acc_empty[b], 8); }
        sh->abort_flag = 0; mbar_init_fence();
    }
    const int ntiles = DENSE ? (a.dense_n + TN - 1) / TN : __ldcg(a.ntiles), nitems = ntiles * MB;
    auto tile_at = [&](const int i) {
        return DENSE ? MoeTile{0, a.dense_p0 + i * TN, min(TN, a.dense_n - i * TN), 0} : ldcg_tile(a.tiles + i);
    };
    // The CTA acquires the maps that it will read through, all of them before its first copy and each by a thread of its own: that adds 0.5 us to a layer of two
    // such kernels (301 tokens 97.6 -> 98.1 us, 2048 168.2 -> 169.0).  By the weight warp ahead of each item it added 6.5 us, by the decode warps while
    // the first copies were under way 15 us: an acquire takes 0.25 us, more with copies in flight.  Its scope makes no difference.
    auto maps_of = [&](const MoeTile &t) { return a.maps + (a.call_maps ? t.u : t.ex); };
    auto acquire = [&](const TMap *m) { if (a.call_maps) tma_acquire_map_gpu(m); else tma_acquire_map_sys(m); };
    if (warp >= 4 && warp < 12) {
#pragma unroll 1
        for (int i = blockIdx.x + (lane * 8 + warp - 4) * gridDim.x; i < nitems; i += 256 * gridDim.x) {
            const ExpertMaps *e = maps_of(tile_at(i / MB));
            if (GATEUP) { acquire(&e->gate); acquire(&e->up); } else acquire(&e->down);
            if (DENSE) break;                                          // one matrix
        }
    }
    if (warp == 2) tmem_alloc(&sh->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tb = sh->tmem_base;
    bool live = true;
    // launched programmatically: the weights start to come in before the wait (the tile list is two kernels old), everything else after it.  Warp 0, which does not
    // wait, leaves the trigger to the others: the first one counts for the CTA, and a successor may read what is two kernels old before its own wait
    if (warp != 0) { pdl_wait(); pdl_trigger(); }
    if (DENSE && tid == 0) span_begin(a.span);

    // where item number i of this CTA keeps its accumulators (half 0, then half 1, n2 columns in all); over: they cover columns of the item before it
    uint32_t acc_prev = 0;
    auto acc_place = [&](const uint32_t i, const uint32_t n2, bool &over) {
        over = n2 + acc_prev > (uint32_t)SH::ACC; acc_prev = n2;
        return i & 1 ? (uint32_t)SH::ACC - n2 : 0u;
    };

    if (warp >= 4 && warp < 12) {
        // ---------------- decode: this warp's 32 rows of both halves, every second block, from the shared-memory ring ----------------
        const int q4 = warp & 3, par = (warp - 4) >> 2, R = q4 * 32 + lane;       // R: row inside a half = tensor-memory lane
        const uint32_t a_lane = tb + ((uint32_t)(q4 * 32) << 16) + ACOL;
        uint32_t wcnt = 0;
#pragma unroll 1
        for (int item = blockIdx.x; item < nitems && live; item += gridDim.x) {
#pragma unroll 1
            for (int sb = 0; sb < NSB && live; sb++, wcnt++) {
                const int ws = wcnt % WST;
                if (!mbar_wait(&sh->w_full[ws], (wcnt / WST) & 1, abortp)) { live = false; break; }
                const uint8_t *wr = wsm + ws * UM_WBYTES + R * 128;
#pragma unroll
                for (int q = par, qq = 0; qq < BPS / 2 && live; qq++, q += 2) {      // this warp's blocks of the weight stage
                    const uint32_t b = BPS * wcnt + q, as = b % NA, bo = b - NA;      // bo: the block that had the A stage before
#pragma unroll
                    for (int u = 0; u < 2 * BW; u++) {                   // 128 columns of one half at a time
                        const int sub = u >> 1, half = u & 1, c = 2 * (BW * q + sub);
                        const uint8_t *w_ = wr + half * (128 * 128);
                        const uint4 v0 = *reinterpret_cast<const uint4 *>(w_ + ((c ^ (R & 7)) << 4)), v1 = *reinterpret_cast<const uint4 *>(w_ + (((c + 1) ^ (R & 7)) << 4));
                        const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
                        uint32_t o[32];
                        // gate+up and dense: left shifts, which the multiply pipe can take beside the masks; the operand is 64 x code and the epilogue shifts the
                        // sums back, exactly (at most 192 * 127 * 2048 = 5e7).  2048 tokens: gate+up 51.0 -> 49.5 us between events, 4096: 80.7 -> 79.1.  The down
                        // kernel has fewer blocks per epilogue and loses (38.4 -> 39.3): plain codes.
#pragma unroll
                        for (int sft = 0; sft < 4; sft++)
#pragma unroll
                            for (int j = 0; j < 8; j++) o[sft * 8 + j] = DOWN ? (w[j] >> (2 * sft)) & 0x03030303u : (w[j] << (6 - 2 * sft)) & 0xC0C0C0C0u;
                        if (u == 0) {
                            if (b >= NA && !mbar_wait(&sh->k_empty[bo % BST], (bo / BST) & 1, abortp)) { live = false; break; }
                            tc_fence_after();
                        }
                        tmem_st32(a_lane + as * (64 * BW) + half * (32 * BW) + sub * 32, o);
                    }
                    if (!live) break;
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->k_full[b % BST]);
                }
                if (live && lane == 0) mbar_arrive(&sh->w_empty[ws]);
            }
        }
    } else if (warp == 0) {
        // ---------------- weight TMA (one lane): per stage the 128 rows of half 0 and the 128 of half 1, 512 columns ----------------
        if (lane == 0) {
            uint32_t wcnt = 0; const uint64_t once = l2_evict_first();
            MoeTile tnext = blockIdx.x < nitems ? tile_at(blockIdx.x / MB) : MoeTile{0, 0, 0, 0};      // one item ahead: no load latency at an item's start
#pragma unroll 1
            for (int item = blockIdx.x; item < nitems && live; item += gridDim.x) {
                const MoeTile tile = tnext;
                if (item + (int)gridDim.x < nitems) {
                    tnext = tile_at((item + gridDim.x) / MB);
                    const ExpertMaps *en = maps_of(tnext);              // the next item's expert: its maps are in the descriptor cache when its copies start
                    if (GATEUP) { tma_prefetch_map(&en->gate); tma_prefetch_map(&en->up); } else tma_prefetch_map(&en->down);
                }
                const int mb = item % MB;
                const ExpertMaps *em = maps_of(tile);
#pragma unroll 1
                for (int sb = 0; sb < NSB && live; sb++, wcnt++) {
                    const int ws = wcnt % WST;
                    if (!mbar_wait(&sh->w_empty[ws], ((wcnt / WST) & 1) ^ 1, abortp)) { live = false; break; }
                    const uint32_t dst = smem_u32(wsm + ws * UM_WBYTES);
                    mbar_expect_tx(&sh->w_full[ws], UM_WBYTES);
                    if (GATEUP) {
                        tma_load_2d(dst, &em->gate, sb * 128, mb * 128, &sh->w_full[ws], once);
                        tma_load_2d(dst + 128 * 128, &em->up, sb * 128, mb * 128, &sh->w_full[ws], once);
                    } else {
                        tma_load_3d(dst, &em->down, sb * 128, 0, mb * 128, &sh->w_full[ws], once);             // the even rows of the 256-row block
                        tma_load_3d(dst + 128 * 128, &em->down, sb * 128, 1, mb * 128, &sh->w_full[ws], once);   // the odd rows
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- B TMA (one lane): per 128-column block one box of the pair-ordered int8 activations ----------------
        if (lane == 0) {
            uint32_t bcnt = 0;
            MoeTile tnext = blockIdx.x < nitems ? tile_at(blockIdx.x / MB) : MoeTile{0, 0, 0, 0};
#pragma unroll 1
            for (int item = blockIdx.x; item < nitems && live; item += gridDim.x) {
                const MoeTile tile = tnext;
                if (item + (int)gridDim.x < nitems) tnext = tile_at((item + gridDim.x) / MB);
                // only as many rows as the tile has pairs, in steps of 32 (the MMA reads (cnt + 15) & ~15 <= that many)
                const int bi = tile.cnt > 0 ? (tile.cnt - 1) >> 5 : 0;
#pragma unroll 1
                for (int kb = 0; kb < KB && live; kb++, bcnt++) {
                    const int s = bcnt % BST;
                    if (!mbar_wait(&sh->k_empty[s], ((bcnt / BST) & 1) ^ 1, abortp)) { live = false; break; }
                    mbar_expect_tx(&sh->k_full[s], 128 * BW * 32 * (bi + 1));
#pragma unroll
                    for (int i = 0; i < BW; i++) tma_load_2d(smem_u32(bsm + s * SH::BBYTES + i * UM_TN * 128), &bmap.m[bi], kb * SH::KCOLS + i * 128, tile.p0, &sh->k_full[s]);
                }
            }
        }
    } else if (warp < 4) {
        // ---------------- MMA issue: warp 2 accumulator half 0, warp 3 half 1.  While one of them is inside a wait, the other's
        // MMAs keep the tensor pipe busy.  The whole warp walks the loop and waits; one elected lane issues and commits ----------------
        const uint32_t h = warp - 2;
        const uint64_t bdesc0 = smem_desc_k128(__shfl_sync(0xffffffffu, smem_u32(bsm), 0), 0);
        const uint32_t kfull0 = smem_u32(&sh->k_full[0]), kempty0 = smem_u32(&sh->k_empty[0]);
        uint32_t as = 0, bs = 0, bp = 0, icnt = 0;
        int cnt_next = blockIdx.x < nitems ? tile_at(blockIdx.x / MB).cnt : 0;
#pragma unroll 1
        for (int item = blockIdx.x; item < nitems && live; item += gridDim.x, icnt++) {
            const int cnt = __shfl_sync(0xffffffffu, cnt_next, 0);
            if (item + (int)gridDim.x < nitems) cnt_next = tile_at((item + gridDim.x) / MB).cnt;
            const uint32_t N = (uint32_t)((cnt + 15) & ~15), idesc = idesc_i8_u8s8(N);
            bool over;
            const uint32_t buf = icnt % NACC, d = tb + acc_place(icnt, 2 * N, over) + h * N;
            if (!mbar_wait(&sh->acc_empty[buf], ((icnt / NACC) & 1) ^ 1, abortp)) { live = false; break; }
            if (over && icnt && !mbar_wait(&sh->acc_empty[buf ^ 1], ((icnt - 1) / NACC) & 1, abortp)) { live = false; break; }
            tc_fence_after();
#pragma unroll 1
            for (int kb = 0; kb < KB; kb++) {
                if (!mbar_wait_addr(kfull0 + bs * 8, bp, abortp)) { live = false; break; }
                tc_fence_after();
                const uint32_t acol = tb + ACOL + as * (64 * BW) + h * (32 * BW), kb_empty = kempty0 + bs * 8;
                const uint64_t bd = bdesc0 + (uint64_t)(bs * (SH::BBYTES >> 4));
                if (++as == NA) as = 0;
                if (++bs == BST) { bs = 0; bp ^= 1; }
                if (BW == 2) umma_i8_block<false>(d, acol, bd, idesc, kb != 0, 0);
                umma_i8_block<true>(d, acol + 32 * (BW - 1), bd + (BW - 1) * (UM_TN * 128 >> 4), idesc, BW == 2 || kb != 0, kb_empty);
            }
            if (live && elect_one()) umma_commit(&sh->acc_full[buf]);
            __syncwarp();
        }
    } else {
        // ---------------- epilogue: lane = weight row, columns = tokens; warps 12-15 take the even 16-column pieces, 16-19 the odd ----------------
        const int ew = warp - 12, q4 = warp & 3, half = ew >> 2, row = q4 * 32 + lane;   // a warp reaches the tensor-memory lanes 32 (warp % 4) ..
        uint32_t icnt = 0;
        // An item's header is a chain tile -> scale and code sum of its tokens, and tile -> pointer table -> row
        // scales: the tile is read two items ahead, the pointer table and the tokens' values one item ahead (into registers; they go
        // to shared memory when the item starts), so that an item starts without a dependent global read in front of it.
        const int stride = gridDim.x;
        constexpr int HN = TN / 32;
        MoeTile t1 = blockIdx.x < nitems ? tile_at(blockIdx.x / MB) : MoeTile{0, 0, 0, 0};
        MoeTile t2 = (int)blockIdx.x + stride < nitems ? tile_at((blockIdx.x + stride) / MB) : MoeTile{0, 0, 0, 0};
        ExpertPtrs ep1 = a.tab[t1.ex];
        float h_qs[HN]; int h_qsum[HN]; unsigned long long h_dst[HN];
        auto header_load = [&](const MoeTile &t) {      // the values of tokens lane, lane + 32, lane + 64 of tile t (clamped to its pairs)
#pragma unroll
            for (int i = 0; i < HN; i++) {
                const int n = lane + 32 * i, pair = t.p0 + (n < t.cnt ? n : 0);
                h_qs[i] = GATEUP ? a.hqs[pair] : a.aqs[pair];
                h_qsum[i] = GATEUP ? a.hqsum[pair] : (DENSE ? a.aqsum[pair] : 32768 - a.aqsum[pair]);
                if (DOWN && FULL && a.rx_src) { const int2 sp = a.rx_src[pair]; h_dst[i] = (unsigned long long)(uintptr_t)(a.peer_wire[sp.x] + (size_t)sp.y * WIRE_PITCH); }
            }
        };
        if (blockIdx.x < nitems) header_load(t1);
        // the row scales of an item are read while the item before it is worked on (the pointer table they hang off has arrived by then)
        float s0n = 0.0f, s1n = 0.0f;
        auto scales_load = [&](const ExpertPtrs &e, const int it) {
            const int r = GATEUP ? (it % MB) * 128 + row : (it % MB) * 256 + 2 * row;
            s0n = GATEUP ? e.gs[r] : (DENSE ? e.ds[r] : 0.0f); s1n = GATEUP ? e.us[r] : (DENSE ? e.ds[r + 1] : 0.0f);
        };
        if (blockIdx.x < nitems) scales_load(ep1, blockIdx.x);
#pragma unroll 1
        for (int item = blockIdx.x; item < nitems && live; item += stride, icnt++) {
            const MoeTile tile = t1;
            const int mb = item % MB, cnt = tile.cnt, N = (cnt + 15) & ~15;
            const uint32_t buf = icnt % NACC;
            const int r0 = GATEUP ? mb * 128 + row : mb * 256 + 2 * row;      // down: half 0 holds row r0, half 1 row r0 + 1
            const float s0 = s0n, s1 = s1n;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < HN; i++) {
                sh->m_qs[ew][lane + 32 * i] = h_qs[i]; sh->m_qsum[ew][lane + 32 * i] = h_qsum[i];
                if (DOWN && FULL && a.rx_src) sh->m_dst[ew][lane + 32 * i] = h_dst[i];
            }
            __syncwarp();
            t1 = t2; ep1 = a.tab[t1.ex];
            if (item + 2 * stride < nitems) t2 = tile_at((item + 2 * stride) / MB);
            if (item + stride < nitems) header_load(t1);                     // in flight while this item's pieces are worked on
            if (!mbar_wait(&sh->acc_full[buf], (icnt / NACC) & 1, abortp)) { live = false; break; }
            tc_fence_after();
            bool over;
            const uint32_t d_lane = tb + ((uint32_t)(q4 * 32) << 16) + acc_place(icnt, 2 * (uint32_t)N, over);
            auto release = [&]() { tc_fence_before(); __syncwarp(); if (lane == 0) mbar_arrive(&sh->acc_empty[buf]); };
            auto piece = [&](const int c0, uint32_t (&v0)[16], uint32_t (&v1)[16]) {
                const int lim = cnt - c0;                                 // tokens of this piece that exist
                if (GATEUP || DENSE) {
                    float o0[16], o1[16];
                    {   // scale and code-sum correction of the piece's 16 tokens: eight 128-bit shared-memory reads
                        const int4 *qsv = reinterpret_cast<const int4 *>(&sh->m_qsum[ew][c0]);
                        const float4 *qfv = reinterpret_cast<const float4 *>(&sh->m_qs[ew][c0]);
#pragma unroll
                        for (int g4 = 0; g4 < 4; g4++) {
                            const int4 qs4 = qsv[g4]; const float4 qf4 = qfv[g4];
                            const int qsum[4] = {qs4.x, qs4.y, qs4.z, qs4.w}; const float qs[4] = {qf4.x, qf4.y, qf4.z, qf4.w};
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const int j = g4 * 4 + k, d0 = ((int)v0[j] >> 6) - qsum[k], d1 = ((int)v1[j] >> 6) - qsum[k];
                                o0[j] = __fmul_rn(__fmul_rn((float)d0, qs[k]), s0); o1[j] = __fmul_rn(__fmul_rn((float)d1, qs[k]), s1);
                                v0[j] = (uint32_t)d0; v1[j] = (uint32_t)d1;
                            }
                        }
                    }
                    if (DENSE) {      // fp32 rows of the projection: this thread's two neighbouring rows of every token of the piece
                        float *dp = a.down + (size_t)(tile.p0 + c0) * a.down_stride + r0;
#pragma unroll
                        for (int j = 0; j < 16; j++) if (j < lim) *reinterpret_cast<float2 *>(dp + (size_t)j * a.down_stride) = make_float2(o0[j], o1[j]);
                        return;
                    }
                    // one base pointer per thread; the token index only adds a constant, so a store is one instruction
                    float *gp = a.gate + (size_t)(tile.p0 + c0) * 512 + r0, *up_ = a.up + (size_t)(tile.p0 + c0) * 512 + r0;
#pragma unroll
                    for (int j = 0; j < 16; j++) if (j < lim) { gp[j * 512] = o0[j]; up_[j * 512] = o1[j]; }
                    if (FULL && a.gu_dots) {
                        int *dp = a.gu_dots + (size_t)(tile.p0 + c0) * 1024 + r0;
#pragma unroll
                        for (int j = 0; j < 16; j++) if (j < lim) { dp[j * 1024] = (int)v0[j]; dp[j * 1024 + 512] = (int)v1[j]; }
                    }
                }
            };
            // down: (dot + 32768) of this thread's two rows in one 32-bit word per token (the scales are applied where the rows are
            // combined); cd = two more bits per value, nonzero only when a value needs more than 16 bits (|dot| >= 32768)
            auto pack = [&](const int c0, uint32_t (&v0)[16], uint32_t (&v1)[16], uint32_t (&pk)[16], unsigned long long &cd) {
                const int4 *qsv = reinterpret_cast<const int4 *>(&sh->m_qsum[ew][c0]);
                uint32_t high = 0u;
#pragma unroll
                for (int g4 = 0; g4 < 4; g4++) {
                    const int4 qs4 = qsv[g4]; const int bq[4] = {qs4.x, qs4.y, qs4.z, qs4.w};       // 32768 - qsum
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int j = g4 * 4 + k;
                        v0[j] += (uint32_t)bq[k]; v1[j] += (uint32_t)bq[k];
                        pk[j] = __byte_perm(v0[j], v1[j], 0x5410);
                        high |= v0[j] | v1[j];
                    }
                }
                // the two more bits are looked at only where the warp has one that is set (or a stage comparison wants the sums): per token and thread that is
                // four instructions instead of thirteen
                cd = 0ull;
                if (__any_sync(0xffffffffu, high >> 16) || (FULL && a.dn_dots)) {
#pragma unroll
                    for (int j = 0; j < 16; j++) cd |= (unsigned long long)(((v0[j] >> 16) & 3u) | (((v1[j] >> 16) & 3u) << 2)) << (4 * j);
                }
            };
            auto store = [&](const int c0, const uint32_t (&pk)[16], const unsigned long long cd) {
                const int lim = cnt - c0;                                 // tokens of this piece that exist
                const bool esc = __any_sync(0xffffffffu, cd != 0ull);
                const size_t rec0 = (size_t)a.wire_cap * WIRE_PITCH;            // the records sit behind the rows
                const bool recw = mb == 0 && q4 == 0 && lane < 16 && lane < lim; // one warp per piece writes the tokens' records
                if (!FULL || !a.rx_src) {
                    uint8_t *rowp = a.wire + (size_t)(tile.p0 + c0) * WIRE_PITCH;
                    uint32_t *dp = reinterpret_cast<uint32_t *>(rowp) + (r0 >> 1);
#pragma unroll
                    for (int j = 0; j < 16; j++) if (j < lim) dp[j * (WIRE_PITCH / 4)] = pk[j];
                    if (recw) *reinterpret_cast<int2 *>(a.wire + rec0 + (size_t)(tile.p0 + c0 + lane) * WIRE_REC) = make_int2(__float_as_int(sh->m_qs[ew][c0 + lane]), tile.ex);
                    if (esc) {
#pragma unroll
                        for (int j = 0; j < 16; j++) if (j < lim) {
                            const uint32_t code = (uint32_t)(cd >> (4 * j)) & 15u;
                            if (code) {
                                atomicOr(reinterpret_cast<uint32_t *>(rowp + (size_t)j * WIRE_PITCH + 4096) + (r0 >> 4), code << ((r0 & 15) * 2));
                                atomicOr(reinterpret_cast<int *>(a.wire + rec0 + (size_t)(tile.p0 + c0 + j) * WIRE_REC + 8), 1 << (r0 >> 7));
                            }
                        }
                    }
                } else {
                    // expert parallel: each row goes to the rank that owns the token
                    const ulonglong2 *dv = reinterpret_cast<const ulonglong2 *>(&sh->m_dst[ew][c0]);
#pragma unroll
                    for (int j2 = 0; j2 < 8; j2++) {
                        const ulonglong2 d2 = dv[j2];
                        if (2 * j2 < lim) reinterpret_cast<uint32_t *>((uintptr_t)d2.x)[r0 >> 1] = pk[2 * j2];
                        if (2 * j2 + 1 < lim) reinterpret_cast<uint32_t *>((uintptr_t)d2.y)[r0 >> 1] = pk[2 * j2 + 1];
                    }
                    if (recw) {
                        const int2 sp = a.rx_src[tile.p0 + c0 + lane];
                        *reinterpret_cast<int2 *>(a.peer_wire[sp.x] + rec0 + (size_t)sp.y * WIRE_REC) = make_int2(__float_as_int(sh->m_qs[ew][c0 + lane]), tile.ex);
                    }
                    if (esc) {
#pragma unroll
                        for (int j = 0; j < 16; j++) if (j < lim) {
                            const uint32_t code = (uint32_t)(cd >> (4 * j)) & 15u;
                            if (code) {
                                const int2 sp = a.rx_src[tile.p0 + c0 + j];
                                uint8_t *pb = a.peer_wire[sp.x];
                                atomicOr(reinterpret_cast<uint32_t *>(pb + (size_t)sp.y * WIRE_PITCH + 4096) + (r0 >> 4), code << ((r0 & 15) * 2));
                                atomicOr(reinterpret_cast<int *>(pb + rec0 + (size_t)sp.y * WIRE_REC + 8), 1 << (r0 >> 7));
                            }
                        }
                    }
                }
                if (FULL && a.dn_dots) {      // (dot + 32768) again from the 16 stored bits and the two escape bits: 0, +65536 or -65536 on top
                    int *ip = a.dn_dots + (size_t)(tile.p0 + c0) * 2048 + r0;
#pragma unroll
                    for (int j = 0; j < 16; j++) if (j < lim) {
                        const uint32_t code = (uint32_t)(cd >> (4 * j)) & 15u;
                        const int h0 = ((int)((code & 3u) ^ 2u) - 2) << 16, h1 = ((int)((code >> 2) ^ 2u) - 2) << 16;
                        *reinterpret_cast<int2 *>(ip + j * 2048) = make_int2((int)(pk[j] & 0xFFFFu) + h0 - 32768, (int)(pk[j] >> 16) + h1 - 32768);
                    }
                }
            };
            // this warp's pieces: c0 = 16 half, + 32, ...
            const int np = (N / 16 - half + 1) / 2;
            if (DOWN) {
                // piece by piece: 16 bits per value in registers, then the stores; the accumulators go back to the MMA warps as soon as
                // the last piece has been read
                if (np == 0) release();
#pragma unroll 1
                for (int k = 0; k < np; k++) {
                    uint32_t v0[16], v1[16], pk[16]; unsigned long long cd;
                    const int c0 = half * 16 + 32 * k;
                    tmem_ld16(d_lane + c0, v0); tmem_ld16(d_lane + N + c0, v1);
                    tmem_ld_wait();
                    if (k == np - 1) release();
                    pack(c0, v0, v1, pk, cd);
                    store(c0, pk, cd);
                }
            } else {
                if (np == 0) release();
                int c0 = half * 16;
#pragma unroll 1
                for (int k = 0; k < np; k++, c0 += 32) {
                    uint32_t v0[16], v1[16];
                    tmem_ld16(d_lane + c0, v0); tmem_ld16(d_lane + N + c0, v1);
                    tmem_ld_wait();
                    if (np - k == 1) release();
                    piece(c0, v0, v1);
                }
            }
            if (item + stride < nitems) scales_load(ep1, item + stride);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (DENSE && tid == 0) span_end(a.span);
    if (warp == 2) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tb, 512);
        if (lane == 0 && sh->abort_flag && a.err) *a.err = 1;
    }
}

template <int K, int MODE, bool FULL, int BW>
static void launch(cudaStream_t st, const ExpertArgs *a, const TMap4 *bmap) {
    const size_t smem = (size_t)UM_WSTAGES * UM_WBYTES + UmShape<BW>::BST * UmShape<BW>::BBYTES + 1024;
    static int sms = 0;
    if (!sms) {
        int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(expert_umma_kernel<K, MODE, FULL, BW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    if (a->fresh_maps || MODE == 2) launch_k(expert_umma_kernel<K, MODE, FULL, BW>, sms, 640, smem, st, *a, *bmap);
    else launch_pdl(expert_umma_kernel<K, MODE, FULL, BW>, sms, 640, smem, st, *a, *bmap);
    k_count_add(1);
}
// Blocks of 256 columns halve the hand-overs but leave the accumulators 256 columns of tensor memory instead of 320, which two items of more than 64 pairs do not share.
// A layer with blocks of 128 and of 256: 176 tokens 76.6 and 74.4 us, 301 83.1 and 82.0, 511 94.7 and 93.5, 843 101.2 and 99.8, 1300 119.5 and 119.4, 1500 127.2 and 127.7,
// 2048 148.9 and 155.0.  (As many tiles as there could be: the line lies at 1307 tokens.)
#define UM_WIDE_TILES (1300 * 8 / UMMA_TN + 256)
template <int K, int MODE, bool FULL>
static void launch_by_size(cudaStream_t st, const ExpertArgs *a, const TMap4 *bmap) {
    if (a->max_tiles <= 0) return;
    if (a->max_tiles <= UM_WIDE_TILES) launch<K, MODE, FULL, 2>(st, a, bmap); else launch<K, MODE, FULL, 1>(st, a, bmap);
}
extern "C" void k_gateup_umma(cudaStream_t st, const ExpertArgs *a, const TMap4 *bmap) {
    if (a->gu_dots) launch_by_size<2048, 0, true>(st, a, bmap); else launch_by_size<2048, 0, false>(st, a, bmap);
}
extern "C" void k_down_umma(cudaStream_t st, const ExpertArgs *a, const TMap4 *bmap) {
    if (a->dn_dots || a->rx_src) launch_by_size<512, 1, true>(st, a, bmap); else launch_by_size<512, 1, false>(st, a, bmap);
}
/* dense projections: tab[ex].ds / maps[ex].down of a matrix of 256 * a->dense_mblocks rows x 2048 columns, B rows = the tokens' int8 rows */
extern "C" void k_dense_umma(cudaStream_t st, const ExpertArgs *a, const TMap4 *bmap) { if (a->dense_n > 0) launch<2048, 2, false, 2>(st, a, bmap); }

// ---- rows of the per-token int8 matrix copied into pair (expert-grouped) order: the B operand the TMA can tile ----
__global__ void __launch_bounds__(256) gather_rows_kernel(const int8_t *__restrict__ src, const float *__restrict__ qs, const int *__restrict__ qsum, const int *__restrict__ rows,
                                                          int8_t *__restrict__ dst, float *__restrict__ dqs, int *__restrict__ dqsum, int np) {
    pdl_wait(); pdl_trigger();
    // 8 pairs per CTA: each thread moves one 16-byte piece of four rows, all four loads in flight together
    const int p0 = blockIdx.x * 8 + (threadIdx.x >> 7) * 4, c = threadIdx.x & 127;
    int r[4]; uint4 v[4];
#pragma unroll
    for (int k = 0; k < 4; k++) r[k] = p0 + k < np ? rows[p0 + k] : 0;
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = reinterpret_cast<const uint4 *>(src + (size_t)r[k] * 2048)[c];
#pragma unroll
    for (int k = 0; k < 4; k++) if (p0 + k < np) reinterpret_cast<uint4 *>(dst + (size_t)(p0 + k) * 2048)[c] = v[k];
#pragma unroll
    for (int k = 0; k < 4; k++) if (c == 32 * k && p0 + k < np) { dqs[p0 + k] = qs[r[k]]; dqsum[p0 + k] = qsum[r[k]]; }
}
extern "C" void k_gather_rows(cudaStream_t st, const int8_t *src, const float *qs, const int *qsum, const int *rows, int8_t *dst, float *dqs, int *dqsum, int np) {
    if (np <= 0) return;
    launch_pdl(gather_rows_kernel, (np + 7) / 8, 256, 0, st, src, qs, qsum, rows, dst, dqs, dqsum, np);
    k_count_add(1);
}

// The same from the tokens' side, for groupings made on the card (tp[8 b ..]: the slots of token b's pairs): a warp reads its token's row once, before the wait for the
// grouping (the row is older), and writes it eight times.  Reading the row
// again for every pair, behind the pair's token index: a layer of 301 / 843 / 2048 tokens 85.1 / 103.2 / 153.5 us, like this 84.2 / 101.7 / 151.3.
__global__ void __launch_bounds__(128) scatter_rows_kernel(const int8_t *__restrict__ src, const float *__restrict__ qs, const int *__restrict__ qsum, const int *__restrict__ tp,
                                                          int8_t *__restrict__ dst, float *__restrict__ dqs, int *__restrict__ dqsum, int nb) {
    const int lane = threadIdx.x & 31, b = blockIdx.x * 4 + (threadIdx.x >> 5);
    uint4 v[4]; float s = 0.0f; int t = 0;
    if (b < nb) {
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = __ldcg(reinterpret_cast<const uint4 *>(src + (size_t)b * 2048) + 32 * i + lane);
        s = __ldcg(qs + b); t = __ldcg(qsum + b);
    }
    pdl_wait(); pdl_trigger();
    if (b >= nb) return;
    const int4 a = reinterpret_cast<const int4 *>(tp + (size_t)b * 8)[0], c = reinterpret_cast<const int4 *>(tp + (size_t)b * 8)[1];
    const int slot[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
#pragma unroll
    for (int k = 0; k < 8; k++) {
        uint4 *d = reinterpret_cast<uint4 *>(dst + (size_t)slot[k] * 2048) + lane;
#pragma unroll
        for (int i = 0; i < 4; i++) d[32 * i] = v[i];
        if (lane == k) { dqs[slot[k]] = s; dqsum[slot[k]] = t; }
    }
}
extern "C" void k_scatter_rows(cudaStream_t st, const int8_t *src, const float *qs, const int *qsum, const int *tp, int8_t *dst, float *dqs, int *dqsum, int nb) {
    if (nb <= 0) return;
    launch_pdl(scatter_rows_kernel, (nb + 3) / 4, 128, 0, st, src, qs, qsum, tp, dst, dqs, dqsum, nb);
    k_count_add(1);
}

// The same behind a grouping that has left the places open (GroupArgs.place_base): pair k of token b goes to the start of its expert's pairs of b's word of 32 tokens
// plus the number of them in front of b.  The grouping runs in 8 or 16 CTAs, whose scattered stores these are otherwise; here they are spread over nb / 4.
__global__ void __launch_bounds__(128) place_rows_kernel(const GroupArgs g, const int8_t *__restrict__ src, const float *__restrict__ qs, const int *__restrict__ qsum,
                                                         int8_t *__restrict__ dst, float *__restrict__ dqs, int *__restrict__ dqsum) {
    const int lane = threadIdx.x & 31, k = lane & 7, b = blockIdx.x * 4 + (threadIdx.x >> 5);
    uint4 v[4]; float s = 0.0f, w = 0.0f; int t = 0, x = 0;
    if (b < g.nb) {                                              // older than the grouping: read before the wait
        x = __ldcg(g.top + (size_t)b * 8 + k); w = __ldcg(g.topw + (size_t)b * 8 + k);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = __ldcg(reinterpret_cast<const uint4 *>(src + (size_t)b * 2048) + 32 * i + lane);
        s = __ldcg(qs + b); t = __ldcg(qsum + b);
    }
    pdl_wait(); pdl_trigger();
    if (b >= g.nb) return;
    const size_t at = (size_t)(b >> 5) * 256 + x;
    const int slot = g.place_base[at] + __popc(g.place_bits[at] & ((1u << (b & 31)) - 1u));      // lanes 8 i + k: the same eight
    int rank = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) rank += __shfl_sync(0xffffffffu, slot, j) < slot;
    if (lane < 8) {
        g.utok[slot] = b; g.uw[slot] = w; if (g.uexp) g.uexp[slot] = x;
        g.slot[(size_t)b * 8 + k] = slot; g.tp[(size_t)b * 8 + rank] = slot;
        dqs[slot] = s; dqsum[slot] = t;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
        uint4 *d = reinterpret_cast<uint4 *>(dst + (size_t)__shfl_sync(0xffffffffu, slot, j) * 2048) + lane;
#pragma unroll
        for (int i = 0; i < 4; i++) d[32 * i] = v[i];
    }
}
extern "C" void k_place_rows(cudaStream_t st, const GroupArgs *g, const int8_t *src, const float *qs, const int *qsum, int8_t *dst, float *dqs, int *dqsum) {
    if (g->nb <= 0) return;
    launch_pdl(place_rows_kernel, (g->nb + 3) / 4, 128, 0, st, *g, src, qs, qsum, dst, dqs, dqsum);
    k_count_add(1);
}
