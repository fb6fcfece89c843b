// k_tables.cu -- the tables of a reference-shaped call from one page-locked host block to their places on the card, sm_100a.
//
// Bound by the link: the block (330 KB at 2048 tokens) is read in place, 16 bytes per thread and load, all segments at once.  One launch
// instead of twelve copies of pageable memory and a wait (about 120 us of the call before; 10 us now).
#include <cuda_runtime.h>
#include <stdint.h>
#include "kernels.h"
#include "launch.cuh"
#include "umma.cuh"

extern "C" void k_count_add(long n);

__global__ void __launch_bounds__(256) tables_kernel(const __grid_constant__ TableSegs t) {
    pdl_trigger();                                                       // a successor launched programmatically waits for the whole kernel all the same
    const unsigned words = t.words[blockIdx.y], step = gridDim.x * 256;
    const uint32_t *src = static_cast<const uint32_t *>(t.src[blockIdx.y]);
    uint32_t *dst = static_cast<uint32_t *>(t.dst[blockIdx.y]);
    const bool wide = ((uintptr_t)dst & 15) == 0;                       // the sources are 16-byte aligned
    const unsigned vecs = wide ? words / 4 : 0;
    for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < vecs; i += step) reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
    for (unsigned i = vecs * 4 + blockIdx.x * 256 + threadIdx.x; i < words; i += step) dst[i] = src[i];
    tma_release_maps();                                                  // some segments are tensor maps
}
extern "C" void k_tables(cudaStream_t st, const TableSegs *t) {
    if (t->n <= 0) return;
    unsigned most = 1;
    for (int i = 0; i < t->n; i++) if (t->words[i] > most) most = t->words[i];
    unsigned ctas = (most / 4 + 255) / 256;
    if (ctas < 1) ctas = 1;
    if (ctas > 64) ctas = 64;
    launch_k(tables_kernel, dim3(ctas, (unsigned)t->n), 256, 0, st, *t);
    k_count_add(1);
}

__global__ void __launch_bounds__(256) rows_kernel(uint4 *__restrict__ dst, const uint4 *__restrict__ src, unsigned n) {
    const unsigned i = blockIdx.x * 256 + threadIdx.x;
    pdl_wait(); pdl_trigger();
    if (i < n) dst[i] = src[i];
}
extern "C" void k_rows(cudaStream_t st, void *dst, const void *src, size_t bytes) {
    const unsigned n = (unsigned)(bytes / 16);
    if (!n) return;
    launch_pdl(rows_kernel, (n + 255) / 256, 256, 0, st, static_cast<uint4 *>(dst), static_cast<const uint4 *>(src), n);
    k_count_add(1);
}

__global__ void __launch_bounds__(32) span_sum_kernel(unsigned long long *span, int n, unsigned long long *ns) {
    unsigned long long sum = 0;
    for (int i = threadIdx.x; i < n; i += 32) {
        const unsigned long long start = ~span[2 * i], end = span[2 * i + 1];
        if (end > start) sum += end - start;
        span[2 * i] = span[2 * i + 1] = 0;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (threadIdx.x == 0) *ns = sum;
}
extern "C" void k_span_sum(cudaStream_t st, unsigned long long *span, int n, unsigned long long *ns) {
    launch_k(span_sum_kernel, 1, 32, 0, st, span, n, ns);
    k_count_add(1);
}
