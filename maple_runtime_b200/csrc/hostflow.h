/* hostflow.h -- rows between a caller's host buffers and the card, in chunks, with a computation per chunk in between. */
#ifndef MAPLE_HOSTFLOW_H
#define MAPLE_HOSTFLOW_H
#include <stddef.h>
#include <stdint.h>
#include <cuda_runtime_api.h>

#define FLOW_OUTS 3
typedef struct {
    int rows;                  /* tokens */
    int chunk;                 /* largest number of tokens per chunk (0: chosen by the rows' size) */
    /* in: `src` rows of `row` bytes.  quant = 0: they go to `dst` unchanged.  quant = 1: rows of 2048 fp32 values become int8 rows on the way
     * (hostio.h), dst = int8 rows; their scales and sums go to host arrays (hqs, hqsum) and, with dst_qs set, to dst_qs[row] and
     * dst_qs[row + qs_pitch] on the card. */
    const void *src; size_t row; void *dst; int quant;
    float *hqs; int *hqsum; float *dst_qs; size_t qs_pitch;
    int (*compute)(void *ctx, int row0, int n); void *ctx;      /* queues the chunk's kernels on the library's stream; 0 = queued */
    int (*meanwhile)(void *mctx); void *mctx;                     /* the calling thread's own work while the rows are being read; non-zero = give up */
    /* out: `nout` arrays of `orow` bytes per row on the card, to host arrays */
    int nout; const void *osrc[FLOW_OUTS]; void *odst[FLOW_OUTS]; size_t orow[FLOW_OUTS];
} Flow;
/* Runs the flow on stream st (chunks beyond the first also on the flow's own copy streams).  With outputs it returns when they are
 * complete; without, when the caller's source has been read (the copies to the card may still be under way on st).  0, or a CUDA error. */
cudaError_t flow_run(Flow *f, cudaStream_t st);
#endif
