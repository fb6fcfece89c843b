/* hostflow.c -- moves rows between pageable (or page-locked) host buffers and the card.
 *
 * A chunk's life: helper threads fill a page-locked slot from the caller's rows -> copy to the card -> the chunk's kernels -> copy into a
 * page-locked slot -> helper threads empty it into the caller's rows.  The stages of neighbouring chunks overlap: the link carries both
 * directions at once (54 GB/s each way measured on page-locked memory) while the host's cores copy at 70 GB/s and more.  Page-locked
 * caller buffers skip their slot.  The calling thread drives the chunks and does pieces of the host's work while it waits. */
#include <immintrin.h>
#include <string.h>
#include "hostflow.h"
#include "hostio.h"

#define SLOTS 6
#define SLOT_BYTES (3u << 20)             /* 256 tokens of the widest row (12 KB) */
#define CHUNK_MIN (1024u << 10)           /* a chunk costs about 10 us of calls into the driver; 300 tokens through the plug-in call 589 us at 512 KB, 566 at 1 MB */
#define STREAM_BYTES (8u << 20)           /* results larger than this are stored past the caches */

typedef struct { Flow *f; int slot, row0, n, per; } Part;
static struct {
    int ready;
    uint8_t *in[SLOTS], *out[SLOTS];
    cudaStream_t sin, sout;
    cudaEvent_t begun, in_done[SLOTS], ran[SLOTS], out_done[SLOTS];
    int in_used[SLOTS];                   /* in_done[] has been recorded and not yet seen complete */
    Part fill[SLOTS], drain[SLOTS];
} FL;

static cudaError_t setup(void) {
    if (FL.ready) return cudaSuccess;
    cudaError_t e = cudaStreamCreateWithFlags(&FL.sin, cudaStreamNonBlocking);
    if (!e) e = cudaStreamCreateWithFlags(&FL.sout, cudaStreamNonBlocking);
    if (!e) e = cudaEventCreateWithFlags(&FL.begun, cudaEventDisableTiming);
    for (int s = 0; s < SLOTS && !e; s++) {
        e = cudaHostAlloc((void **)&FL.in[s], SLOT_BYTES, cudaHostAllocDefault);
        if (!e) e = cudaHostAlloc((void **)&FL.out[s], SLOT_BYTES, cudaHostAllocDefault);
        if (!e) e = cudaEventCreateWithFlags(&FL.in_done[s], cudaEventDisableTiming);
        if (!e) e = cudaEventCreateWithFlags(&FL.ran[s], cudaEventDisableTiming);
        if (!e) e = cudaEventCreateWithFlags(&FL.out_done[s], cudaEventDisableTiming);
    }
    FL.ready = e == cudaSuccess;
    return e;
}
static int page_locked(const void *p, size_t bytes) {
    struct cudaPointerAttributes a;
    const char *q = p;
    if (!bytes) return 0;
    for (int i = 0; i < 2; i++, q += bytes - 1)
        if (cudaPointerGetAttributes(&a, q) != cudaSuccess) { cudaGetLastError(); return 0; } else if (a.type != cudaMemoryTypeHost) return 0;
    return 1;
}
static size_t in_row(const Flow *f) { return f->quant ? 2048 + 8 : f->row; }
static void fill_piece(void *p, int i) {
    const Part *c = p; Flow *f = c->f;
    const int a = i * c->per, n = c->n - a < c->per ? c->n - a : c->per;
    const uint8_t *src = (const uint8_t *)f->src + (size_t)(c->row0 + a) * f->row;
    if (f->quant) hio_quant_rows((const float *)src, n, (int8_t *)FL.in[c->slot] + (size_t)a * 2048, f->hqs + c->row0 + a, f->hqsum + c->row0 + a);
    else memcpy(FL.in[c->slot] + (size_t)a * f->row, src, (size_t)n * f->row);
}
static void drain_piece(void *p, int i) {
    const Part *c = p; Flow *f = c->f;
    const int a = i * c->per, n = c->n - a < c->per ? c->n - a : c->per;
    const uint8_t *src = FL.out[c->slot];
    for (int k = 0; k < f->nout; k++) {
        const size_t r = f->orow[k];
        hio_copy((uint8_t *)f->odst[k] + (size_t)(c->row0 + a) * r, src + (size_t)a * r, (size_t)n * r, (size_t)f->rows * r > STREAM_BYTES);
        src += (size_t)c->n * r;
    }
}
/* a chunk's host work: at once when it is small, else as a job of the pool */
static int start_part(Part *c, hio_fn fn, size_t row_bytes, unsigned *ticket) {
    const size_t bytes = (size_t)c->n * row_bytes;
    c->per = bytes < HIO_POOL_BYTES ? c->n : (int)(HIO_PIECE_BYTES / row_bytes) + 1;
    const int pieces = (c->n + c->per - 1) / c->per;
    if (pieces <= 1) { fn(c, 0); return 0; }
    *ticket = hio_submit(fn, c, pieces);
    return 1;
}
static cudaError_t copy_in(Flow *f, int direct, int slot, int row0, int n, cudaStream_t st) {
    const size_t row = f->quant ? 2048 : f->row;
    const void *src = direct ? (const uint8_t *)f->src + (size_t)row0 * row : FL.in[slot];
    cudaError_t e = cudaMemcpyAsync((uint8_t *)f->dst + (size_t)row0 * row, src, (size_t)n * row, cudaMemcpyHostToDevice, st);
    if (!e && f->quant && f->dst_qs) {      /* the chunk's scales and sums travel in the slot, behind its rows */
        uint8_t *tail = FL.in[slot] + (size_t)n * 2048;
        memcpy(tail, f->hqs + row0, (size_t)n * 4); memcpy(tail + (size_t)n * 4, f->hqsum + row0, (size_t)n * 4);
        e = cudaMemcpy2DAsync(f->dst_qs + row0, f->qs_pitch * 4, tail, (size_t)n * 4, (size_t)n * 4, 2, cudaMemcpyHostToDevice, st);
    }
    return e;
}
static cudaError_t copy_out(Flow *f, int direct, int slot, int row0, int n, cudaStream_t st) {
    uint8_t *dst = FL.out[slot];
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < f->nout && !e; k++) {
        const size_t r = f->orow[k];
        e = cudaMemcpyAsync(direct ? (uint8_t *)f->odst[k] + (size_t)row0 * r : dst, (const uint8_t *)f->osrc[k] + (size_t)row0 * r, (size_t)n * r, cudaMemcpyDeviceToHost, st);
        dst += (size_t)n * r;
    }
    return e;
}
static cudaError_t slot_free(int s, int wait) {       /* cudaSuccess: the slot's last copy to the card has been made */
    if (!FL.in_used[s]) return cudaSuccess;
    const cudaError_t e = wait ? cudaEventSynchronize(FL.in_done[s]) : cudaEventQuery(FL.in_done[s]);
    if (e == cudaSuccess) FL.in_used[s] = 0;
    return e;
}

static cudaError_t run(Flow *f, cudaStream_t st) {
    cudaError_t e = setup();
    if (e) return e;
    size_t widest = f->src ? in_row(f) : 1, orow = 0;
    for (int k = 0; k < f->nout; k++) orow += f->orow[k];
    if (orow > widest) widest = orow;
    /* about seven chunks (the first one's filling and the last one's emptying overlap with nothing), none under CHUNK_MIN */
    const size_t host_row = f->src && f->row > orow ? f->row : orow, share = (size_t)f->rows * host_row / 7;
    const int most = (int)(SLOT_BYTES / widest);
    int chunk = (int)((share > CHUNK_MIN ? share : CHUNK_MIN) / host_row) + 1;
    if (chunk > most) chunk = most;
    if (f->chunk && f->chunk < chunk) chunk = f->chunk;
    const int nch = (f->rows + chunk - 1) / chunk;
    const int din = f->src && !f->quant && page_locked(f->src, (size_t)f->rows * f->row);
    int dout = f->nout > 0;
    for (int k = 0; k < f->nout; k++) dout = dout && page_locked(f->odst[k], (size_t)f->rows * f->orow[k]);
    unsigned tin[SLOTS] = {0}, tout[SLOTS] = {0}; int jin[SLOTS] = {0}, jout[SLOTS] = {0};      /* a slot's job and whether it is still to be waited for */
    const cudaStream_t sin = nch > 1 ? FL.sin : st, sout = nch > 1 ? FL.sout : st;
    if (nch > 1 && f->src) { e = cudaEventRecord(FL.begun, st); if (!e) e = cudaStreamWaitEvent(sin, FL.begun, 0); }
    int filled = 0, issued = 0, arrived = 0, drained = 0;     /* chunks that reached: host fill started, card work queued, result on the host, result handed over */
    while (!e && (f->nout ? drained : issued) < nch) {
        int moved = 0;
        if (f->src && filled < nch && filled - issued < SLOTS) {
            const int s = filled % SLOTS;
            const cudaError_t q = din ? cudaSuccess : slot_free(s, 0);
            if (q == cudaSuccess) {
                Part *c = &FL.fill[s]; c->f = f; c->slot = s; c->row0 = filled * chunk; c->n = f->rows - c->row0 < chunk ? f->rows - c->row0 : chunk;
                jin[s] = din ? 0 : start_part(c, fill_piece, f->quant ? 8192 : f->row, &tin[s]);
                filled++; moved = 1;
            } else if (q != cudaErrorNotReady) { e = q; break; }
        }
        if (f->meanwhile && (filled == nch || filled == SLOTS)) {      /* the helpers have the rows: the calling thread's own part */
            if (f->meanwhile(f->mctx)) { e = cudaErrorInvalidValue; break; }
            f->meanwhile = NULL;
        }
        if (issued < nch && (!f->src || (issued < filled && (!jin[issued % SLOTS] || hio_done(tin[issued % SLOTS])))) && (!f->nout || issued - drained < SLOTS)) {
            const int s = issued % SLOTS, row0 = issued * chunk, n = f->rows - row0 < chunk ? f->rows - row0 : chunk;
            jin[s] = 0;
            if (f->src) {
                e = copy_in(f, din, s, row0, n, sin);
                if (!e && (nch > 1 || !f->nout) ) { e = cudaEventRecord(FL.in_done[s], sin); FL.in_used[s] = !din; if (!e && sin != st) e = cudaStreamWaitEvent(st, FL.in_done[s], 0); }
            }
            if (!e && f->compute && f->compute(f->ctx, row0, n)) e = cudaErrorUnknown;
            if (!e && f->nout) {
                if (sout != st) { e = cudaEventRecord(FL.ran[s], st); if (!e) e = cudaStreamWaitEvent(sout, FL.ran[s], 0); }
                if (!e) e = copy_out(f, dout, s, row0, n, sout);
                if (!e && nch > 1) e = cudaEventRecord(FL.out_done[s], sout);
            }
            if (e) break;
            issued++; moved = 1;
        }
        if (arrived < issued && f->nout) {
            const int s = arrived % SLOTS;
            const cudaError_t q = nch > 1 ? cudaEventQuery(FL.out_done[s]) : cudaStreamSynchronize(st);
            if (q == cudaSuccess) {
                Part *c = &FL.drain[s]; c->f = f; c->slot = s; c->row0 = arrived * chunk; c->n = f->rows - c->row0 < chunk ? f->rows - c->row0 : chunk;
                jout[s] = dout ? 0 : start_part(c, drain_piece, orow, &tout[s]);
                arrived++; moved = 1;
            } else if (q != cudaErrorNotReady) { e = q; break; }
        }
        if (drained < arrived && (!jout[drained % SLOTS] || hio_done(tout[drained % SLOTS]))) { jout[drained % SLOTS] = 0; drained++; moved = 1; }
        if (!moved && !hio_help()) _mm_pause();
    }
    for (int s = 0; s < SLOTS; s++) {                          /* only after an error: the parts and the caller's rows are still in use */
        if (jin[s]) hio_wait(tin[s]);
        if (jout[s]) hio_wait(tout[s]);
    }
    return e;
}
cudaError_t flow_run(Flow *f, cudaStream_t st) { hio_begin(HIO_ROWS); const cudaError_t e = run(f, st); hio_end(); return e; }
