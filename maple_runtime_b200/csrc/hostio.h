/* hostio.h -- the host side of a call that takes pageable buffers: a small pool of helper threads and the row work it does. */
#ifndef MAPLE_HOSTIO_H
#define MAPLE_HOSTIO_H
#include <stddef.h>
#include <stdint.h>

/* A job is fn(arg, piece) for piece = 0..pieces-1, in any order, on any of the pool's threads and on the caller's (hio_help).  One
 * thread submits; jobs are started in the order of their submission.  arg must live until hio_done. */
typedef void (*hio_fn)(void *arg, int piece);
/* around a call that uses the pool (they nest; the outermost one's kind counts): its threads, once it has woken them, stay awake to its end, and for
 * a moment longer where a call of that kind is usually followed by another at once */
enum { HIO_ROWS, HIO_LAYER, HIO_PLUGIN, HIO_ROPE, HIO_QKV, HIO_O, HIO_KINDS };
void hio_begin(int kind);
void hio_end(void);
unsigned hio_submit(hio_fn fn, void *arg, int pieces);
int hio_done(unsigned ticket);
int hio_help(void);                       /* runs one unclaimed piece; 0 = there is none */
void hio_wait(unsigned ticket);           /* helps until the job is done */

/* prep of maple.c:184-194 for rows of 2048 values: per-row absmax int8, scale and code sum, the bits of the device's norm_prep_kernel */
void hio_quant_rows(const float *x, int rows, int8_t *q, float *qs, int *qsum);
/* memcpy whose stores go past the caches when `stream` is set (a destination that is larger than them) */
void hio_copy(void *dst, const void *src, size_t bytes, int stream);
/* memcpy of a large buffer by the pool (by the calling thread alone below HIO_POOL_BYTES, where it is done before a helper has seen the job) */
#define HIO_POOL_BYTES (160u << 10)
#define HIO_PIECE_BYTES (24u << 10)       /* a thread's unit of work: about 1.5 us */
void hio_copy_shared(void *dst, const void *src, size_t bytes);
#endif
