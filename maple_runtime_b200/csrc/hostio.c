/* hostio.c -- helper threads for the calls that take pageable host buffers.
 *
 * The driver moves a pageable buffer through its own staging with one thread: 20 GB/s for 16.8 MB (a 2048-token chunk of hidden rows,
 * 841 us), against 54 GB/s for page-locked memory.  One core copies at 18.5 GB/s from memory, four at 72 GB/s, so a few threads that
 * fill (and empty) page-locked slots keep the link busy.  The threads are started by the first call that has enough work for them, stay
 * awake from the beginning of a call to its end (the card's part lies between the filling and the emptying) and sleep when it returns: the
 * cores are the host's again.  Only where the last call of the same kind was followed by another within TAIL_CYCLES do they wait so long for
 * the next (being woken costs a call 4 us: the sides of attention, 64 tokens, 5140 us for 72 calls without, 4850 with it).  Without them (one
 * core, a forked child) the calling thread does every piece itself.
 *
 * What they cost a host on 16 cores, and its threads them (2048-token plug-in calls, 5 helpers).  A host that computes on all cores right after
 * a call, 285 us alone: 295 us; 570 when the helpers spun for another 400 us, 550 for 20 (a worker that is woken meanwhile is put behind another
 * one).  A host whose 15 workers never sleep: 1.8 ms per call (mean) with helpers that offer their core now and then while they wait, 2.1 without
 * helpers, 2.7 to 7.2 with helpers that only spin: one that has used up its time slice so is stopped in the middle of a piece.  A host that
 * leaves cores free: 0.73 ms with any of them. */
#define _GNU_SOURCE
#include <immintrin.h>
#include <pthread.h>
#include <sched.h>
#include <stdatomic.h>
#include <string.h>
#include "hostio.h"

#define NJOB 64                           /* jobs outstanding at most; the submitter helps while its slot is still in use */
/* Two 2048-token plug-in calls on 16 cores take 1.89 ms with 3 helpers, 1.68 with 5, 1.54 with 7; but every thread of a process makes its
 * munmap calls slower (the page tables are shared): a host that maps and frees its arrays loses with 7 what it gains */
#define MAXHELP 5
#define YIELD_EVERY 256                   /* polls, about 10 us */
#define TAIL_CYCLES 125000ull             /* about 50 us */
#define CALL_CYCLES 50000000ull           /* about 20 ms without a piece: the call waits for something else */

/* state of a slot: sequence number of its job (24 bits) | pieces (20) | next piece (20); a claim is one compare-and-swap of the whole word,
 * so a thread that was delayed can never take a piece of the job that has since moved into the slot */
#define ST(seq, n, i) (((uint64_t)((seq) & 0xFFFFFFu) << 40) | ((uint64_t)(n) << 20) | (uint64_t)(i))
#define ST_SEQ(v) ((unsigned)((v) >> 40))
#define ST_N(v) ((unsigned)((v) >> 20) & 0xFFFFFu)
#define ST_I(v) ((unsigned)(v) & 0xFFFFFu)
static struct { _Atomic uint64_t state; atomic_int left; hio_fn fn; void *arg; } J[NJOB] __attribute__((aligned(64)));
static atomic_uint head, tail;            /* jobs head..tail-1 may have unclaimed pieces */
static pthread_t th[MAXHELP];
static int nth = -1;                      /* -1: not started yet */
static atomic_int stop, sleepers;
static struct { atomic_int in_call, tail_on; } now __attribute__((aligned(64)));      /* written by the caller only, polled by the helpers */
static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static pthread_cond_t cv = PTHREAD_COND_INITIALIZER;

int hio_help(void) {
    for (;;) {
        const unsigned h = atomic_load_explicit(&head, memory_order_acquire);
        if (h == atomic_load_explicit(&tail, memory_order_acquire)) return 0;
        uint64_t v = atomic_load_explicit(&J[h % NJOB].state, memory_order_acquire);
        if (ST_SEQ(v) != (h & 0xFFFFFFu)) continue;                 /* head has moved on */
        if (ST_I(v) >= ST_N(v)) { unsigned e = h; atomic_compare_exchange_strong(&head, &e, h + 1); continue; }
        if (!atomic_compare_exchange_weak_explicit(&J[h % NJOB].state, &v, v + 1, memory_order_acq_rel, memory_order_relaxed)) continue;
        J[h % NJOB].fn(J[h % NJOB].arg, (int)ST_I(v));
        atomic_fetch_sub_explicit(&J[h % NJOB].left, 1, memory_order_release);
        return 1;
    }
}
static void *helper(void *p) {
    (void)p;
    uint64_t t0 = __rdtsc(); unsigned polls = 0; int was = 0;
    while (!atomic_load_explicit(&stop, memory_order_relaxed)) {
        if (hio_help()) { t0 = __rdtsc(); continue; }
        const int busy = atomic_load_explicit(&now.in_call, memory_order_relaxed);
        if (busy != was) { was = busy; t0 = __rdtsc(); }
        if (__rdtsc() - t0 < (busy ? CALL_CYCLES : atomic_load_explicit(&now.tail_on, memory_order_relaxed) ? TAIL_CYCLES : 0)) {
            if (++polls % YIELD_EVERY) _mm_pause(); else sched_yield();
            continue;
        }
        pthread_mutex_lock(&mu);
        atomic_fetch_add(&sleepers, 1);
        while (atomic_load(&head) == atomic_load(&tail) && !atomic_load(&stop)) pthread_cond_wait(&cv, &mu);
        atomic_fetch_sub(&sleepers, 1);
        pthread_mutex_unlock(&mu);
        t0 = __rdtsc();
    }
    return NULL;
}
static void wake(void) { pthread_mutex_lock(&mu); pthread_cond_broadcast(&cv); pthread_mutex_unlock(&mu); }
static void forked(void) { nth = 0; atomic_store(&sleepers, 0); }   /* a child has none of the threads */
static void start(void) {
    cpu_set_t cs;
    int cores = sched_getaffinity(0, sizeof cs, &cs) == 0 ? CPU_COUNT(&cs) : 1, want = cores / 2 - 1;
    if (want > MAXHELP) want = MAXHELP;
    nth = 0;
    pthread_atfork(NULL, NULL, forked);
    while (nth < want && pthread_create(&th[nth], NULL, helper, NULL) == 0) nth++;
}
__attribute__((destructor)) static void finish_threads(void) {
    if (nth <= 0) return;
    atomic_store(&stop, 1); wake();
    for (int i = 0; i < nth; i++) pthread_join(th[i], NULL);
    nth = 0;
}
static int depth, kind_of_last, followed[HIO_KINDS];      /* followed: by kind of call, another one began within TAIL_CYCLES of its end */
static uint64_t ended;
void hio_begin(int kind) {
    if (depth++) return;
    followed[kind_of_last] = __rdtsc() - ended < TAIL_CYCLES; kind_of_last = kind;
    atomic_store_explicit(&now.in_call, 1, memory_order_release);
}
void hio_end(void) {
    if (--depth) return;
    ended = __rdtsc();
    if (atomic_load_explicit(&now.tail_on, memory_order_relaxed) != followed[kind_of_last]) atomic_store_explicit(&now.tail_on, followed[kind_of_last], memory_order_release);
    atomic_store_explicit(&now.in_call, 0, memory_order_release);
}
unsigned hio_submit(hio_fn fn, void *arg, int pieces) {
    if (nth < 0) start();
    const unsigned t = atomic_load_explicit(&tail, memory_order_relaxed);
    while (atomic_load_explicit(&J[t % NJOB].left, memory_order_acquire) > 0) if (!hio_help()) _mm_pause();
    while (t - atomic_load(&head) >= NJOB) hio_help();              /* the slot's old job is done but not yet passed */
    J[t % NJOB].fn = fn; J[t % NJOB].arg = arg;
    atomic_store_explicit(&J[t % NJOB].left, pieces, memory_order_relaxed);
    atomic_store_explicit(&J[t % NJOB].state, ST(t, pieces, 0), memory_order_release);
    atomic_store(&tail, t + 1);                                     /* ordered before the read of sleepers, as a sleeper's count is before its read of tail */
    if (atomic_load(&sleepers)) wake();
    return t;
}
int hio_done(unsigned t) {
    if (ST_SEQ(atomic_load_explicit(&J[t % NJOB].state, memory_order_acquire)) != (t & 0xFFFFFFu)) return 1;   /* the slot has a later job */
    return atomic_load_explicit(&J[t % NJOB].left, memory_order_acquire) == 0;
}
void hio_wait(unsigned t) { while (!hio_done(t)) if (!hio_help()) _mm_pause(); }

/* ---- prep (maple.c:184-194) ---------------------------------------------------------------------------------------
 * s = max|x| / 127 (1 for a zero row), q = round-half-even(x * (1 / s)), qsum = sum q.  What the device does for values that are no
 * number or out of an int's range (conversion saturates, NaN -> 0) is kept by the scalar form, which takes the rows whose 1 / s is not
 * finite (a maximum below 127 times the smallest subnormal, or infinite) or that hold a NaN. */
static int cvt_rn(float t) {              /* cvt.rni.s32.f32 */
    if (t != t) return 0;
    if (t >= 2147483648.0f) return 2147483647;
    if (t < -2147483648.0f) return -2147483647 - 1;
    return _mm_cvtss_si32(_mm_set_ss(t));
}
static void quant_row_scalar(const float *x, int8_t *q, float *qs, int *qsum) {
    float mx = 0.0f;
    for (int i = 0; i < 2048; i++) { const float a = __builtin_fabsf(x[i]); if (a > mx) mx = a; }
    const float s = mx > 0.0f ? mx / 127.0f : 1.0f, inv = 1.0f / s;
    unsigned tot = 0;
    for (int i = 0; i < 2048; i++) { const int v = cvt_rn(x[i] * inv); q[i] = (int8_t)(v & 0xFF); tot += (unsigned)v; }
    *qs = s; *qsum = (int)tot;
}
__attribute__((target("avx2"))) static int quant_row_avx2(const float *x, int8_t *q, float *qs, int *qsum) {
    const __m256 sign = _mm256_set1_ps(-0.0f);
    __m256 m0 = _mm256_setzero_ps(), m1 = m0, m2 = m0, m3 = m0, nan = m0;
    for (int i = 0; i < 2048; i += 32) {
        const __m256 a = _mm256_loadu_ps(x + i), b = _mm256_loadu_ps(x + i + 8), c = _mm256_loadu_ps(x + i + 16), d = _mm256_loadu_ps(x + i + 24);
        nan = _mm256_or_ps(nan, _mm256_or_ps(_mm256_cmp_ps(a, b, _CMP_UNORD_Q), _mm256_cmp_ps(c, d, _CMP_UNORD_Q)));
        m0 = _mm256_max_ps(_mm256_andnot_ps(sign, a), m0); m1 = _mm256_max_ps(_mm256_andnot_ps(sign, b), m1);
        m2 = _mm256_max_ps(_mm256_andnot_ps(sign, c), m2); m3 = _mm256_max_ps(_mm256_andnot_ps(sign, d), m3);
    }
    if (_mm256_movemask_ps(nan)) return 0;
    m0 = _mm256_max_ps(_mm256_max_ps(m0, m1), _mm256_max_ps(m2, m3));
    __m128 m = _mm_max_ps(_mm256_castps256_ps128(m0), _mm256_extractf128_ps(m0, 1));
    m = _mm_max_ps(m, _mm_movehl_ps(m, m)); m = _mm_max_ss(m, _mm_shuffle_ps(m, m, 1));
    const float mx = _mm_cvtss_f32(m), s = mx > 0.0f ? mx / 127.0f : 1.0f, inv = 1.0f / s;
    if (!(inv < 3.4e38f) || !(inv > 0.0f)) return 0;
    const __m256 vi = _mm256_set1_ps(inv);
    const __m256i order = _mm256_setr_epi32(0, 4, 1, 5, 2, 6, 3, 7), ones = _mm256_set1_epi16(1), one8 = _mm256_set1_epi8(1);
    __m256i tot = _mm256_setzero_si256();
    for (int i = 0; i < 2048; i += 32) {      /* |x * inv| <= 127.0001: the saturating packs change nothing */
        const __m256i a = _mm256_cvtps_epi32(_mm256_mul_ps(_mm256_loadu_ps(x + i), vi)), b = _mm256_cvtps_epi32(_mm256_mul_ps(_mm256_loadu_ps(x + i + 8), vi));
        const __m256i c = _mm256_cvtps_epi32(_mm256_mul_ps(_mm256_loadu_ps(x + i + 16), vi)), d = _mm256_cvtps_epi32(_mm256_mul_ps(_mm256_loadu_ps(x + i + 24), vi));
        const __m256i p = _mm256_permutevar8x32_epi32(_mm256_packs_epi16(_mm256_packs_epi32(a, b), _mm256_packs_epi32(c, d)), order);
        _mm256_storeu_si256((__m256i *)(q + i), p);
        /* the next row, on its way while this one is converted (a prefetch past the last row's end is no access) */
        _mm_prefetch((const char *)(x + 2048 + i), _MM_HINT_T0); _mm_prefetch((const char *)(x + 2048 + i + 16), _MM_HINT_T0);
        tot = _mm256_add_epi32(tot, _mm256_madd_epi16(_mm256_maddubs_epi16(one8, p), ones));
    }
    int t[8]; _mm256_storeu_si256((__m256i *)t, tot);
    *qs = s; *qsum = t[0] + t[1] + t[2] + t[3] + t[4] + t[5] + t[6] + t[7];
    return 1;
}
void hio_quant_rows(const float *x, int rows, int8_t *q, float *qs, int *qsum) {
    static int avx2 = -1;
    if (avx2 < 0) avx2 = __builtin_cpu_supports("avx2") != 0;
    const unsigned csr = _mm_getcsr(); _mm_setcsr(0x1F80);          /* round to nearest, subnormals kept, whatever the host program runs with */
    for (int r = 0; r < rows; r++)
        if (!avx2 || !quant_row_avx2(x + (size_t)r * 2048, q + (size_t)r * 2048, qs + r, qsum + r)) quant_row_scalar(x + (size_t)r * 2048, q + (size_t)r * 2048, qs + r, qsum + r);
    _mm_setcsr(csr);
}
__attribute__((target("avx2"))) static void copy_stream(uint8_t *d, const uint8_t *s, size_t n) {
    size_t pre = (32 - ((uintptr_t)d & 31)) & 31;
    if (pre > n) pre = n;
    memcpy(d, s, pre); d += pre; s += pre; n -= pre;
    for (; n >= 128; n -= 128, d += 128, s += 128) {
        _mm_prefetch((const char *)s + 2048, _MM_HINT_T0); _mm_prefetch((const char *)s + 2112, _MM_HINT_T0);
        const __m256i a = _mm256_loadu_si256((const __m256i *)s), b = _mm256_loadu_si256((const __m256i *)(s + 32));
        const __m256i c = _mm256_loadu_si256((const __m256i *)(s + 64)), e = _mm256_loadu_si256((const __m256i *)(s + 96));
        _mm256_stream_si256((__m256i *)d, a); _mm256_stream_si256((__m256i *)(d + 32), b);
        _mm256_stream_si256((__m256i *)(d + 64), c); _mm256_stream_si256((__m256i *)(d + 96), e);
    }
    memcpy(d, s, n);
    _mm_sfence();
}
void hio_copy(void *dst, const void *src, size_t bytes, int stream) {
    static int avx2 = -1;
    if (avx2 < 0) avx2 = __builtin_cpu_supports("avx2") != 0;
    if (stream && avx2) copy_stream(dst, src, bytes); else memcpy(dst, src, bytes);
}
typedef struct { uint8_t *d; const uint8_t *s; size_t n; } Shared;
static void shared_piece(void *p, int i) {
    const Shared *c = p;
    const size_t a = (size_t)i * HIO_PIECE_BYTES, n = c->n - a < HIO_PIECE_BYTES ? c->n - a : HIO_PIECE_BYTES;
    memcpy(c->d + a, c->s + a, n);
}
void hio_copy_shared(void *dst, const void *src, size_t bytes) {
    if (bytes < HIO_POOL_BYTES) { memcpy(dst, src, bytes); return; }
    Shared c = {dst, src, bytes};
    hio_wait(hio_submit(shared_piece, &c, (int)((bytes + HIO_PIECE_BYTES - 1) / HIO_PIECE_BYTES)));
}
