/* ff_copy.c -- a copy of pageable memory into a page-locked buffer, shared among a few threads.
 *
 * One thread moves 16-18 GB/s on the measured host and four move 56 GB/s, what a PCIe 5 x16 link takes; the driver's own
 * staging of a pageable copy is one thread (12 GB/s at 150 MB).  The job is cut into pieces that whoever is awake
 * claims under a mutex, the caller included: helpers that are slow to wake cost nothing, they find less to do.
 * A helper looks for the next job for some 50 us before it sleeps, which spans the gap between two chunks of a call.
 *
 * A copy whose destination a device reads next uses streaming stores: lines left dirty in the caches of several cores
 * slow the copy engine's reads down (2.56 MB, copied by one thread and sent: 259-309 us with plain stores, 199-231 with
 * streaming ones; the driver's own staging 242).
 */
#define _GNU_SOURCE
#include "ff_copy.h"

#include <pthread.h>
#include <sched.h>
#include <signal.h>
#include <stdatomic.h>
#include <stdlib.h>
#include <string.h>
#include <time.h>
#include <unistd.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#define FF_COPY_MAX_HELPERS 3
#define FF_COPY_PIECE ((size_t)128 << 10)
#define FF_COPY_MIN_SHARED ((size_t)512 << 10)
#define FF_COPY_SPIN_NS 50000

struct ff_copy_pool {
    pthread_mutex_t mu;
    pthread_cond_t wake;
    char* dst;               /* the job, under mu */
    const char* src;
    size_t bytes, next;      /* next: first byte nobody has claimed */
    _Atomic size_t open;     /* bytes nobody has claimed, readable without the mutex */
    _Atomic size_t left;     /* bytes not copied yet */
    int streaming;           /* of the job */
    int wanted, started, stop, sleeping;
    pthread_t th[FF_COPY_MAX_HELPERS];
    pid_t owner;             /* a process forked from the owner has no helpers, and the locks as the fork found them */
};

static void relax(void)
{
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#endif
}

static long long now_ns(void)
{
    struct timespec t;
    clock_gettime(CLOCK_MONOTONIC, &t);
    return (long long)t.tv_sec * 1000000000ll + t.tv_nsec;
}

static void copy_streaming(char* d, const char* s, size_t n)
{
#if defined(__SSE2__)
    const size_t head = (64 - ((size_t)d & 63)) & 63;
    if (n >= 256) {
        memcpy(d, s, head);
        d += head; s += head; n -= head;
        for (; n >= 64; d += 64, s += 64, n -= 64) {
            const __m128i a = _mm_loadu_si128((const __m128i*)s), b = _mm_loadu_si128((const __m128i*)(s + 16));
            const __m128i c = _mm_loadu_si128((const __m128i*)(s + 32)), e = _mm_loadu_si128((const __m128i*)(s + 48));
            _mm_stream_si128((__m128i*)d, a);
            _mm_stream_si128((__m128i*)(d + 16), b);
            _mm_stream_si128((__m128i*)(d + 32), c);
            _mm_stream_si128((__m128i*)(d + 48), e);
        }
        _mm_sfence();                /* streaming stores are not ordered by the release that follows */
    }
#endif
    memcpy(d, s, n);
}

/* claims and copies one piece; 0 when there is none.  Called with the mutex held, returns with it held. */
static int copy_piece(ff_copy_pool* p)
{
    if (p->next >= p->bytes) return 0;
    const size_t o = p->next;
    const size_t n = p->bytes - o < FF_COPY_PIECE ? p->bytes - o : FF_COPY_PIECE;
    char* d = p->dst + o;
    const char* s = p->src + o;
    const int streaming = p->streaming;
    p->next = o + n;
    atomic_store_explicit(&p->open, p->bytes - p->next, memory_order_relaxed);
    pthread_mutex_unlock(&p->mu);
    if (streaming) copy_streaming(d, s, n);
    else memcpy(d, s, n);
    atomic_fetch_sub_explicit(&p->left, n, memory_order_release);
    pthread_mutex_lock(&p->mu);
    return 1;
}

static void* helper(void* arg)
{
    ff_copy_pool* p = (ff_copy_pool*)arg;
    pthread_mutex_lock(&p->mu);
    while (!p->stop) {
        if (copy_piece(p)) continue;
        pthread_mutex_unlock(&p->mu);
        const long long until = now_ns() + FF_COPY_SPIN_NS;
        while (atomic_load_explicit(&p->open, memory_order_relaxed) == 0 && now_ns() < until)
            for (int i = 0; i < 16; i++) relax();
        pthread_mutex_lock(&p->mu);
        while (!p->stop && p->next >= p->bytes) {
            p->sleeping++;
            pthread_cond_wait(&p->wake, &p->mu);
            p->sleeping--;
        }
    }
    pthread_mutex_unlock(&p->mu);
    return NULL;
}

ff_copy_pool* ff_copy_pool_create(int helpers)
{
    ff_copy_pool* p = (ff_copy_pool*)calloc(1, sizeof(ff_copy_pool));
    if (!p) return NULL;
    cpu_set_t set;
    int cpus = 1;
    if (sched_getaffinity(0, sizeof set, &set) == 0) cpus = CPU_COUNT(&set);
    if (helpers > FF_COPY_MAX_HELPERS) helpers = FF_COPY_MAX_HELPERS;
    if (helpers > cpus / 3) helpers = cpus / 3;
    p->wanted = helpers < 0 ? 0 : helpers;
    p->owner = getpid();
    if (pthread_mutex_init(&p->mu, NULL) != 0) { free(p); return NULL; }
    if (pthread_cond_init(&p->wake, NULL) != 0) { pthread_mutex_destroy(&p->mu); free(p); return NULL; }
    return p;
}

static void start_helpers(ff_copy_pool* p)
{
    /* the caller's signals stay the caller's */
    sigset_t all, old;
    sigfillset(&all);
    const int masked = pthread_sigmask(SIG_SETMASK, &all, &old) == 0;
    while (p->started < p->wanted) {
        if (pthread_create(&p->th[p->started], NULL, helper, p) != 0) { p->wanted = p->started; break; }
        p->started++;
    }
    if (masked) pthread_sigmask(SIG_SETMASK, &old, NULL);
}

void ff_copy_pool_destroy(ff_copy_pool* p)
{
    if (!p) return;
    if (p->owner != getpid()) return;            /* left as it is: the condition's sleepers would be waited for for good */
    pthread_mutex_lock(&p->mu);
    p->stop = 1;
    pthread_cond_broadcast(&p->wake);
    pthread_mutex_unlock(&p->mu);
    for (int i = 0; i < p->started; i++) pthread_join(p->th[i], NULL);
    pthread_cond_destroy(&p->wake);
    pthread_mutex_destroy(&p->mu);
    free(p);
}

void ff_copy(ff_copy_pool* p, void* dst, const void* src, size_t bytes, int streaming)
{
    if (!p || p->wanted == 0 || bytes < FF_COPY_MIN_SHARED || p->owner != getpid()) {
        if (streaming) copy_streaming((char*)dst, (const char*)src, bytes);
        else memcpy(dst, src, bytes);
        return;
    }
    if (p->started < p->wanted) start_helpers(p);
    pthread_mutex_lock(&p->mu);
    p->dst = (char*)dst; p->src = (const char*)src; p->bytes = bytes; p->next = 0; p->streaming = streaming;
    atomic_store_explicit(&p->left, bytes, memory_order_relaxed);
    atomic_store_explicit(&p->open, bytes, memory_order_relaxed);
    if (p->sleeping) pthread_cond_broadcast(&p->wake);
    while (copy_piece(p)) { }
    pthread_mutex_unlock(&p->mu);
    /* pieces the helpers hold: at most one each; give the CPU away if one of them has lost its own */
    for (int spin = 0; atomic_load_explicit(&p->left, memory_order_acquire) != 0; spin++) {
        if (spin < 2000) relax();
        else sched_yield();
    }
}
