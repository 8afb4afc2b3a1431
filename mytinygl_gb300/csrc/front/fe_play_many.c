/*
 * fe_play_many.c — mtgl_play_many: the command streams of many contexts played at once.
 *
 * No counterpart in the reference, where one thread drives one current context
 * (gl_api.c:14-23). Contexts share no front-end state and, outside an unfinished batch (one
 * writing their framebuffer or reading their resources), no back-end state either, so
 * distinct contexts play on a pool of threads, kept between calls: each thread claims the next
 * unplayed stream (longest first), makes its context current and plays it. Staging copies,
 * index scans and state snapshots of different frames then run on all host cores instead of one.
 */
#include <errno.h>
#include <pthread.h>
#include <time.h>
#include <unistd.h>

#include "fe_internal.h"

typedef struct play_job {
    GLState *const *ctxs;
    const void *const *streams;
    const size_t *bytes;
    int32_t n;
    int *status;
    const int32_t *order; /* claim order (null: stream order) */
    int32_t next;         /* next unclaimed position of the order */
    int32_t helpers;      /* helpers it may still take, and those playing it now (under g_mu) */
    int32_t active;
    struct play_job *link;
} play_job;

static void play_streams(play_job *j)
{
    for (;;) {
        int32_t k = __atomic_fetch_add(&j->next, 1, __ATOMIC_RELAXED);
        if (k >= j->n) break;
        const int32_t i = j->order ? j->order[k] : k;
        j->status[i] = mtgl_play(j->ctxs[i], j->streams[i], j->bytes[i]);
    }
}

/* Helper threads, kept between calls: starting 15 threads took 50 us each on the calling thread,
 * more than playing 256 frames of resident geometry takes alone (453 us; 952 us with 16 fresh
 * threads). A helper takes the first listed job that wants one, and ends after two idle
 * seconds, at library unload, or (by not existing there) in a forked child. Jobs of several
 * calling threads share the helpers; every caller also plays its own job. Every helper is
 * joined, by the next that ends or at unload, so that none is in this code when it goes. */
#define PLAY_MAX_THREADS 64
#define PLAY_IDLE_SECONDS 2

static pthread_mutex_t g_mu = PTHREAD_MUTEX_INITIALIZER;
static pthread_cond_t g_work = PTHREAD_COND_INITIALIZER; /* a job was listed, or the library unloads */
static pthread_cond_t g_idle = PTHREAD_COND_INITIALIZER; /* a helper left its job, or was started */
static play_job *g_jobs;
/* A helper's place. FREE -> TAKEN (being started) -> its thread id known; it ends on its own;
 * with both, it may be joined. */
enum { SLOT_FREE = 0, SLOT_TAKEN = 1, SLOT_STARTED = 2, SLOT_ENDED = 4 };
static struct play_slot {
    pthread_t tid;
    int state;
} g_slot[PLAY_MAX_THREADS];
static int32_t g_helpers, g_waiting; /* helpers not ended; of those, waiting for work */
static int g_unload;

static play_job *wanting_job(void)
{
    for (play_job *j = g_jobs; j; j = j->link)
        if (j->helpers > 0 && __atomic_load_n(&j->next, __ATOMIC_RELAXED) < j->n) return j;
    return NULL;
}

/* Joins the helpers that have ended (g_mu held; given up meanwhile). They hold no lock any more. */
static void join_ended(void)
{
    pthread_t tid[PLAY_MAX_THREADS];
    int n = 0;
    for (int i = 0; i < PLAY_MAX_THREADS; i++)
        if (g_slot[i].state == (SLOT_TAKEN | SLOT_STARTED | SLOT_ENDED)) {
            tid[n++] = g_slot[i].tid;
            g_slot[i].state = SLOT_FREE;
        }
    if (!n) return;
    pthread_mutex_unlock(&g_mu);
    for (int i = 0; i < n; i++) pthread_join(tid[i], NULL);
    pthread_mutex_lock(&g_mu);
}

static void *play_helper(void *arg)
{
    struct play_slot *slot = (struct play_slot *)arg;
    pthread_mutex_lock(&g_mu);
    while (!g_unload) {
        play_job *j = wanting_job();
        if (!j) {
            struct timespec until;
            clock_gettime(CLOCK_REALTIME, &until);
            until.tv_sec += PLAY_IDLE_SECONDS;
            g_waiting++;
            const int r = pthread_cond_timedwait(&g_work, &g_mu, &until);
            g_waiting--;
            if (r == ETIMEDOUT && !wanting_job()) break;
            continue;
        }
        j->helpers--;
        j->active++;
        pthread_mutex_unlock(&g_mu);
        play_streams(j);
        gl_make_current(NULL);
        pthread_mutex_lock(&g_mu);
        j->active--;
        pthread_cond_broadcast(&g_idle);
    }
    if (!g_unload) join_ended();
    slot->state |= SLOT_ENDED;
    g_helpers--;
    pthread_mutex_unlock(&g_mu);
    return NULL;
}

static void fork_child(void)
{
    pthread_mutex_init(&g_mu, NULL);
    pthread_cond_init(&g_work, NULL);
    pthread_cond_init(&g_idle, NULL);
    g_jobs = NULL;
    for (int i = 0; i < PLAY_MAX_THREADS; i++) g_slot[i].state = SLOT_FREE;
    g_helpers = g_waiting = 0;
}
static void fork_prepare(void) { pthread_mutex_lock(&g_mu); }
static void fork_parent(void) { pthread_mutex_unlock(&g_mu); }
static pthread_once_t g_once = PTHREAD_ONCE_INIT;
static void play_init(void) { pthread_atfork(fork_prepare, fork_parent, fork_child); }

__attribute__((destructor)) static void play_unload(void)
{
    pthread_mutex_lock(&g_mu);
    g_unload = 1;
    pthread_cond_broadcast(&g_work);
    for (int i = 0; i < PLAY_MAX_THREADS; i++) {
        while (g_slot[i].state != SLOT_FREE && !(g_slot[i].state & SLOT_STARTED)) pthread_cond_wait(&g_idle, &g_mu);
        if (g_slot[i].state == SLOT_FREE || pthread_equal(g_slot[i].tid, pthread_self())) continue;
        const pthread_t tid = g_slot[i].tid;
        g_slot[i].state = SLOT_FREE;
        pthread_mutex_unlock(&g_mu);
        pthread_join(tid, NULL);
        pthread_mutex_lock(&g_mu);
    }
    pthread_mutex_unlock(&g_mu);
}

/* Starts a helper unless there are `want` (g_mu held; given up meanwhile, so that those already
 * started get on with the job). Returns 0 when none is to be had. */
static int start_helper(int32_t want)
{
    struct play_slot *slot = NULL;
    if (g_unload || g_helpers >= want || g_helpers >= PLAY_MAX_THREADS) return 0;
    for (int i = 0; i < PLAY_MAX_THREADS && !slot; i++)
        if (g_slot[i].state == SLOT_FREE) slot = &g_slot[i];
    if (!slot) return 0;
    slot->state = SLOT_TAKEN;
    g_helpers++;
    pthread_mutex_unlock(&g_mu);
    pthread_t tid;
    const int failed = pthread_create(&tid, NULL, play_helper, slot);
    pthread_mutex_lock(&g_mu);
    if (failed) {
        slot->state = SLOT_FREE;
        g_helpers--;
    } else {
        slot->tid = tid;
        slot->state |= SLOT_STARTED;
    }
    pthread_cond_broadcast(&g_idle);
    return !failed;
}

/* Plays the job with up to `helpers` other threads; returns when every stream is played. */
static void play_shared(play_job *j, int32_t helpers)
{
    pthread_once(&g_once, play_init);
    pthread_mutex_lock(&g_mu);
    j->helpers = helpers;
    j->active = 0;
    j->link = g_jobs;
    g_jobs = j;
    const int32_t woken = g_waiting < helpers ? g_waiting : helpers;
    for (int32_t k = 0; k < woken; k++) pthread_cond_signal(&g_work);
    while (__atomic_load_n(&j->next, __ATOMIC_RELAXED) < j->n && start_helper(helpers)) {
    }
    pthread_mutex_unlock(&g_mu);
    play_streams(j); /* this thread plays too; with no helper it plays every stream in order */
    pthread_mutex_lock(&g_mu);
    j->helpers = 0;
    while (j->active > 0) pthread_cond_wait(&g_idle, &g_mu);
    for (play_job **p = &g_jobs; *p; p = &(*p)->link)
        if (*p == j) {
            *p = j->link;
            break;
        }
    pthread_mutex_unlock(&g_mu);
}

/* longest streams first (a stream's bytes stand for its work), so that the last streams
 * claimed are short and the threads finish together */
static const size_t *g_sort_bytes;
static int cmp_longer(const void *a, const void *b)
{
    const size_t x = g_sort_bytes[*(const int32_t *)a], y = g_sort_bytes[*(const int32_t *)b];
    if (x != y) return x > y ? -1 : 1;
    return *(const int32_t *)a - *(const int32_t *)b;
}

static int cmp_ptr(const void *a, const void *b)
{
    uintptr_t x = (uintptr_t) * (GLState *const *)a, y = (uintptr_t) * (GLState *const *)b;
    return x < y ? -1 : (x > y);
}

/* threads to use: MTGL_PLAY_THREADS, else the online cores; at most one per stream */
static int32_t play_threads(int32_t n)
{
    const char *e = getenv("MTGL_PLAY_THREADS");
    long t = (e && *e) ? strtol(e, NULL, 10) : sysconf(_SC_NPROCESSORS_ONLN);
    if (t < 1) t = 1;
    if (t > PLAY_MAX_THREADS) t = PLAY_MAX_THREADS;
    return t > n ? n : (int32_t)t;
}

/* 1 when every context is non-null, distinct and in no unfinished batch. (A context in one
 * plays on the calling thread, where its first device operation waits for the batch, as a
 * single mtgl_play would.) */
static int can_share(GLState *const *ctxs, int32_t n)
{
    GLState **sorted = (GLState **)malloc((size_t)n * sizeof(GLState *));
    int ok = sorted != NULL;
    for (int32_t i = 0; ok && i < n; i++) {
        ok = ctxs[i] != NULL && !mtgl_dev_in_batch(ctxs[i]->dev);
        if (ok) sorted[i] = ctxs[i];
    }
    if (ok) {
        qsort(sorted, (size_t)n, sizeof(GLState *), cmp_ptr);
        for (int32_t i = 1; ok && i < n; i++) ok = sorted[i] != sorted[i - 1];
    }
    free(sorted);
    return ok;
}

int mtgl_play_many(GLState *const *ctxs, const void *const *streams, const size_t *bytes, int32_t n)
{
    if (n < 0 || (n > 0 && (!ctxs || !streams || !bytes))) return MTGL_ERR_INVALID;
    if (n == 0) return MTGL_OK;
    GLState *prev = gl_get_current_context();
    int *status = (int *)calloc((size_t)n, sizeof(int));
    if (!status) return MTGL_ERR_OOM;
    int32_t threads = play_threads(n);
    if (threads > 1 && !can_share(ctxs, n)) threads = 1;
    int32_t *order = NULL;
    if (threads > 1 && (order = (int32_t *)malloc((size_t)n * sizeof(int32_t))) != NULL) {
        for (int32_t i = 0; i < n; i++) order[i] = i;
        static pthread_mutex_t sort_lock = PTHREAD_MUTEX_INITIALIZER;  /* qsort has no context argument */
        pthread_mutex_lock(&sort_lock);
        g_sort_bytes = bytes;
        qsort(order, (size_t)n, sizeof(int32_t), cmp_longer);
        pthread_mutex_unlock(&sort_lock);
    }
    play_job job = {ctxs, streams, bytes, n, status, order, 0, 0, 0, NULL};
    if (threads > 1) play_shared(&job, threads - 1);
    else play_streams(&job);
    gl_make_current(prev);
    free(order);
    int st = MTGL_OK;
    for (int32_t i = 0; i < n && st == MTGL_OK; i++) st = status[i];
    free(status);
    return st;
}
