/*
 * label_stream.c — labeling straight into a host sink, with the device-to-
 * host copy and the sink overlapped with the labeling of the next window.
 *
 * The reference's disk worker labels an HBM window, then copies it to a
 * pinned stage and writes it, strictly one after the other
 * (tools/disk-wipe-bench/disk_wipe_bench.cu:646-697).  Here the region is cut
 * into windows of whole super-chunks labelled alternately into two device
 * buffers; a worker thread copies each finished window into a pinned host
 * buffer on its own stream and hands it to the sink, while the calling thread
 * already labels the next ones.  A window of few chunk copies leaves most of
 * the GPU idle for the length of their chain, so consecutive windows are
 * labelled in one call until it has some eight copies per SM
 * (PB_STREAM_UNITS_PER_SM); the sink still gets them one by one, in order.  The sink
 * has the shape of the reference's pose_label_sink_fn
 * (common/include/graph.h:244-245) and, as there, may be called from a worker
 * thread.
 */
#include "pose_b200.h"
#include "dev_alloc.h"
#include "topo_internal.h"

#include <nvtx3/nvToolsExt.h>
#include <cuda_runtime_api.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <time.h>

/* Chunk copies per SM of one labelling call.  On 148 SMs, 2048 chunks of 4096
 * blocks in windows of 256 chunks, 512 copies: 19.9 ms a call; 1024 copies
 * 28.5, 1536 copies about 36, 4096 copies 78. */
#define PB_STREAM_UNITS_PER_SM 8u

typedef struct {
    pthread_mutex_t mu;
    pthread_cond_t cv;
    /* job handed to the worker (valid when posted): the windows in dev[buf],
     * len bytes, the first at byte offset off */
    int posted, quit;
    int buf;
    size_t len;
    uint64_t off;
    /* per buffer: 1 while the worker still uses it */
    int busy[2];
    int error;
    size_t window; /* bytes */
    double d2h_ms, sink_ms;
    /* resources */
    uint8_t *dev[2], *host;
    cudaStream_t stream;
    int device;
    pose_b200_sink_fn sink;
    void *ctx;
} stream_state_t;

static double now_ms(void)
{
    struct timespec ts;
    clock_gettime(CLOCK_MONOTONIC, &ts);
    return 1e3 * (double)ts.tv_sec + 1e-6 * (double)ts.tv_nsec;
}

/* Copy the windows of one labelling call to the pinned buffer and sink them,
 * one after the other. */
static int sink_windows(stream_state_t *s, int i, size_t len, uint64_t off)
{
    for (size_t at = 0; at < len; at += s->window) {
        const size_t n = len - at < s->window ? len - at : s->window;
        const double t0 = now_ms();
        if (cudaMemcpyAsync(s->host, s->dev[i] + at, n, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
            cudaStreamSynchronize(s->stream) != cudaSuccess) {
            fprintf(stderr, "pose_b200_label_stream: D2H copy failed: %s\n", cudaGetErrorString(cudaGetLastError()));
            return -1;
        }
        const double t1 = now_ms();
        if (s->sink(s->ctx, s->host, n, off + at) != 0) {
            fprintf(stderr, "pose_b200_label_stream: sink failed at offset %llu\n", (unsigned long long)(off + at));
            return -1;
        }
        s->d2h_ms += t1 - t0;
        s->sink_ms += now_ms() - t1;
    }
    return 0;
}

static void *sink_worker(void *arg)
{
    stream_state_t *s = (stream_state_t *)arg;
    cudaSetDevice(s->device);
    /* pinned here, while the first windows are labelled */
    const int have = cudaMallocHost((void **)&s->host, s->window) == cudaSuccess;
    if (!have) {
        cudaGetLastError();
        s->host = NULL;
        fprintf(stderr, "pose_b200_label_stream: pinned buffer of %llu bytes failed\n", (unsigned long long)s->window);
    }
    pthread_mutex_lock(&s->mu);
    if (!have) s->error = 1;
    for (;;) {
        while (!s->posted && !s->quit) pthread_cond_wait(&s->cv, &s->mu);
        if (!s->posted && s->quit) break;
        int i = s->buf;
        size_t len = s->len;
        uint64_t off = s->off;
        s->posted = 0;
        pthread_cond_broadcast(&s->cv);
        const int skip = s->error; /* nothing is sunk after a failure */
        pthread_mutex_unlock(&s->mu);
        const int err = skip ? -1 : sink_windows(s, i, len, off);
        pthread_mutex_lock(&s->mu);
        if (err) s->error = 1;
        s->busy[i] = 0;
        pthread_cond_broadcast(&s->cv);
    }
    pthread_mutex_unlock(&s->mu);
    return NULL;
}

static int pose_b200_label_stream_impl(const pose_hbm_topo_t *topo, const uint8_t *session_seed, size_t seed_len,
                           uint64_t region_bytes, uint64_t region_block_offset, uint64_t byte_offset,
                           size_t window_bytes, pose_b200_sink_fn sink, void *sink_ctx,
                           const pose_b200_sched_t *sched, pose_b200_stats_t *stats)
{
    if (stats) memset(stats, 0, sizeof(*stats));
    if (!topo || !sink) {
        fprintf(stderr, "pose_b200_label_stream: NULL topology or sink\n");
        return -1;
    }
    pb_topo_internal_t ti;
    if (pb_topo_internal(topo, &ti) != 0) return -1;
    const uint32_t cb = ti.cb;
    const uint64_t sb = ti.super_bytes;
    const uint64_t nsuper = region_bytes / sb;
    if (nsuper == 0) return 0;
    uint64_t W = window_bytes / sb;
    if (W == 0) W = 1;
    if (W > nsuper) W = nsuper;
    /* windows per labelling call: up to PB_STREAM_UNITS_PER_SM chunk copies
     * an SM, half the region (the first half is sunk while the second is
     * labelled) and a quarter of the free device memory; a caller's schedule
     * is for its own window */
    uint64_t per = 1;
    if (!sched) {
        const uint64_t units = (uint64_t)PB_STREAM_UNITS_PER_SM * (uint64_t)(ti.sms > 0 ? ti.sms : 1);
        const uint64_t copies = W * ti.copies, half = (nsuper + W - 1) / W / 2;
        size_t fr = 0, tot = 0;
        if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
            cudaGetLastError();
            fr = 0;
        }
        per = (units + copies - 1) / copies;
        if (per > half) per = half;
        while (per > 1 && 2 * per * W * sb > fr / 4) per--;
        if (per == 0) per = 1;
    }
    const uint64_t wbytes = W * sb;

    stream_state_t s;
    memset(&s, 0, sizeof(s));
    pthread_mutex_init(&s.mu, NULL);
    pthread_cond_init(&s.cv, NULL);
    s.sink = sink;
    s.ctx = sink_ctx;
    s.window = wbytes;
    cudaGetDevice(&s.device);
    int rc = -1, started = 0;
    pthread_t th;
    double t0 = now_ms(), kernel_ms = 0;
    uint64_t nodes = 0;
    uint32_t launches = 0;
    pose_b200_stats_t last;
    memset(&last, 0, sizeof(last));

    for (int i = 0; i < 2; i++) {
        const uint64_t cbytes = per * wbytes;
        if (pb_dev_malloc((void **)&s.dev[i], cbytes) != cudaSuccess) {
            cudaGetLastError();
            if (per > 1) { /* one window a call then */
                per = 1;
                if (i) cudaFree(s.dev[0]);
                s.dev[0] = NULL;
                i = -1;
                continue;
            }
            fprintf(stderr, "pose_b200_label_stream: window buffers of %llu bytes failed\n",
                    (unsigned long long)cbytes);
            goto out;
        }
    }
    if (cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking) != cudaSuccess) goto out;
    if (pthread_create(&th, NULL, sink_worker, &s) != 0) goto out;
    started = 1;

    for (uint64_t k = 0, first = 0; first < nsuper; k++, first += per * W) {
        const int i = (int)(k & 1);
        const uint64_t n = nsuper - first < per * W ? nsuper - first : per * W;
        pthread_mutex_lock(&s.mu);
        while (s.busy[i] && !s.error) pthread_cond_wait(&s.cv, &s.mu);
        int err = s.error;
        pthread_mutex_unlock(&s.mu);
        if (err) goto out;
        pose_b200_stats_t st;
        if (pose_b200_topo_label(topo, session_seed, seed_len, s.dev[i], n * sb,
                                 region_block_offset + first * (uint64_t)cb, sched, &st) != 0)
            goto out;
        kernel_ms += st.kernel_ms;
        nodes += st.nodes;
        launches += st.kernel_launches;
        last = st;
        pthread_mutex_lock(&s.mu);
        while (s.posted) pthread_cond_wait(&s.cv, &s.mu);
        s.busy[i] = 1;
        s.buf = i;
        s.len = n * sb;
        s.off = byte_offset + first * sb;
        s.posted = 1;
        pthread_cond_broadcast(&s.cv);
        pthread_mutex_unlock(&s.mu);
    }
    pthread_mutex_lock(&s.mu);
    while ((s.posted || s.busy[0] || s.busy[1]) && !s.error) pthread_cond_wait(&s.cv, &s.mu);
    rc = s.error ? -1 : 0;
    pthread_mutex_unlock(&s.mu);

out:
    if (started) {
        pthread_mutex_lock(&s.mu);
        while (s.posted || s.busy[0] || s.busy[1]) {
            if (s.error && !s.posted) break;
            pthread_cond_wait(&s.cv, &s.mu);
        }
        s.quit = 1;
        pthread_cond_broadcast(&s.cv);
        pthread_mutex_unlock(&s.mu);
        pthread_join(th, NULL);
    }
    if (stats) {
        *stats = last;
        stats->kernel_ms = kernel_ms;
        stats->total_ms = now_ms() - t0;
        stats->super_chunks = nsuper;
        stats->units = nsuper * (last.units && last.super_chunks ? last.units / last.super_chunks : 2);
        stats->nodes = nodes;
        stats->kernel_launches = launches;
    }
    for (int i = 0; i < 2; i++) cudaFree(s.dev[i]);
    if (s.host) cudaFreeHost(s.host);
    if (s.stream) cudaStreamDestroy(s.stream);
    pthread_mutex_destroy(&s.mu);
    pthread_cond_destroy(&s.cv);
    return rc;
}

int pose_b200_label_stream(const pose_hbm_topo_t *topo, const uint8_t *session_seed, size_t seed_len,
                           uint64_t region_bytes, uint64_t region_block_offset, uint64_t byte_offset,
                           size_t window_bytes, pose_b200_sink_fn sink, void *sink_ctx,
                           const pose_b200_sched_t *sched, pose_b200_stats_t *stats)
{
    nvtxRangePushA("pose_b200: streamed labeling");
    int rc = pose_b200_label_stream_impl(topo, session_seed, seed_len, region_bytes, region_block_offset, byte_offset, window_bytes, sink, sink_ctx, sched, stats);
    nvtxRangePop();
    return rc;
}
