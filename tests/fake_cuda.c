/*
 * fake_cuda.c — a CUDA runtime and kernel launchers that do nothing, for the
 * CPU tests of the host side's plans: what is allocated, what is launched and
 * with which sizes (test_host_plans.py).  "Device" memory is host memory.
 */
#include "kernels.h"
#include "topology.h"

#include <cuda_runtime_api.h>
#include <pthread.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define SMS 148
#define MAX_SMEM (227 * 1024)

/* what the tests read and set */
typedef struct {
    uint32_t kind; /* 1 k_label, 2 k_label_multi, 3 k_label_ws, 4 k_label_wsc */
    uint32_t grid, warps, units_per, nunits, nbatches, smem;
    uint64_t scratch; /* bytes that its CTAs use of the launch's scratch */
} fake_launch_t;

static pthread_mutex_t mu = PTHREAD_MUTEX_INITIALIZER;
static fake_launch_t launches[4096];
static int nlaunches;
static uint64_t free_bytes = (uint64_t)170 << 30, live_bytes;
static uint64_t event_seq, events_done = UINT64_MAX; /* events up to this one are complete */
static int fail_multi_occupancy, occupancy_queries, node_priorities, priority_streams;

int fake_launches(fake_launch_t *out, int max)
{
    pthread_mutex_lock(&mu);
    const int n = nlaunches < max ? nlaunches : max;
    memcpy(out, launches, (size_t)n * sizeof(*out));
    pthread_mutex_unlock(&mu);
    return n;
}
void fake_reset(void)
{
    pthread_mutex_lock(&mu);
    nlaunches = 0;
    occupancy_queries = priority_streams = 0;
    pthread_mutex_unlock(&mu);
}
void fake_set_free(uint64_t bytes) { free_bytes = bytes; }
uint64_t fake_live(void) { return live_bytes; }
void fake_hold_events(void) { pthread_mutex_lock(&mu); events_done = event_seq; pthread_mutex_unlock(&mu); }
void fake_finish_events(void) { pthread_mutex_lock(&mu); events_done = UINT64_MAX; pthread_mutex_unlock(&mu); }
void fake_fail_multi_occupancy(int on) { fail_multi_occupancy = on; }
int fake_occupancy_queries(void) { return occupancy_queries; }
int fake_priority_streams(void) { return priority_streams; }
int fake_node_priorities(void) { return node_priorities; } /* of the last graph */

static int record(uint32_t kind, uint32_t grid, uint32_t warps, uint32_t per, uint32_t nunits, uint32_t nbatches,
                  uint32_t smem, uint64_t scratch)
{
    pthread_mutex_lock(&mu);
    if (nlaunches < (int)(sizeof(launches) / sizeof(launches[0])))
        launches[nlaunches++] = (fake_launch_t){kind, grid, warps, per, nunits, nbatches, smem, scratch};
    pthread_mutex_unlock(&mu);
    return 0;
}

/* ── runtime ─────────────────────────────────────────────────────────────── */

typedef struct { size_t bytes; uint64_t pad; } head_t;
static head_t *take(size_t bytes)
{
    head_t *h = (head_t *)calloc(1, sizeof(head_t) + bytes);
    if (h) h->bytes = bytes;
    return h;
}
cudaError_t cudaMalloc(void **p, size_t bytes)
{
    pthread_mutex_lock(&mu);
    const int full = live_bytes + bytes > free_bytes;
    if (!full) live_bytes += bytes;
    pthread_mutex_unlock(&mu);
    head_t *h = full ? NULL : take(bytes);
    *p = h ? h + 1 : NULL;
    return h ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p)
{
    if (p) {
        pthread_mutex_lock(&mu);
        live_bytes -= ((head_t *)p)[-1].bytes;
        pthread_mutex_unlock(&mu);
        free((head_t *)p - 1);
    }
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) { *p = calloc(1, bytes ? bytes : 1); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned f) { (void)f; return cudaMallocHost(p, bytes); }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned f) { (void)f; *d = h; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *fr, size_t *tot)
{
    *tot = (size_t)180 << 30;
    *fr = free_bytes > live_bytes ? (size_t)(free_bytes - live_bytes) : 0;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind k) { (void)k; memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    (void)st;
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void *d, int v, size_t n) { (void)d; (void)v; (void)n; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) { (void)d; (void)v; (void)n; (void)st; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { (void)d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr a, int d)
{
    (void)d;
    *v = a == cudaDevAttrMultiProcessorCount ? SMS : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { *lo = 0; *hi = -5; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { (void)e; return "fake"; }
cudaError_t cudaStreamCreate(cudaStream_t *s) { *s = (cudaStream_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned f) { (void)f; return cudaStreamCreate(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int p)
{
    (void)f; (void)p;
    priority_streams++;
    return cudaStreamCreate(s);
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { (void)s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) { (void)s; (void)e; (void)f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode m) { (void)s; (void)m; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) { (void)s; *g = (cudaGraph_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long f)
{
    (void)g;
    node_priorities = (f & cudaGraphInstantiateFlagUseNodePriority) != 0;
    *x = (cudaGraphExec_t)calloc(1, 8);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) { (void)x; (void)s; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)calloc(1, 8); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned f) { (void)f; return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    (void)s;
    pthread_mutex_lock(&mu);
    *(uint64_t *)e = ++event_seq;
    pthread_mutex_unlock(&mu);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e)
{
    pthread_mutex_lock(&mu);
    const int done = *(uint64_t *)e <= events_done;
    pthread_mutex_unlock(&mu);
    return done ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { (void)e; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) { (void)a; (void)b; *ms = 1.0f; return cudaSuccess; }

/* ── kernels ─────────────────────────────────────────────────────────────── */

uint32_t pb_ws_smem_bytes(uint32_t G, uint32_t warps)
{
    const uint32_t nthr = 32u * warps, slots = nthr / G;
    return (5u + 34u * G + 2u * G * (PB_CSM + 1u) + 6u * slots + 12u * nthr) * 16u;
}
int pb_dev_label_ws_prepare(uint32_t *max) { if (max) *max = MAX_SMEM - 16; return 0; }
int pb_dev_label_ws_occupancy(uint32_t cta, uint32_t smem, int *n)
{
    occupancy_queries++;
    *n = cta > 512 || smem > MAX_SMEM ? 0 : 1;
    return 0;
}
int pb_dev_label_wsc_max_clusters(uint32_t C, uint32_t warps, uint32_t smem, int *n)
{
    (void)warps; (void)smem;
    occupancy_queries++;
    *n = SMS / (int)C - (C > 4 ? 2 : 0);
    return 0;
}
int pb_dev_label_ws(const pb_depth_params_t *p, uint32_t grid, uint32_t smem, cudaStream_t s)
{
    (void)s;
    return record(3, grid, p->team_warps, p->units_per_cta, p->nunits, p->nbatches, smem,
                  (uint64_t)grid * p->units_per_cta * p->unit_scratch_bytes);
}
int pb_dev_label_wsc(const pb_depth_params_t *p, uint32_t smem, cudaStream_t s)
{
    (void)s;
    return record(4, p->nunits * p->cluster, p->team_warps, 1, p->nunits, p->nunits, smem,
                  p->nunits * p->unit_scratch_bytes);
}
int pb_dev_label(const pb_label_params_t *p, uint32_t grid, uint32_t cta, uint32_t smem, cudaStream_t s)
{
    (void)cta; (void)s;
    return record(1, grid, p->team_warps, p->units_per_team, p->nunits, p->nbatches, smem, grid * p->team_scratch_bytes);
}
int pb_dev_label_occupancy(uint32_t cta, int *n)
{
    *n = (int)(1024u / cta) > 32 ? 32 : (int)(1024u / cta);
    return 0;
}
int pb_dev_label_balance_smem(uint32_t cta, uint32_t per, uint32_t *smem) { (void)cta; (void)per; *smem = 0; return 0; }
int pb_dev_label_multi(const pb_multi_params_t *p, uint32_t grid, uint32_t cta, uint32_t smem, cudaStream_t s)
{
    (void)s;
    return record(2, grid, cta / 32, 0, 0, p->nbatches, smem, grid * p->team_scratch_bytes);
}
int pb_dev_label_multi_occupancy(uint32_t cta, int *n, uint32_t *alone)
{
    if (fail_multi_occupancy) return -1;
    *n = (int)(1024u / cta);
    if (alone) *alone = MAX_SMEM - 128;
    return 0;
}
int pb_dev_seed_jobs(const void *jobs, uint32_t n, const uint8_t *blob, uint32_t *seeds, cudaStream_t s)
{
    (void)jobs; (void)n; (void)blob; (void)seeds; (void)s;
    return 0;
}
int pb_dev_chunk_seeds(const uint8_t *d, uint32_t len, uint64_t rbo, uint32_t cb, uint32_t n, uint64_t first,
                       uint32_t *seeds, unsigned int *queue, cudaStream_t s)
{
    (void)d; (void)len; (void)rbo; (void)cb; (void)n; (void)first; (void)seeds; (void)queue; (void)s;
    return 0;
}
int pb_dev_set_keys(const uint32_t a[8], const uint32_t b[8], const uint32_t c[8]) { (void)a; (void)b; (void)c; return 0; }
int pb_dev_cv0_table(const void *r, uint32_t S, uint32_t c, void *cv0, cudaStream_t s)
{
    (void)r; (void)S; (void)c; (void)cv0; (void)s;
    return 0;
}
int pb_dev_compare_blocks(const void *a, const void *b, uint64_t n, uint64_t per, unsigned long long *bad, uint32_t grid,
                          cudaStream_t s)
{
    (void)a; (void)b; (void)n; (void)per; (void)bad; (void)grid; (void)s;
    return 0;
}
int pb_dev_gather_labels(const void *w, const uint64_t *src, uint32_t n, void *out, cudaStream_t s)
{
    (void)w; (void)src; (void)n; (void)out; (void)s;
    return 0;
}
int pb_dev_count_nonzero(const void *b, uint64_t n, unsigned long long *c, uint32_t grid, cudaStream_t s)
{
    (void)b; (void)n; (void)c; (void)grid; (void)s;
    return 0;
}
int pb_noalloc_residue(int dev, unsigned long long *c, uint32_t grid, cudaStream_t s)
{
    (void)dev; (void)c; (void)grid; (void)s;
    return 0;
}
int pb_dev_label_single(uint32_t *o, int src, uint64_t i, const uint32_t *in, int a, int b, cudaStream_t s)
{
    (void)o; (void)src; (void)i; (void)in; (void)a; (void)b; (void)s;
    return -1;
}
int pb_dev_compress_bench(uint32_t g, uint32_t i, uint32_t salt, uint32_t *sink, cudaStream_t s)
{
    (void)g; (void)i; (void)salt; (void)sink; (void)s;
    return 0;
}
int pb_dev_compress_latency(uint32_t i, unsigned long long *c, uint32_t *sink, cudaStream_t s)
{
    (void)i; (void)c; (void)sink; (void)s;
    return 0;
}
int pose_b200_topo_label_noalloc(const void *t, const uint8_t *k, size_t n, void *p, size_t len, uint64_t rbo)
{
    (void)t; (void)k; (void)n; (void)p; (void)len; (void)rbo;
    return -1;
}
