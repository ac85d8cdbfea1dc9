/*
 * label_batch.c — batched labeling (C11 host side of k_label_multi).
 *
 * Many requests — each one session seed, one topology (chunk_blocks), one
 * device buffer and one region_block_offset, with the semantics of a
 * pose_graph_hbm_topo_label call — run in one persistent launch:
 *
 *   - every super-chunk of every request contributes its two chunk copies
 *     (units); its chunk seed is derived on the device from a seed job
 *     (session seed in a packed blob, chunk index (rbo + j*cb)/cb);
 *   - units of one topology are grouped G at a time into batches that a team
 *     of T warps runs in lockstep.  A warp with no node in a level skips it,
 *     so the ALU work of a batch is sum over levels of ceil(G*w/32) warp
 *     passes whatever T is, while its chain is sum of ceil(G*w/(32T)): wide
 *     teams shorten the deep topologies' chains for free, and a shallow
 *     topology packs G units while its chain stays under the deepest one's;
 *   - T and the packing rule are chosen by an estimate of the makespan (the
 *     longest chain against the ALU time of all warp passes);
 *   - batches are queued longest first (by passes), so the deep topologies
 *     start at once and the short ones fill in behind them;
 *   - seed derivation, queue reset, the labeling kernel and the scratch
 *     zeroing are captured once into a CUDA graph and replayed.
 */
#include "batch_internal.h"
#include "dev_alloc.h"
#include "kernels.h"
#include "topo_internal.h"
#include "pose_b200.h"

#include <nvtx3/nvToolsExt.h>
#include <cuda_runtime_api.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

/* One launch of a batch: its tables, scratch and queue.  kind 0 runs the
 * lockstep multi-topology kernel, kind 1 the multi-unit depth kernel (one
 * topology; v2, units_per_cta and smem describe it). */
typedef struct {
    void *d_topos, *d_batches, *d_units, *d_jobs, *d_seeds, *d_scratch, *d_queue;
    uint64_t scratch_bytes, nodes, super_chunks, units, nbatches, njobs;
    uint32_t teams, T, Gmax, cv0, grid, cta_threads;
    uint64_t team_scratch;
    int kind;
    pb_topo_view2_t v2;
    uint32_t units_per_cta, smem;
} batch_part_t;

struct pose_b200_batch {
    int device;
    cudaStream_t stream, stream2, stream3;
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    cudaEvent_t ev[8]; /* 0/3: replay start/end; 1/2: first launch's kernel; 4/5, 6/7: fork/join */
    void *d_blob; /* the requests' session seeds, back to back */
    size_t blob_len;
    int nparts;
    batch_part_t part[3]; /* part[1]: the deep requests, when split; part[2]: the next-deepest topology's */
    uint64_t scratch_bytes, nodes, super_chunks, units;
    uint32_t nbatches, teams, T, Gmax, cv0;
};

typedef struct {
    uint64_t cost;
    pb_mbatch_t b;
} batch_sort_t;

static int cmp_batch(const void *a, const void *b)
{
    uint64_t x = ((const batch_sort_t *)a)->cost, y = ((const batch_sort_t *)b)->cost;
    return x < y ? 1 : x > y ? -1 : 0;
}

static void batch_free(pose_b200_batch_t *b)
{
    if (!b) return;
    if (b->stream) {
        for (int i = 0; i < b->nparts; i++) {
            batch_part_t *q = &b->part[i];
            if (q->d_scratch) cudaMemsetAsync(q->d_scratch, 0, q->scratch_bytes, b->stream);
            if (q->d_seeds) cudaMemsetAsync(q->d_seeds, 0, (size_t)q->njobs * 32, b->stream);
        }
        /* the session seeds go with the batch */
        if (b->d_blob) cudaMemsetAsync(b->d_blob, 0, b->blob_len ? b->blob_len : 1, b->stream);
        cudaStreamSynchronize(b->stream);
    }
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    for (int i = 0; i < 3; i++) {
        batch_part_t *q = &b->part[i];
        cudaFree(q->d_topos); cudaFree(q->d_batches); cudaFree(q->d_units); cudaFree(q->d_jobs);
        cudaFree(q->d_seeds); cudaFree(q->d_scratch); cudaFree(q->d_queue);
    }
    cudaFree(b->d_blob);
    for (int i = 0; i < 8; i++) if (b->ev[i]) cudaEventDestroy(b->ev[i]);
    if (b->stream3) cudaStreamDestroy(b->stream3);
    if (b->stream2) cudaStreamDestroy(b->stream2);
    if (b->stream) cudaStreamDestroy(b->stream);
    free(b);
}

void pose_b200_batch_destroy(pose_b200_batch_t *b) { batch_free(b); }

#define BK(call, what)                                                                    \
    do {                                                                                  \
        if ((call) != cudaSuccess) {                                                      \
            fprintf(stderr, "pose_b200_batch_create: %s: %s\n", what,                     \
                    cudaGetErrorString(cudaGetLastError()));                              \
            goto fail;                                                                    \
        }                                                                                 \
    } while (0)

void pb_plan_free(pb_plan_tables_t *p)
{
    if (!p) return;
    free(p->views);
    free(p->units);
    free(p->unit_req);
    free(p->jobs);
    free(p->batches);
    memset(p, 0, sizeof(*p));
}

int pb_plan_requests(const pb_req_t *reqs, size_t n, uint32_t T, uint32_t gcap, double eff_min, double target,
                     pb_plan_tables_t *out)
{
    memset(out, 0, sizeof(*out));
    const pose_hbm_topo_t **topo_list = (const pose_hbm_topo_t **)calloc(n ? n : 1, sizeof(*topo_list));
    pb_topo_internal_t *ti = (pb_topo_internal_t *)calloc(n ? n : 1, sizeof(*ti));
    uint32_t *G = NULL, *nunits_t = NULL, *ucount = NULL;
    uint64_t *ufirst = NULL;
    batch_sort_t *bs = NULL;
    size_t ntopo = 0;
    uint64_t njobs = 0, total_units = 0;
    int dev = -1, rc = -1;
    if (!topo_list || !ti) goto done;
    cudaGetDevice(&dev);
    for (size_t i = 0; i < n; i++) {
        const pb_req_t *r = &reqs[i];
        pb_topo_internal_t x;
        if (pb_topo_internal(r->topo, &x) != 0) { fprintf(stderr, "pose_b200: request %zu has no topology\n", i); goto done; }
        if (x.device != dev) { fprintf(stderr, "pose_b200: request %zu: topology of another device\n", i); goto done; }
        uint64_t ns = r->len / x.super_bytes;
        if (ns && !r->dev_ptr) { fprintf(stderr, "pose_b200: request %zu: NULL buffer\n", i); goto done; }
        size_t k = 0;
        while (k < ntopo && topo_list[k] != r->topo) k++;
        if (k == ntopo) { topo_list[ntopo] = r->topo; ti[ntopo] = x; ntopo++; }
        njobs += ns;
        total_units += ns * x.copies;
    }
    if (total_units > 0xFFFFFFFFull) { fprintf(stderr, "pose_b200: too many chunk copies\n"); goto done; }
    out->ntopo = ntopo;
    out->nunits = total_units;
    out->njobs = njobs;
    out->sms = ntopo ? (uint32_t)ti[0].sms : 0;
    out->all_cv0 = 1;
    G = (uint32_t *)calloc(ntopo + 1, 4);
    nunits_t = (uint32_t *)calloc(ntopo + 1, 4);
    ufirst = (uint64_t *)calloc(ntopo + 1, 8);
    ucount = (uint32_t *)calloc(ntopo + 1, 4);
    out->views = (pb_topo_view_t *)calloc(ntopo + 1, sizeof(pb_topo_view_t));
    out->units = (pb_munit_t *)calloc(total_units + 1, sizeof(pb_munit_t));
    out->unit_req = (uint32_t *)calloc(total_units + 1, sizeof(uint32_t));
    out->jobs = (pb_seedjob_t *)calloc(njobs + 1, sizeof(pb_seedjob_t));
    if (!G || !nunits_t || !ufirst || !ucount || !out->views || !out->units || !out->unit_req || !out->jobs) goto done;
    for (size_t i = 0; i < n; i++) {
        size_t k = 0;
        while (topo_list[k] != reqs[i].topo) k++;
        nunits_t[k] += (uint32_t)((reqs[i].len / ti[k].super_bytes) * ti[k].copies);
    }
    {
        uint64_t acc = 0;
        for (size_t k = 0; k < ntopo; k++) {
            ufirst[k] = acc;
            acc += nunits_t[k];
            out->views[k] = ti[k].view;
            if (!ti[k].view.cv0) out->all_cv0 = 0;
        }
    }
    {
        uint64_t job = 0;
        for (size_t i = 0; i < n; i++) {
            const pb_req_t *r = &reqs[i];
            size_t k = 0;
            while (topo_list[k] != r->topo) k++;
            uint64_t ns = r->len / ti[k].super_bytes;
            for (uint64_t j = 0; j < ns; j++, job++) {
                out->jobs[job].chunk_index = (r->rbo + j * (uint64_t)ti[k].cb) / ti[k].cb;
                out->jobs[job].seed_off = r->seed_off;
                out->jobs[job].seed_len = r->seed_len;
                for (uint32_t c = 0; c < ti[k].copies; c++) {
                    out->unit_req[ufirst[k] + ucount[k]] = (uint32_t)i;
                    pb_munit_t *u = &out->units[ufirst[k] + ucount[k]++];
                    u->out = (uint64_t)(uintptr_t)r->dev_ptr + j * ti[k].super_bytes;
                    u->seed = (uint32_t)job;
                    u->copy = c;
                }
            }
        }
    }
    /* G per topology.  eff_min > 0: the smallest power of two whose lane
     * efficiency G*S / (passes * 32T) reaches eff_min.  eff_min <= 0: pack
     * units as long as the batch's chain of passes stays within the longest
     * chain of the launch at G = 1 (the deepest topology sets the makespan;
     * packing shallower ones costs no time and fills partial warps).
     * target > 0 replaces both rules: as many units as a batch finishes in
     * that many clocks, spread evenly.  target < 0 keeps the rule, within
     * -target clocks a batch. */
    uint64_t chain_cap = 0;
    for (size_t k = 0; k < ntopo; k++) {
        uint64_t p1 = pb_topo_passes(topo_list[k], T, 1);
        if (p1 > chain_cap) chain_cap = p1;
    }
    uint64_t nb = 0;
    for (size_t k = 0; k < ntopo; k++) {
        uint32_t g = 1;
        if (target > 0 && nunits_t[k]) {
            const uint32_t most = gcap < nunits_t[k] ? gcap : nunits_t[k];
            while (g < most && g < 32 * T && pb_topo_lockstep_clocks(topo_list[k], T, g + 1) <= target) g++;
            const uint32_t even = (nunits_t[k] + g - 1) / g;
            g = (nunits_t[k] + even - 1) / even;
        }
        while (target <= 0 && g * 2 <= gcap && g * 2 <= 32 * T && g < nunits_t[k]) {
            if (eff_min > 0) {
                uint64_t passes = pb_topo_passes(topo_list[k], T, g);
                double eff = (double)g * ti[k].view.S / ((double)passes * 32.0 * T);
                if (eff >= eff_min) break;
            } else if (pb_topo_passes(topo_list[k], T, g * 2) > chain_cap) {
                break;
            }
            if (target < 0 && pb_topo_lockstep_clocks(topo_list[k], T, g * 2) > -target) break;
            g *= 2;
        }
        G[k] = g;
        if (g > out->Gmax) out->Gmax = g;
        nb += (nunits_t[k] + g - 1) / g;
        uint64_t ts = (uint64_t)g * ti[k].view.pool * 32;
        if (ts > out->team_scratch) out->team_scratch = ts;
        out->nodes += (uint64_t)nunits_t[k] * ti[k].view.S;
    }
    bs = (batch_sort_t *)calloc(nb + 1, sizeof(*bs));
    out->batches = (pb_mbatch_t *)calloc(nb + 1, sizeof(pb_mbatch_t));
    if (!bs || !out->batches) goto done;
    {
        uint64_t q = 0;
        for (size_t k = 0; k < ntopo; k++) {
            uint64_t passes = pb_topo_passes(topo_list[k], T, G[k]);
            const uint64_t order = target > 0 && nunits_t[k] ? (uint64_t)pb_topo_lockstep_clocks(topo_list[k], T, G[k])
                                                             : passes;
            for (uint32_t f = 0; f < nunits_t[k]; f += G[k]) {
                bs[q].b.topo = (uint32_t)k;
                bs[q].b.first_unit = (uint32_t)(ufirst[k] + f);
                bs[q].b.count = nunits_t[k] - f < G[k] ? nunits_t[k] - f : G[k];
                bs[q].b.G = G[k];
                bs[q].cost = order;
                if (passes > out->max_chain) out->max_chain = passes;
                q++;
            }
        }
        qsort(bs, nb, sizeof(*bs), cmp_batch);
        for (uint64_t i = 0; i < nb; i++) out->batches[i] = bs[i].b;
    }
    out->nbatches = nb;
    /* warps of a team that have no node of a level skip it, so the ALU work
     * of a batch is its one-warp pass count: sum over levels of ceil(G*w/32) */
    out->warp_passes = 0;
    for (size_t k = 0; k < ntopo; k++)
        out->warp_passes += (double)((nunits_t[k] + G[k] - 1) / G[k]) * (double)pb_topo_passes(topo_list[k], 1, G[k]);
    rc = 0;
done:
    free(topo_list); free(ti); free(G); free(nunits_t); free(ufirst); free(ucount); free(bs);
    if (rc != 0) pb_plan_free(out);
    return rc;
}

double pb_plan_makespan(const pb_plan_tables_t *p, uint32_t T, uint64_t R)
{
    /* per pass: ~3500 clocks when latency-bound; ALU: a warp-pass is 32 lanes
     * x 2 compressions (~1400 operations a lane) at ~72 lane-operations per
     * clock per SM */
    (void)T;
    double chain = (double)p->max_chain * 3500.0;
    double sms = p->sms ? p->sms : 148;
    double alu = p->warp_passes * 32.0 * 1400.0 / (72.0 * sms);
    double waves = R && p->nbatches > R ? 1.0 + (double)(p->nbatches - R) / (double)R * 0.5 : 1.0;
    return (chain > alu ? chain : alu) * waves;
}

static int cmp_cand(const void *a, const void *b)
{
    double x = ((const pb_cand_t *)a)->est, y = ((const pb_cand_t *)b)->est;
    return x < y ? -1 : x > y;
}

int pb_plan_rank(const pb_req_t *pr, size_t n, const pose_b200_sched_t *sched, pb_cand_t *out, int cap)
{
    /* every team size and packing rule the caller left open, by estimated
     * makespan (chain-bounded packing, or a lane-efficiency target) */
    const uint32_t gcap = sched && sched->units_per_team ? sched->units_per_team : 32;
    const uint32_t t_lo = sched && sched->team_warps ? sched->team_warps : 1;
    const uint32_t t_hi = sched && sched->team_warps ? sched->team_warps : 8;
    double rules[4] = {0.0, 0.5, 0.7, 0.85};
    int nrules = 4;
    if (sched && sched->lane_efficiency) {
        rules[0] = sched->lane_efficiency == POSE_B200_PACK_CHAIN ? 0.0 : sched->lane_efficiency / 100.0;
        nrules = 1;
    }
    int k = 0;
    for (uint32_t tT = t_lo; tT <= t_hi; tT <<= 1) {
        for (int e = 0; e < nrules && k < cap; e++) {
            pb_plan_tables_t cand;
            if (pb_plan_requests(pr, n, tT, gcap, rules[e], 0.0, &cand) != 0) return -1;
            out[k].T = tT;
            out[k].eff = rules[e];
            out[k].est = pb_plan_makespan(&cand, tT, (uint64_t)cand.sms * 32 / tT);
            k++;
            pb_plan_free(&cand);
        }
    }
    qsort(out, (size_t)k, sizeof(*out), cmp_cand);
    return k;
}

int pb_plan_choose(const pb_req_t *pr, size_t n, const pose_b200_sched_t *sched, uint32_t *T_out, double *eff_out)
{
    pb_cand_t c[16];
    int k = pb_plan_rank(pr, n, sched, c, 16);
    if (k <= 0) return -1;
    *T_out = c[0].T;
    *eff_out = c[0].eff;
    return 0;
}

/* Requests whose topology's chain with 8-warp teams is at least 3/4 of the
 * deepest one's, when some other request's topology is shallower: they run
 * as their own launch beside the rest (1 = deep, 0 = rest, in deep[]).
 * Requests shorter than one super-chunk label nothing and stay with the
 * rest.  Returns the number of deep requests (0 = no split). */
static size_t split_deep(const pb_req_t *pr, size_t n, uint8_t *deep)
{
    uint64_t maxc = 0, minc = UINT64_MAX;
    for (size_t i = 0; i < n; i++) {
        pb_topo_internal_t x;
        deep[i] = 0;
        if (pb_topo_internal(pr[i].topo, &x) != 0 || pr[i].len < x.super_bytes) continue;
        const uint64_t c = pb_topo_passes(pr[i].topo, 8, 1);
        if (c > maxc) maxc = c;
        if (c < minc) minc = c;
        deep[i] = 1; /* has work; decided below */
    }
    if (maxc == 0 || 4 * minc >= 3 * maxc) {
        memset(deep, 0, n);
        return 0; /* every request with work is about as deep as the deepest */
    }
    size_t nd = 0;
    for (size_t i = 0; i < n; i++) {
        if (!deep[i]) continue;
        deep[i] = 4 * pb_topo_passes(pr[i].topo, 8, 1) >= 3 * maxc;
        nd += deep[i];
    }
    return nd;
}

/* The second deep part: among the requests split_deep left shallow, those of
 * the deepest remaining topology, when its chain (8-warp team, one unit) is
 * at least a third of the deepest request's.  They are marked 2 in `deep`;
 * returns how many. */
static size_t split_second(const pb_req_t *pr, size_t n, uint8_t *deep)
{
    uint64_t maxc = 0, c2 = 0;
    const pose_hbm_topo_t *t2 = NULL;
    for (size_t i = 0; i < n; i++) {
        pb_topo_internal_t x;
        if (pb_topo_internal(pr[i].topo, &x) != 0 || pr[i].len < x.super_bytes) continue;
        const uint64_t c = pb_topo_passes(pr[i].topo, 8, 1);
        if (c > maxc) maxc = c;
        if (!deep[i] && c > c2) {
            c2 = c;
            t2 = pr[i].topo;
        }
    }
    if (!t2 || 3 * c2 < maxc) return 0;
    size_t n2 = 0;
    for (size_t i = 0; i < n; i++) {
        pb_topo_internal_t x;
        if (deep[i] || pr[i].topo != t2 || pb_topo_internal(pr[i].topo, &x) != 0 || pr[i].len < x.super_bytes)
            continue;
        deep[i] = 2;
        n2++;
    }
    return n2;
}

/* Size, allocate and upload one launch of a batch; `cap` is the most teams it
 * may hold and `budget` bounds its scratch.  One team per CTA.  Returns 0, or
 * -1 (message on stderr). */
static int part_setup(pose_b200_batch_t *b, batch_part_t *q, const pb_plan_tables_t *pl, uint32_t T,
                      uint64_t cap, uint64_t budget, const pose_b200_sched_t *sched)
{
    q->T = T;
    q->nbatches = pl->nbatches;
    q->njobs = pl->njobs;
    q->units = pl->nunits;
    q->super_chunks = pl->njobs;
    q->nodes = pl->nodes;
    q->Gmax = pl->Gmax;
    q->cv0 = pl->all_cv0;
    q->team_scratch = pl->team_scratch;
    uint64_t R = budget / pl->team_scratch;
    if (R > cap) R = cap;
    if (R > pl->nbatches) R = pl->nbatches;
    if (sched && sched->max_teams && R > sched->max_teams) R = sched->max_teams;
    if (R == 0) {
        fprintf(stderr, "pose_b200_batch_create: one team needs %llu bytes of scratch, over the budget\n",
                (unsigned long long)pl->team_scratch);
        return -1;
    }
    q->grid = (uint32_t)R;
    q->cta_threads = 32 * T;
    q->teams = (uint32_t)R;
    q->scratch_bytes = R * pl->team_scratch;
    if (pb_dev_malloc(&q->d_topos, pl->ntopo * sizeof(pb_topo_view_t)) != cudaSuccess ||
        pb_dev_malloc(&q->d_batches, pl->nbatches * sizeof(pb_mbatch_t)) != cudaSuccess ||
        pb_dev_malloc(&q->d_units, pl->nunits * sizeof(pb_munit_t)) != cudaSuccess ||
        pb_dev_malloc(&q->d_jobs, pl->njobs * sizeof(pb_seedjob_t)) != cudaSuccess ||
        pb_dev_malloc(&q->d_seeds, pl->njobs * 32) != cudaSuccess ||
        pb_dev_malloc(&q->d_scratch, q->scratch_bytes) != cudaSuccess ||
        pb_dev_malloc(&q->d_queue, 64) != cudaSuccess) {
        fprintf(stderr, "pose_b200_batch_create: alloc: %s\n", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    if (cudaMemcpyAsync(q->d_topos, pl->views, pl->ntopo * sizeof(pb_topo_view_t), cudaMemcpyHostToDevice,
                        b->stream) != cudaSuccess ||
        cudaMemcpyAsync(q->d_batches, pl->batches, pl->nbatches * sizeof(pb_mbatch_t), cudaMemcpyHostToDevice,
                        b->stream) != cudaSuccess ||
        cudaMemcpyAsync(q->d_units, pl->units, pl->nunits * sizeof(pb_munit_t), cudaMemcpyHostToDevice,
                        b->stream) != cudaSuccess ||
        cudaMemcpyAsync(q->d_jobs, pl->jobs, pl->njobs * sizeof(pb_seedjob_t), cudaMemcpyHostToDevice,
                        b->stream) != cudaSuccess ||
        cudaStreamSynchronize(b->stream) != cudaSuccess) {
        fprintf(stderr, "pose_b200_batch_create: upload: %s\n", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    return 0;
}

/* Scratch of one chunk copy on the depth kernel. */
static uint64_t depth_copy_bytes(const pb_topo_view2_t *v) { return (uint64_t)(v->gpool ? v->gpool : 1) * 32; }

/* A part on the depth kernel: every unit of pl (one topology, records v2), G
 * (1 to 8) units per CTA, at most `ctas` CTAs, 15 hashing warps.  The caller
 * bounds ctas by the SMs and the scratch budget.  Returns 0, or -1 (message
 * on stderr). */
static int part_setup_wsg(pose_b200_batch_t *b, batch_part_t *q, const pb_plan_tables_t *pl,
                          const pb_topo_view2_t *v2, uint32_t G, uint32_t ctas, uint32_t smem)
{
    const uint32_t NC = 15;
    q->kind = 1;
    q->v2 = *v2;
    q->units_per_cta = G;
    q->T = NC;
    q->units = pl->nunits;
    q->njobs = pl->njobs;
    q->super_chunks = pl->njobs;
    q->nodes = pl->nodes;
    q->Gmax = G;
    q->cv0 = 1;
    q->nbatches = (pl->nunits + G - 1) / G;
    q->grid = (uint32_t)(q->nbatches < ctas ? q->nbatches : ctas);
    q->teams = q->grid;
    q->cta_threads = 32 * (NC + 1);
    q->smem = smem;
    q->team_scratch = (uint64_t)G * depth_copy_bytes(v2);
    q->scratch_bytes = (uint64_t)q->grid * q->team_scratch;
    uint32_t max_smem = 0;
    if (pb_dev_label_ws_prepare(&max_smem) != 0 || pb_ws_smem_bytes(G, NC) > max_smem) {
        fprintf(stderr, "pose_b200_batch_create: shared memory attribute: %s\n", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    if (q->smem > max_smem) q->smem = max_smem;
    if (pb_dev_malloc(&q->d_units, pl->nunits * sizeof(pb_munit_t)) != cudaSuccess ||
        pb_dev_malloc(&q->d_jobs, pl->njobs * sizeof(pb_seedjob_t)) != cudaSuccess ||
        pb_dev_malloc(&q->d_seeds, pl->njobs * 32) != cudaSuccess ||
        pb_dev_malloc(&q->d_scratch, q->scratch_bytes) != cudaSuccess ||
        pb_dev_malloc(&q->d_queue, 64) != cudaSuccess) {
        fprintf(stderr, "pose_b200_batch_create: alloc: %s\n", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    if (cudaMemcpyAsync(q->d_units, pl->units, pl->nunits * sizeof(pb_munit_t), cudaMemcpyHostToDevice,
                        b->stream) != cudaSuccess ||
        cudaMemcpyAsync(q->d_jobs, pl->jobs, pl->njobs * sizeof(pb_seedjob_t), cudaMemcpyHostToDevice,
                        b->stream) != cudaSuccess ||
        cudaStreamSynchronize(b->stream) != cudaSuccess) {
        fprintf(stderr, "pose_b200_batch_create: upload: %s\n", cudaGetErrorString(cudaGetLastError()));
        return -1;
    }
    return 0;
}

/* Capture what one launch needs first onto stream s: chunk seeds and the
 * queue reset. */
static int part_capture_seeds(const pose_b200_batch_t *b, const batch_part_t *q, cudaStream_t s)
{
    if (pb_dev_seed_jobs(q->d_jobs, (uint32_t)q->njobs, (const uint8_t *)b->d_blob, (uint32_t *)q->d_seeds, s) != 0)
        return -1;
    return cudaMemsetAsync(q->d_queue, 0, 64, s) == cudaSuccess ? 0 : -1;
}

/* Capture one launch onto stream s: labeling, scratch and chunk-seed zeroing
 * (events e0/e1 around the labeling kernel when not NULL).  A replay leaves
 * no label or chunk seed behind; the session seeds stay for the next replay
 * and are zeroed when the batch is destroyed. */
static int part_capture(const batch_part_t *q, cudaStream_t s, cudaEvent_t e0, cudaEvent_t e1)
{
    pb_multi_params_t p;
    memset(&p, 0, sizeof(p));
    p.topos = (const pb_topo_view_t *)q->d_topos;
    p.batches = (const pb_mbatch_t *)q->d_batches;
    p.units = (const pb_munit_t *)q->d_units;
    p.seeds = (const uint32_t *)q->d_seeds;
    p.scratch = (uint8_t *)q->d_scratch;
    p.team_scratch_bytes = q->team_scratch;
    p.nbatches = (uint32_t)q->nbatches;
    p.team_warps = q->T;
    p.queue = (unsigned int *)q->d_queue;
    p.table = q->cv0;
    int crc = 0;
    if (e0) crc = cudaEventRecord(e0, s) == cudaSuccess ? 0 : -1;
    if (crc == 0 && q->kind == 1) {
        pb_depth_params_t w;
        memset(&w, 0, sizeof(w));
        w.topo = q->v2;
        w.units = (const pb_munit_t *)q->d_units;
        w.seeds = (const uint32_t *)q->d_seeds;
        w.scratch = (uint8_t *)q->d_scratch;
        w.unit_scratch_bytes = (uint64_t)q->v2.gpool * 32;
        w.nunits = (uint32_t)q->units;
        w.units_per_cta = q->units_per_cta;
        w.team_warps = q->T;
        w.nbatches = (uint32_t)q->nbatches;
        w.queue = (unsigned int *)q->d_queue;
        crc = pb_dev_label_ws(&w, q->grid, q->smem, s);
    } else if (crc == 0) {
        crc = pb_dev_label_multi(&p, q->grid, q->cta_threads, q->smem, s);
    }
    if (crc == 0 && e1) crc = cudaEventRecord(e1, s) == cudaSuccess ? 0 : -1;
    if (crc == 0) crc = cudaMemsetAsync(q->d_scratch, 0, q->scratch_bytes, s) == cudaSuccess ? 0 : -1;
    if (crc == 0) crc = cudaMemsetAsync(q->d_seeds, 0, (size_t)q->njobs * 32, s) == cudaSuccess ? 0 : -1;
    return crc;
}

/* Units (chunk copies) of n requests. */
static uint64_t request_units(const pb_req_t *pr, size_t n)
{
    uint64_t u = 0;
    for (size_t i = 0; i < n; i++) {
        pb_topo_internal_t x;
        if (pb_topo_internal(pr[i].topo, &x) == 0) u += (uint64_t)(pr[i].len / x.super_bytes) * x.copies;
    }
    return u;
}

/* The one topology of all requests with something to label, or NULL. */
static const pose_hbm_topo_t *one_topology(const pb_req_t *pr, size_t n)
{
    const pose_hbm_topo_t *t = NULL;
    for (size_t i = 0; i < n; i++) {
        pb_topo_internal_t x;
        if (pb_topo_internal(pr[i].topo, &x) != 0) return NULL;
        if (pr[i].len < x.super_bytes) continue;
        if (t && t != pr[i].topo) return NULL;
        t = pr[i].topo;
    }
    return t;
}

/* SM clocks of n requests on 16-warp lockstep teams of 16 units, and the
 * longest single unit's; the larger of the latter and the work spread over
 * the SMs is what they need at least. */
static double shallow_work(const pb_req_t *pr, size_t n, double *longest, uint32_t *sms)
{
    double work = 0;
    *longest = 0;
    *sms = 148;
    const pose_hbm_topo_t *last = NULL;
    double c16 = 0, c1 = 0;
    for (size_t i = 0; i < n; i++) {
        pb_topo_internal_t x;
        if (pb_topo_internal(pr[i].topo, &x) != 0 || pr[i].len < x.super_bytes) continue;
        if (pr[i].topo != last) {
            last = pr[i].topo;
            c16 = pb_topo_lockstep_clocks(last, 16, 16) / 16.0;
            c1 = pb_topo_lockstep_clocks(last, 16, 1);
        }
        work += (double)(pr[i].len / x.super_bytes) * x.copies * c16;
        if (c1 > *longest) *longest = c1;
        if (x.sms > 0) *sms = (uint32_t)x.sms;
    }
    return work;
}

static double shallow_makespan(const pb_req_t *pr, size_t n, uint32_t sms)
{
    double longest;
    uint32_t all;
    const double work = shallow_work(pr, n, &longest, &all);
    if (sms == 0 || sms > all) sms = all;
    return longest > work / sms ? longest : work / sms;
}

/* pb_plan_requests with at most gcap units a team, fewer where a team's
 * scratch would not fit `room` (one unit at the least). */
static int plan_within(const pb_req_t *pr, size_t n, uint32_t T, uint32_t gcap, double eff, double target,
                       uint64_t room, pb_plan_tables_t *out)
{
    while (pb_plan_requests(pr, n, T, gcap, eff, target, out) == 0) {
        if (out->team_scratch <= room || gcap == 1) return 0;
        pb_plan_free(out);
        gcap /= 2;
    }
    return -1;
}

int pb_plan_fill(const pb_req_t *reqs, size_t n, uint32_t sms, uint32_t T, uint64_t room, pb_plan_tables_t *out)
{
    const double target = shallow_makespan(reqs, n, sms) / 2.0;
    return plan_within(reqs, n, T, 32, 0.0, target > 0 ? target : 1.0, room, out);
}

/* Batches of the other requests, beside deep parts, take at most this part of
 * the whole's estimate. */
#define PB_FILL_PART (1.0 / 3.0)

/* Add n jobs of t clocks to the SMs' loads, each on the one free first: job
 * k of an SM starts at its load + k t, and the n jobs take the n earliest
 * starts.  Of many jobs all but a few are placed at once, those that start
 * before a time that fewer than n do. */
static void place_jobs(double *load, uint32_t sms, uint64_t n, double t)
{
    if (n > 4ull * sms && t > 0) {
        double lo = 0, hi = t;
        for (uint32_t i = 0; i < sms; i++)
            if (load[i] + t * ((double)n / sms + 1.0) > hi) hi = load[i] + t * ((double)n / sms + 1.0);
        for (int k = 0; k < 40; k++) {
            const double mid = 0.5 * (lo + hi);
            double starts = 0;
            for (uint32_t i = 0; i < sms; i++) starts += load[i] < mid ? ceil((mid - load[i]) / t) : 0.0;
            if (starts <= (double)n) lo = mid;
            else hi = mid;
        }
        for (uint32_t i = 0; i < sms; i++) {
            uint64_t k = load[i] < lo ? (uint64_t)ceil((lo - load[i]) / t) : 0;
            if (k > n) k = n;
            load[i] += t * (double)k;
            n -= k;
        }
    }
    for (uint64_t j = 0; j < n; j++) {
        uint32_t m = 0;
        for (uint32_t i = 1; i < sms; i++)
            if (load[i] < load[m]) m = i;
        load[m] += t;
    }
}

static double most_loaded(const double *load, uint32_t sms)
{
    double m = load[0];
    for (uint32_t i = 1; i < sms; i++)
        if (load[i] > m) m = load[i];
    return m;
}

/* One deep part: G copies per CTA on `ctas` CTAs (0: no such part). */
typedef struct {
    uint32_t G, ctas;
} deep_part_t;

/* Clocks until b1 jobs of t1 on c1 CTAs, then b2 of t2 on c2 CTAs (each on the
 * SM that is free first), and `rest` clocks of other work behind them are
 * done.  That work comes in batches of PB_FILL_PART of an even fill's
 * makespan, which is *even: a choice that leaves the SMs to the deep parts
 * until the end pays for the last batches (256 sessions of 2^12..2^17 blocks,
 * 4 and 5 copies a CTA on 103 and 45 SMs: 1602 ms, 5 and 5 on 82 and 66:
 * 1203). */
static double deep_makespan(double *load, uint32_t sms, uint32_t c1, uint64_t b1, double t1, uint32_t c2, uint64_t b2,
                            double t2, double rest, double *even)
{
    for (uint32_t i = 0; i < sms; i++) load[i] = i < c1 ? t1 * (double)(b1 / c1 + (i < b1 % c1)) : 0.0;
    /* the c2 least loaded SMs are the last ones */
    if (c2) place_jobs(load + (sms - c2), c2, b2, t2);
    double sum = rest;
    for (uint32_t i = 0; i < sms; i++) sum += load[i];
    *even = most_loaded(load, sms);
    if (sum / sms > *even) *even = sum / sms;
    if (rest > 0) place_jobs(load, sms, (uint64_t)(rest / (*even * PB_FILL_PART)) + 1, *even * PB_FILL_PART);
    return most_loaded(load, sms);
}

/* The most scratch that one chunk copy of n requests takes on the lockstep
 * kernel. */
static uint64_t lockstep_copy_bytes(const pb_req_t *pr, size_t n)
{
    uint64_t most = 0;
    for (size_t i = 0; i < n; i++) {
        pb_topo_internal_t x;
        if (pb_topo_internal(pr[i].topo, &x) != 0 || pr[i].len < x.super_bytes) continue;
        if ((uint64_t)x.view.pool * 32 > most) most = (uint64_t)x.view.pool * 32;
    }
    return most;
}

/* CTAs of a depth part: one per batch and SM, as many as `room` holds. */
static uint32_t depth_ctas(uint64_t batches, uint32_t sms, uint64_t room, uint64_t cta_bytes)
{
    uint64_t c = room / cta_bytes;
    if (c > batches) c = batches;
    return (uint32_t)(c < sms ? c : sms);
}

/* Copies per CTA of the two deep parts (pd: nd requests of one topology; pd2:
 * nd2 of another, or none) that the schedule model finishes first, with the
 * other requests ps filled in behind them; fix1, fix2 (nonzero) fix them.
 * Both parts and one copy of the others fit the scratch budget; a part that
 * memory limits has fewer CTAs, which loop over its batches.
 * Among choices that finish together the one with the least work on the SMs.
 * On the 256-session workload that is 5 and 8: 82 CTAs of the 2^17 sessions
 * and 49 of the 2^16 ones beside them.  Where no choice has room for both
 * parts the second is left to the others.  Returns 0, or -1 when no choice
 * fits the shared memory and the budget. */
static int plan_deep(const pb_req_t *pd, size_t nd, const pb_req_t *pd2, size_t nd2, const pb_req_t *ps, size_t ns,
                     uint32_t sms, uint64_t budget, uint32_t fix1, uint32_t fix2, deep_part_t part[2],
                     double *makespan)
{
    pb_topo_view2_t v1, v2;
    uint32_t max_smem = 0, n_sms;
    double longest;
    if (pb_topo_view2(pd[0].topo, &v1) != 0 || pb_dev_label_ws_prepare(&max_smem) != 0) return -1;
    double *load = (double *)malloc(sms * sizeof(*load));
    if (!load) return -1;
    const uint64_t u1 = request_units(pd, nd), u2 = nd2 ? request_units(pd2, nd2) : 0;
    double rest = shallow_work(ps, ns, &longest, &n_sms);
    uint64_t keep = lockstep_copy_bytes(ps, ns);
    double best = -1, best_busy = 0;
    for (int second = nd2 && pb_topo_view2(pd2[0].topo, &v2) == 0; second >= 0 && best < 0; second--) {
        if (!second && nd2) { /* with the others */
            const uint64_t copy = lockstep_copy_bytes(pd2, nd2);
            rest += shallow_work(pd2, nd2, &longest, &n_sms);
            if (copy > keep) keep = copy;
        }
        const uint64_t room = budget > keep ? budget - keep : 0;
        for (uint32_t a = 1; a <= PB_WS_MAX_UNITS; a++) {
            if ((fix1 && a != fix1) || pb_ws_smem_bytes(a, 15) > max_smem) continue;
            const uint64_t b1 = (u1 + a - 1) / a, m1 = depth_copy_bytes(&v1) * a;
            const double t1 = pb_topo_depth_clocks(pd[0].topo, a);
            for (uint32_t c = second ? 1 : 0; c <= (second ? PB_WS_MAX_UNITS : 0); c++) {
                if (c && ((fix2 && c != fix2) || pb_ws_smem_bytes(c, 15) > max_smem)) continue;
                const uint64_t b2 = c ? (u2 + c - 1) / c : 0, m2 = c ? depth_copy_bytes(&v2) * c : 0;
                const double t2 = c ? pb_topo_depth_clocks(pd2[0].topo, c) : 0;
                const uint32_t c1 = depth_ctas(b1, sms, room > m2 ? room - m2 : 0, m1);
                const uint32_t c2 = c1 && c ? depth_ctas(b2, sms, room - c1 * m1, m2) : 0;
                if (!c1 || (c && !c2)) continue;
                double even, busy = t1 * (double)b1 + t2 * (double)b2;
                const double m = deep_makespan(load, sms, c1, b1, t1, c2, b2, t2, rest, &even);
                if (best < 0 || m < 0.999 * best || (m < 1.001 * best && busy < best_busy)) {
                    best = m;
                    best_busy = busy;
                    *makespan = even;
                    part[0] = (deep_part_t){a, c1};
                    part[1] = (deep_part_t){c, c2};
                }
            }
        }
    }
    free(load);
    return best < 0 ? -1 : 0;
}

/* The caller fixes nothing: the schedule model plans every part. */
static int open_schedule(const pose_b200_sched_t *s)
{
    return !s || (!s->team_warps && !s->units_per_team && !s->max_teams && !s->lane_efficiency && !s->flags);
}

pose_b200_batch_t *pose_b200_batch_create(const pose_b200_request_t *reqs, size_t n,
                                          const pose_b200_sched_t *sched)
{
    pose_b200_batch_t *b = NULL;
    pb_req_t *pr = NULL, *pd = NULL, *pd2 = NULL, *ps = NULL;
    uint8_t *blob = NULL, *deep = NULL;
    pb_plan_tables_t pl[3];
    memset(pl, 0, sizeof(pl));
    size_t blob_len = 0, nd = 0, nd2 = 0, ns = 0;
    int dev = -1;

    if (!reqs || n == 0) { fprintf(stderr, "pose_b200_batch_create: no requests\n"); return NULL; }
    if (sched && sched->team_warps && sched->team_warps != 1 && sched->team_warps != 2 && sched->team_warps != 4 &&
        sched->team_warps != 8) {
        fprintf(stderr, "pose_b200_batch_create: team_warps must be 1, 2, 4 or 8\n");
        return NULL;
    }
    if (sched && sched->lane_efficiency > 100 && sched->lane_efficiency != POSE_B200_PACK_CHAIN) {
        fprintf(stderr, "pose_b200_batch_create: lane_efficiency must be a percentage or POSE_B200_PACK_CHAIN\n");
        return NULL;
    }
    for (size_t i = 0; i < n; i++) {
        if (!reqs[i].session_seed && reqs[i].seed_len) { fprintf(stderr, "pose_b200_batch_create: request %zu: NULL seed\n", i); return NULL; }
        if (reqs[i].seed_len > 1016) { fprintf(stderr, "pose_b200_batch_create: request %zu: seed longer than 1016 bytes\n", i); return NULL; }
        blob_len += reqs[i].seed_len;
    }
    pr = (pb_req_t *)calloc(n, sizeof(*pr));
    pd = (pb_req_t *)calloc(n, sizeof(*pd));
    pd2 = (pb_req_t *)calloc(n, sizeof(*pd2));
    ps = (pb_req_t *)calloc(n, sizeof(*ps));
    deep = (uint8_t *)calloc(n, 1);
    blob = (uint8_t *)malloc(blob_len ? blob_len : 1);
    if (!pr || !pd || !pd2 || !ps || !deep || !blob) goto fail_host;
    {
        uint64_t off = 0;
        for (size_t i = 0; i < n; i++) {
            pr[i].topo = reqs[i].topo;
            pr[i].dev_ptr = reqs[i].hbm_dev_ptr;
            pr[i].len = reqs[i].hbm_len;
            pr[i].rbo = reqs[i].region_block_offset;
            pr[i].seed_off = (uint32_t)off;
            pr[i].seed_len = (uint32_t)reqs[i].seed_len;
            if (reqs[i].seed_len) memcpy(blob + off, reqs[i].session_seed, reqs[i].seed_len);
            off += reqs[i].seed_len;
        }
    }
    /* the deep part, unless the caller asks for one launch */
    if (!(sched && (sched->flags & POSE_B200_BATCH_ONE_LAUNCH))) {
        for (size_t i = 0; i < n; i++) if (!pr[i].topo) goto no_split;
        nd = split_deep(pr, n, deep);
        /* POSE_B200_DEEP2=0 keeps the next-deepest topology with the rest */
        const char *e2 = getenv("POSE_B200_DEEP2");
        if (nd && !(e2 && e2[0] == '0')) nd2 = split_second(pr, n, deep);
    }
no_split:
    if (nd) {
        size_t a = 0, c = 0;
        for (size_t i = 0; i < n; i++) {
            if (deep[i] == 1) pd[a++] = pr[i];
            else if (deep[i] == 2) pd2[c++] = pr[i];
            else ps[ns++] = pr[i];
        }
    } else {
        memcpy(ps, pr, n * sizeof(*pr));
        ns = n;
    }
    cudaGetDevice(&dev);
    b = (pose_b200_batch_t *)calloc(1, sizeof(*b));
    if (!b) goto fail_host;
    b->device = dev;
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) goto fail;
    if (nd && cudaStreamCreateWithFlags(&b->stream2, cudaStreamNonBlocking) != cudaSuccess) goto fail;
    if (nd2 && cudaStreamCreateWithFlags(&b->stream3, cudaStreamNonBlocking) != cudaSuccess) goto fail;
    for (int i = 0; i < 8; i++) if (cudaEventCreate(&b->ev[i]) != cudaSuccess) goto fail;
    b->blob_len = blob_len;
    if (pb_dev_malloc(&b->d_blob, blob_len ? blob_len : 1) != cudaSuccess) {
        fprintf(stderr, "pose_b200_batch_create: alloc: %s\n", cudaGetErrorString(cudaGetLastError()));
        goto fail;
    }
    if (blob_len && (cudaMemcpyAsync(b->d_blob, blob, blob_len, cudaMemcpyHostToDevice, b->stream) != cudaSuccess ||
                     cudaStreamSynchronize(b->stream) != cudaSuccess))
        goto fail;
    {
        int occ = 0; /* 8-warp CTAs per SM */
        uint32_t alone_smem = 0;
        /* where the query fails, the default shared memory limit stands: teams
         * of at most 8 warps, no padding */
        const int wide = pb_dev_label_multi_occupancy(256, &occ, &alone_smem) == 0 && occ > 0;
        if (!wide) {
            cudaGetLastError();
            occ = 1;
            alone_smem = 0;
        }
        uint64_t budget = pb_topo_scratch_budget(reqs[0].topo, sched ? sched->scratch_cap_bytes : 0);
        uint64_t deep_ctas = 0;
        const int open_sched = open_schedule(sched);
        double makespan = 0; /* estimated, in clocks, when the deep parts are planned by the model */
        /* deep part: 8-warp teams, units packed (G up to 4) until it holds
         * about half the SMs' team slots */
        if (nd) {
            uint64_t dunits = 0;
            uint32_t sms = 148;
            int one_topo = 1;
            for (size_t i = 0; i < nd; i++) {
                pb_topo_internal_t x;
                if (pb_topo_internal(pd[i].topo, &x) != 0) goto fail;
                dunits += (uint64_t)(pd[i].len / x.super_bytes) * x.copies;
                sms = (uint32_t)x.sms;
                if (pd[i].topo != pd[0].topo) one_topo = 0;
            }
            /* one topology: the depth kernel */
            pb_topo_view2_t v2;
            const char *ek = getenv("POSE_B200_DEEP_KERNEL");
            const char *eg = getenv("POSE_B200_DEEP_UNITS");  /* tuning: copies per CTA, 1 to 8 */
            const char *eu = getenv("POSE_B200_DEEP2_UNITS"); /* the same for the second deep part */
            const uint32_t fix1 = eg && eg[0] >= '1' && eg[0] <= '8' && !eg[1] ? (uint32_t)(eg[0] - '0') : 0;
            const uint32_t fix2 = eu && eu[0] >= '1' && eu[0] <= '8' && !eu[1] ? (uint32_t)(eu[0] - '0') : 0;
            deep_part_t dp[2] = {{0, 0}, {0, 0}};
            int wsg = !(ek && ek[0] == '0') && one_topo && pb_topo_view2(pd[0].topo, &v2) == 0;
            if (wsg) {
                /* copies per CTA of both parts */
                wsg = plan_deep(pd, nd, pd2, nd2, ps, ns, sms, budget, fix1, fix2, dp, &makespan) == 0;
                cudaGetLastError();
            }
            if (wsg) {
                if (pb_plan_requests(pd, nd, 8, 1, 0.9999, 0.0, &pl[1]) != 0 || pl[1].nunits == 0) goto fail;
                if (part_setup_wsg(b, &b->part[1], &pl[1], &v2, dp[0].G, dp[0].ctas, pb_ws_smem_bytes(dp[0].G, 15)) !=
                    0)
                    goto fail;
                /* the next-deepest topology's requests: a third launch of the
                 * depth kernel, on the SMs the first leaves and then on those
                 * it is done with */
                if (dp[1].ctas) {
                    pb_topo_view2_t v2b;
                    if (pb_topo_view2(pd2[0].topo, &v2b) != 0 ||
                        pb_plan_requests(pd2, nd2, 8, 1, 0.9999, 0.0, &pl[2]) != 0 || pl[2].nunits == 0)
                        goto fail;
                    if (part_setup_wsg(b, &b->part[2], &pl[2], &v2b, dp[1].G, dp[1].ctas,
                                       pb_ws_smem_bytes(dp[1].G, 15)) != 0)
                        goto fail;
                }
            } else {
                uint32_t g = 1;
                while (g < 4 && 2 * (dunits + g - 1) / g > (uint64_t)sms * occ) g *= 2;
                /* one copy of the others has to fit beside it */
                const uint64_t k1 = lockstep_copy_bytes(ps, ns), k2 = lockstep_copy_bytes(pd2, nd2);
                const uint64_t keep = k1 > k2 ? k1 : k2, room = budget > keep ? budget - keep : 0;
                if (plan_within(pd, nd, 8, g, 0.9999, 0.0, room, &pl[1]) != 0 || pl[1].nunits == 0) goto fail;
                deep_ctas = pl[1].nbatches;
                if (deep_ctas * 2 > (uint64_t)pl[1].sms * occ) deep_ctas = (uint64_t)pl[1].sms * occ / 2;
                if (part_setup(b, &b->part[1], &pl[1], 8, deep_ctas, room, NULL) != 0) goto fail;
            }
            if (nd2 && !dp[1].ctas) { /* the next-deepest requests stay with the rest */
                for (size_t i = 0; i < nd2; i++) ps[ns++] = pd2[i];
                nd2 = 0;
            }
            const uint64_t used = b->part[1].scratch_bytes + (nd2 ? b->part[2].scratch_bytes : 0);
            budget = budget > used ? budget - used : 0;
        }
        const uint32_t gcap = sched && sched->units_per_team ? sched->units_per_team : 32;
        uint32_t T = wide ? 16 : 8;
        double eff = 0.0;
        const pose_hbm_topo_t *only = NULL;
        uint32_t ukern = 0, uT = 0, uG = 0, uteams = 0;
        if (open_sched && !nd && (only = one_topology(ps, ns)) != NULL &&
            (pb_topo_auto_plan(only, request_units(ps, ns), budget, &ukern, &uT, &uG, &uteams) != 0 ||
             (ukern == 1 && uT > T)))
            ukern = 0;
        pb_topo_view2_t uv2;
        uint32_t umax = 0;
        if (ukern == 3 && (pb_topo_view2(only, &uv2) != 0 || pb_dev_label_ws_prepare(&umax) != 0 ||
                           pb_ws_smem_bytes(uG, 15) > umax)) {
            cudaGetLastError();
            ukern = 0;
        }
        if (ukern == 3) {
            /* one topology, few units: the depth kernel, as a single call */
            if (pb_plan_requests(ps, ns, 8, 1, 0.9999, 0.0, &pl[0]) != 0) goto fail;
            T = 15;
            if (part_setup_wsg(b, &b->part[0], &pl[0], &uv2, uG, uteams, pb_ws_smem_bytes(uG, 15)) != 0) goto fail;
        } else if (open_sched) {
            /* 16-warp teams; batches no longer than a third of the deep
             * parts' makespan (they fill the SMs those leave), or half of
             * what the requests need on all SMs */
            double target = ukern == 1 ? 1e30 : makespan * PB_FILL_PART;
            if (target <= 0) target = shallow_makespan(ps, ns, 0) / 2.0;
            if (target <= 0) target = 1.0;
            if (ukern == 1) T = uT;
            if (plan_within(ps, ns, T, ukern == 1 ? uG : 32, 0.0, target, budget, &pl[0]) != 0) goto fail;
        } else {
            /* beside depth CTAs, which hold their SMs, the rest starts late:
             * its batches are bounded as above, and chain-bounded packing
             * fills them up to that.  (64 requests of 2^10..2^14 blocks,
             * 4-warp teams: 90-157 ms unbounded, 56 bounded.) */
            const double bound = makespan * PB_FILL_PART;
            if (pb_plan_choose(ps, ns, sched, &T, &eff) != 0) goto fail;
            /* a caller's own units per team are kept, and refused when they do not fit */
            const uint64_t room = sched && sched->units_per_team ? UINT64_MAX : budget;
            if (plan_within(ps, ns, T, gcap, eff, eff > 0 ? -bound : bound, room, &pl[0]) != 0) goto fail;
        }
        if (pl[0].nunits == 0 && !nd) { fprintf(stderr, "pose_b200_batch_create: no super-chunk to label\n"); goto fail; }
        if (pl[0].nunits && ukern != 3) {
            uint64_t cap;
            if (makespan > 0) {
                /* beside deep parts 16 warps an SM: two 16-warp teams would
                 * both start on the first SM that the deep parts leave and
                 * end when the second one could have ended elsewhere (256
                 * sessions, 5 and 8 copies a CTA: 1284 against 1181 ms) */
                const uint32_t per_sm = 16 / T;
                b->part[0].smem = per_sm == 1 || !wide ? alone_smem : alone_smem / per_sm - 2048;
                cap = (uint64_t)pl[0].sms * per_sm;
            } else if (open_sched) {
                int o = 1;
                if (pb_dev_label_multi_occupancy(32 * T, &o, NULL) != 0 || o <= 0) o = 1;
                cap = (uint64_t)pl[0].sms * (uint64_t)o;
            } else {
                /* 24 warps an SM: with 32 the batches that run longest share
                 * their SM with more others (256 requests in one launch of
                 * 8-warp teams: 444 teams 1910 ms, 582 teams 2218-2409) */
                const uint64_t taken = (uint64_t)b->part[1].grid + (nd2 ? b->part[2].grid : 0);
                uint64_t slots = (uint64_t)pl[0].sms * (occ < 3 ? occ : 3);
                slots = slots > taken ? slots - taken : 1;
                cap = slots * (256 / (32 * T));
            }
            if (part_setup(b, &b->part[0], &pl[0], T, cap, budget, sched) != 0) goto fail;
        }
        b->nparts = nd2 ? 3 : nd ? 2 : 1;
        b->T = T;
        for (int i = 0; i < b->nparts; i++) {
            const batch_part_t *q = &b->part[i];
            b->nbatches += (uint32_t)q->nbatches;
            b->units += q->units;
            b->super_chunks += q->super_chunks;
            b->nodes += q->nodes;
            b->teams += q->teams;
            b->scratch_bytes += q->scratch_bytes;
            if (q->Gmax > b->Gmax) b->Gmax = q->Gmax;
        }
        b->cv0 = (pl[0].nunits == 0 || b->part[0].cv0) && (!nd || b->part[1].cv0) && (!nd2 || b->part[2].cv0);

        /* capture: every launch's seeds on the batch's stream, then the deep
         * parts forked off and the rest.  Nothing orders the three launches,
         * whose nodes all run at one priority.  (A node that delays the rest,
         * for the deep parts' CTAs to be placed first, changes nothing: 256
         * sessions 1189.8-1190.8 ms without one, 1190.9-1191.2 with; three
         * other mixes 140.7, 313.2 and 393.0 ms either way.) */
        if (cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) goto fail;
        int crc = 0;
        for (int i = b->nparts - 1; i >= 0 && crc == 0; i--)
            if (i > 0 || pl[0].nunits) crc = part_capture_seeds(b, &b->part[i], b->stream);
        if (crc == 0 && nd) {
            crc = cudaEventRecord(b->ev[4], b->stream) == cudaSuccess ? 0 : -1;
            if (crc == 0) crc = cudaStreamWaitEvent(b->stream2, b->ev[4], 0) == cudaSuccess ? 0 : -1;
            if (crc == 0) crc = part_capture(&b->part[1], b->stream2, NULL, NULL);
            if (crc == 0) crc = cudaEventRecord(b->ev[5], b->stream2) == cudaSuccess ? 0 : -1;
        }
        if (crc == 0 && nd2) {
            crc = cudaEventRecord(b->ev[6], b->stream) == cudaSuccess ? 0 : -1;
            if (crc == 0) crc = cudaStreamWaitEvent(b->stream3, b->ev[6], 0) == cudaSuccess ? 0 : -1;
            if (crc == 0) crc = part_capture(&b->part[2], b->stream3, NULL, NULL);
            if (crc == 0) crc = cudaEventRecord(b->ev[7], b->stream3) == cudaSuccess ? 0 : -1;
        }
        if (crc == 0 && pl[0].nunits) {
            crc = part_capture(&b->part[0], b->stream, b->ev[1], b->ev[2]);
        }
        if (crc == 0 && nd) crc = cudaStreamWaitEvent(b->stream, b->ev[5], 0) == cudaSuccess ? 0 : -1;
        if (crc == 0 && nd2) crc = cudaStreamWaitEvent(b->stream, b->ev[7], 0) == cudaSuccess ? 0 : -1;
        cudaError_t ce = cudaStreamEndCapture(b->stream, &b->graph);
        if (crc != 0 || ce != cudaSuccess) {
            fprintf(stderr, "pose_b200_batch_create: graph capture failed: %s\n",
                    cudaGetErrorString(ce != cudaSuccess ? ce : cudaGetLastError()));
            goto fail;
        }
        if (cudaGraphInstantiate(&b->exec, b->graph, 0) != cudaSuccess) {
            fprintf(stderr, "pose_b200_batch_create: graph instantiate: %s\n", cudaGetErrorString(cudaGetLastError()));
            goto fail;
        }
    }
    if (blob) explicit_bzero(blob, blob_len);
    free(pr); free(pd); free(pd2); free(ps); free(deep); free(blob);
    pb_plan_free(&pl[0]); pb_plan_free(&pl[1]); pb_plan_free(&pl[2]);
    return b;
fail:
    batch_free(b);
    b = NULL;
fail_host:
    cudaGetLastError();
    if (blob) explicit_bzero(blob, blob_len);
    free(pr); free(pd); free(pd2); free(ps); free(deep); free(blob);
    pb_plan_free(&pl[0]); pb_plan_free(&pl[1]); pb_plan_free(&pl[2]);
    return NULL;
}

static int pose_b200_batch_run_impl(pose_b200_batch_t *b, pose_b200_stats_t *stats)
{
    if (stats) memset(stats, 0, sizeof(*stats));
    if (!b) return -1;
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != b->device) cudaSetDevice(b->device);
    int rc = -1;
    if (cudaEventRecord(b->ev[0], b->stream) != cudaSuccess) goto out;
    if (cudaGraphLaunch(b->exec, b->stream) != cudaSuccess) goto out;
    if (cudaEventRecord(b->ev[3], b->stream) != cudaSuccess) goto out;
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) goto out;
    rc = 0;
    if (stats) {
        float k = 0, t = 0;
        if (cudaEventElapsedTime(&t, b->ev[0], b->ev[3]) != cudaSuccess) { cudaGetLastError(); t = 0; }
        /* the kernel's own events are nodes of the graph; where the CUDA
         * driver does not time them, or two launches overlap, report the replay */
        if (b->nparts > 1 || cudaEventElapsedTime(&k, b->ev[1], b->ev[2]) != cudaSuccess || k <= 0) {
            cudaGetLastError();
            k = t;
        }
        stats->kernel_ms = k;
        stats->total_ms = t;
        stats->super_chunks = b->super_chunks;
        stats->units = b->units;
        stats->nodes = b->nodes;
        stats->scratch_bytes = b->scratch_bytes;
        stats->team_warps = b->T;
        stats->units_per_team = b->Gmax;
        stats->teams = b->teams;
        stats->kernel_launches = 2 * (uint32_t)b->nparts; /* seeds + labeling per launch */
        stats->used_cv0_table = b->cv0;
        stats->kernel = 4;
    }
out:
    if (rc != 0) fprintf(stderr, "pose_b200_batch_run: CUDA error: %s\n", cudaGetErrorString(cudaGetLastError()));
    if (prev >= 0 && prev != b->device) cudaSetDevice(prev);
    return rc;
}

int pose_b200_batch_run(pose_b200_batch_t *b, pose_b200_stats_t *stats)
{
    nvtxRangePushA("pose_b200: batch replay");
    int rc = pose_b200_batch_run_impl(b, stats);
    nvtxRangePop();
    return rc;
}

int pose_b200_label_batch(const pose_b200_request_t *reqs, size_t n, const pose_b200_sched_t *sched,
                          pose_b200_stats_t *stats)
{
    pose_b200_batch_t *b = pose_b200_batch_create(reqs, n, sched);
    if (!b) return -1;
    int rc = pose_b200_batch_run(b, stats);
    pose_b200_batch_destroy(b);
    return rc;
}

pose_b200_batch_t *pose_b200_batch_autotune(const pose_b200_request_t *reqs, size_t n, const pose_b200_sched_t *sched,
                                            uint32_t trials, pose_b200_sched_t *chosen, pose_b200_stats_t *stats)
{
    if (stats) memset(stats, 0, sizeof(*stats));
    if (!reqs || n == 0) { fprintf(stderr, "pose_b200_batch_autotune: no requests\n"); return NULL; }
    pb_req_t *pr = (pb_req_t *)calloc(n, sizeof(*pr));
    if (!pr) return NULL;
    for (size_t i = 0; i < n; i++) { /* the ranking needs no seeds */
        pr[i].topo = reqs[i].topo;
        pr[i].dev_ptr = reqs[i].hbm_dev_ptr;
        pr[i].len = reqs[i].hbm_len;
        pr[i].rbo = reqs[i].region_block_offset;
    }
    pb_cand_t c[16];
    int k = pb_plan_rank(pr, n, sched, c, 16);
    free(pr);
    if (k <= 0) return NULL;
    if (trials == 0) trials = 3;
    if ((int)trials < k) k = (int)trials;
    pose_b200_batch_t *best = NULL;
    double best_ms = 0;
    for (int i = 0; i < k; i++) {
        pose_b200_sched_t s;
        if (sched) s = *sched;
        else memset(&s, 0, sizeof(s));
        s.team_warps = c[i].T;
        s.lane_efficiency = c[i].eff > 0 ? (uint32_t)(c[i].eff * 100.0 + 0.5) : POSE_B200_PACK_CHAIN;
        pose_b200_batch_t *b = pose_b200_batch_create(reqs, n, &s);
        if (!b) continue;
        pose_b200_stats_t st;
        /* the first replay of a process pays one-time costs: warm up once */
        int rc = best ? 0 : pose_b200_batch_run(b, NULL);
        if (rc == 0) rc = pose_b200_batch_run(b, &st);
        if (rc != 0) { pose_b200_batch_destroy(b); continue; }
        if (!best || st.total_ms < best_ms) {
            pose_b200_batch_destroy(best);
            best = b;
            best_ms = st.total_ms;
            if (chosen) *chosen = s;
            if (stats) *stats = st;
        } else {
            pose_b200_batch_destroy(b);
        }
    }
    if (!best) fprintf(stderr, "pose_b200_batch_autotune: no candidate schedule ran\n");
    return best;
}
