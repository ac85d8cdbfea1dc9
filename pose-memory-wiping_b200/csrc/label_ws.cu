/*
 * label_ws.cu — warp-specialised labeling kernels for the depth-bound regime
 * (few chunk copies per SM; sm_100a).
 *
 * When a launch has about one chunk copy per SM, its time is the number of
 * dependency levels times the time of one level, and a level's floor is two
 * dependent compressions (block 1 needs the predecessors, block 2 needs
 * block 1).  Everything else a level does — finding its width, loading node
 * records, block-0 chaining values and predecessors born earlier — is taken
 * off that path, using the pipelined records of topology.c (PB_REF_*):
 *
 *   CTA = NC hashing warps + 1 producer warp; G (1 to 8) chunk copies of one
 *   topology ("units") run in lockstep, so a level of width w is w * G items
 *   (item k: node k / G of unit k % G).
 *   During level l the producer
 *     - copies the records of level l+2 into a three-stage ring (cp.async),
 *       writes that level's start and width into the ring header, and
 *       prefetches records and block-0 values further ahead into L2;
 *     - from the records of level l+1 (copied during level l-1), copies the
 *       block-0 chaining value and every predecessor born at level l-1 or
 *       earlier (complete since the barrier that ended level l-1) of every
 *       item into a two-stage data area (cp.async), then waits for its copies.
 *   During level l the hashing threads hash their item: its record is already
 *   in registers (read during level l-1), its operands are in the data area
 *   or, when born at level l-1, in the unit's shared-memory label pool (or in
 *   global memory when that level overflowed the pool).  Meanwhile they read
 *   their record of level l+1.  One barrier of the whole CTA ends the level.
 *
 * Two ways to hash, chosen per level by its item count:
 *   - at most PB_QUAD_ITEMS items: four lanes per item (quad_compress).  Up
 *     to 32 items are then one warp per SM sub-partition, whose compression
 *     takes 755 clocks instead of 964, in code a third as long; 85 % of the
 *     levels at chunk_blocks 2^17 are at most 32 wide.  Up to 64 items it
 *     still wins (824 clocks for two warps a sub-partition); above, the ALU
 *     pipe is full and one lane per item is faster;
 *   - more: one lane per item, NC * 32 at a time, the first staged by the
 *     producer, further items with direct loads.
 *
 * No thread waits on anything but its own cp.async groups and CTA or cluster
 * barriers: there are no spin-waits.
 */
#include "b3_device.cuh"
#include "kernels.h"

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cg = cooperative_groups;

namespace pb {
namespace {

/* Levels of at most this many items are hashed by the first eight warps
 * alone: the other hashing warps skip to the next wider level. */
constexpr uint32_t PB_NARROW_ITEMS = 64;
constexpr uint32_t PB_NARROW_WARPS = PB_NARROW_ITEMS / 8;
/* How far ahead of the records it copies (in nodes) the producer prefetches
 * into L2: a few levels, so that DRAM latency is not on its path. */
constexpr uint32_t PB_PREFETCH_AHEAD = 512;

__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc)
{
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
/* A value that every lane of the warp holds, in a form that the compiler
 * knows to be so: it then knows that branches on it keep the warp converged,
 * as the shuffles behind them need. */
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __shfl_sync(0xFFFFFFFFu, x, 0); }
/* Barrier of the first `threads` threads of the CTA's narrow group. */
__device__ __forceinline__ void narrow_sync(uint32_t threads)
{
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ void put8(uint32_t *w, uint4 a, uint4 b)
{
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}

/* Dynamic shared memory, in uint4 units from smem[0]:
 *   empty [2]            the record of no node
 *   hdr   [3]            (level start, width) of each ring stage
 *   ctx   [G][2]         UnitCtx of each unit
 *   msg   [G][4]         block 2 of each unit: chunk seed | descriptor
 *   tab   [G][28]        the same laid out for quads (quad_table_entry)
 *   pool  [PB_CSM + 1][G][2]  next-level labels, slot-major: the G lanes of a
 *                        node read and write neighbouring entries (one pool
 *                        after another would put them all on the same banks);
 *                        the last slot is zero, an absent predecessor
 *   rec   [3][slots][2]  records, ring of three levels
 *   dat   [2][nthr][6]   per item: block-0 value, predecessor 0, predecessor 1
 * with nthr = 32 NC hashing threads and slots = nthr / G staged nodes. */
struct Layout {
    uint32_t nthr, slots, G, ctx, msg, tab, pool, rec, dat;
    __device__ __forceinline__ Layout(uint32_t nthr_, uint32_t G_)
        : nthr(nthr_), slots(nthr_ / G_), G(G_), ctx(5), msg(5 + 2 * G_), tab(5 + 6 * G_), pool(5 + 34 * G_),
          rec(pool + 2 * G_ * (PB_CSM + 1)), dat(rec + 6 * (nthr_ / G_))
    {
    }
    static constexpr uint32_t empty = 0, hdr = 2;
    __device__ __forceinline__ uint32_t r(uint32_t st, uint32_t j) const { return rec + (st * slots + j) * 2; }
    __device__ __forceinline__ uint32_t d(uint32_t st, uint32_t k) const { return dat + (st * nthr + k) * 6; }
    __device__ __forceinline__ uint32_t upool(uint32_t u) const { return pool + 2 * u; }
};

struct __align__(16) UnitCtx {
    uint4 *gscr;       /* the unit's global pool, slot * 2 */
    uint8_t *out;      /* where local output rank 0 of its copy goes */
    uint32_t rank_lim; /* ranks below this are kept */
    uint32_t copy;
    uint64_t pad;
};
static_assert(sizeof(UnitCtx) == 32, "two uint4 a unit");

/* A thread's item of a level: its record, and where its operands are in
 * shared memory (byte offsets, so that nothing is left to compute when the
 * level begins): predecessors (a zero entry for an absent one or one that is
 * in the global pool) and block-0 value. */
struct Desc {
    uint32_t x, y, z, gslot, sslot, rank, s0, s1, v;
    uint32_t global; /* nonzero when a predecessor is in the global pool */
};

__device__ __forceinline__ uint4 at16(const uint4 *smem, uint32_t off)
{
    return *reinterpret_cast<const uint4 *>(reinterpret_cast<const char *>(smem) + off);
}

__device__ __forceinline__ bool from_global(uint32_t ref)
{
    return (ref & (PB_REF_PREV | PB_REF_SMEM)) == PB_REF_PREV;
}

/* Where an operand is: staged at `staged`, or in the unit's pool. */
__device__ __forceinline__ uint32_t operand_at(uint32_t place, uint32_t pool, uint32_t staged, uint32_t G2)
{
    return (place & PB_PLACE_STAGED) ? staged : pool + (place & PB_PLACE_SLOT_MASK) * G2;
}

/* Descriptor of a staged item: record at smem[rec], operands staged at dat
 * index `item`; an empty one when !ok.  Free of branches, so that its loads
 * and selects fill the issue slots that a compression leaves idle. */
__device__ __forceinline__ Desc load_desc(const uint4 *smem, bool ok, uint32_t rec, uint32_t item, uint32_t pool,
                                          uint32_t G2)
{
    const uint32_t at = ok ? rec : Layout::empty;
    const uint4 r0 = smem[at], r1 = smem[at + 1];
    Desc d;
    d.x = r0.x;
    d.y = r0.y;
    d.z = r0.z;
    d.gslot = r0.w;
    d.sslot = r1.x;
    d.rank = r1.y;
    d.s0 = operand_at(r1.z, pool, item + 2, G2) * 16;
    d.s1 = operand_at(r1.w, pool, item + 4, G2) * 16;
    d.v = item * 16;
    d.global = (r1.z | r1.w) & PB_PLACE_GLOBAL;
    return d;
}

/* Producer: records of `lv` (when < L) into ring stage lv % 3, its header,
 * and the prefetch of what later levels need (copies: bit per copy in use). */
template <class P>
__device__ __forceinline__ void stage_records(const P &p, uint4 *smem, const Layout &o, uint32_t lv, uint32_t lane,
                                              uint32_t copies)
{
    const pb_topo_view2_t &tp = p.topo;
    const uint32_t st = lv % 3;
    if (lv >= tp.L) { /* past the end: an empty level */
        if (lane == 0) smem[Layout::hdr + st] = make_uint4(0, 0, 0, 0);
        return;
    }
    const uint32_t ls = __ldg(tp.lstart + lv), w = __ldg(tp.lstart + lv + 1) - ls;
    const uint32_t n = w < o.slots ? w : o.slots;
    for (uint32_t j = lane; j < n; j += 32) {
        const uint4 *src = tp.recs2 + 2 * (size_t)(ls + j);
        uint4 *dst = smem + o.r(st, j);
        cp_async16(dst, src);
        cp_async16(dst + 1, src + 1);
        const uint32_t pos = ls + j + PB_PREFETCH_AHEAD;
        if ((pos & 3u) == 0 && pos < tp.S) { /* a 128-byte line: four nodes */
            prefetch_l2(tp.recs2 + 2 * (size_t)pos);
            if (copies & 1u) prefetch_l2(tp.cv0 + 2 * (size_t)pos);
            if (copies & 2u) prefetch_l2(tp.cv0 + 2 * ((size_t)tp.S + pos));
        }
    }
    if (lane == 0) smem[Layout::hdr + st] = make_uint4(ls, w, 0, 0);
}

/* Producer: block-0 values and older predecessors of level `lv` into data
 * stage lv & 1, for every item of the level's staged nodes whose unit is in
 * the batch (cnt units), from its records (ring stage lv % 3, already
 * complete).  The lanes stride over the items; node = item / G by a
 * multiply-high with ginv = ceil(2^32 / G), exact for these counts. */
template <class P>
__device__ __forceinline__ void stage_data(const P &p, uint4 *smem, const Layout &o, uint32_t cnt, uint32_t lv,
                                           uint32_t lane, uint32_t ginv)
{
    if (lv >= p.topo.L) return;
    const uint4 h = smem[Layout::hdr + lv % 3];
    const uint32_t ls = h.x, w = h.y, G = o.G;
    const uint32_t ns = w < o.slots ? w : o.slots;
    const uint32_t rs = lv % 3, ds = lv & 1;
    for (uint32_t k = lane; k < ns * G; k += 32) {
        const uint32_t j = G == 1 ? k : __umulhi(k, ginv), u = k - j * G;
        if (u >= cnt) continue;
        const UnitCtx *cx = reinterpret_cast<const UnitCtx *>(smem + o.ctx) + u;
        const uint4 r0 = smem[o.r(rs, j)];
        uint4 *d = smem + o.d(ds, k);
        const uint4 *c = p.topo.cv0 + ((size_t)cx->copy * p.topo.S + ls + j) * 2;
        cp_async16(d, c);
        cp_async16(d + 1, c + 1);
        const uint32_t np = (r0.x >> PB_REC_NP_SHIFT) & 3u;
        if (np >= 1 && !(r0.y & PB_REF_PREV)) {
            const uint4 *s = cx->gscr + (size_t)(r0.y & PB_REF_SLOT_MASK) * 2;
            cp_async16(d + 2, s);
            cp_async16(d + 3, s + 1);
        }
        if (np >= 2 && !(r0.z & PB_REF_PREV)) {
            const uint4 *s = cx->gscr + (size_t)(r0.z & PB_REF_SLOT_MASK) * 2;
            cp_async16(d + 4, s);
            cp_async16(d + 5, s + 1);
        }
    }
}

/* The batch's units in shared memory: context, block 2 and its quad table
 * (all threads of the CTA; the caller's barrier follows). */
__device__ __forceinline__ void setup_units(const pb_depth_params_t &p, uint4 *smem, const Layout &o, uint32_t batch,
                                            uint32_t cnt, uint32_t pools, uint32_t t, uint32_t nt)
{
    const pb_topo_view2_t &tp = p.topo;
    if (t == 0) smem[Layout::empty] = make_uint4(0, 0, 0, PB_NO_SLOT);
    if (t == 1) smem[Layout::empty + 1] = make_uint4(PB_NO_SLOT, PB_NO_RANK, PB_CSM, PB_CSM);
    for (uint32_t k = t; k < 2 * o.G; k += nt) smem[o.pool + 2 * o.G * PB_CSM + k] = make_uint4(0, 0, 0, 0);
    for (uint32_t k = t; k < cnt * 28; k += nt) {
        const uint32_t u = k / 28, e = k - u * 28;
        const uint32_t unit = batch * o.G + u;
        uint64_t out;
        uint32_t seed, copy;
        if (p.units) {
            const pb_munit_t mu = p.units[unit];
            out = mu.out;
            seed = mu.seed;
            copy = mu.copy;
        } else {
            seed = unit >> p.copies_log2;
            copy = unit & ((1u << p.copies_log2) - 1u);
            out = (uint64_t)(uintptr_t)p.persist + (p.first_super + seed) * p.super_bytes;
        }
        uint32_t m[16];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            m[i] = p.seeds[8 * (size_t)seed + i];
            m[8 + i] = tp.desc[i];
        }
        smem[o.tab + u * 28 + e] = quad_table_entry(m, e);
        if (e < 4) smem[o.msg + u * 4 + e] = make_uint4(m[4 * e], m[4 * e + 1], m[4 * e + 2], m[4 * e + 3]);
        if (e == 4) {
            UnitCtx *cx = reinterpret_cast<UnitCtx *>(smem + o.ctx) + u;
            cx->gscr = reinterpret_cast<uint4 *>(p.scratch + ((uint64_t)pools + u) * p.unit_scratch_bytes);
            cx->out = reinterpret_cast<uint8_t *>(out) + (copy ? (size_t)tp.half_w * 32 : 0);
            cx->rank_lim = copy ? tp.retained : tp.half_w;
            cx->copy = copy;
        }
    }
}

/* One node by one lane: message block 1 in m, chaining value of block 0 in
 * cv, block 2 at smem[msg]; cv becomes the label.  Both blocks run the same
 * code: the compression is long straight-line code, and about two copies of
 * it run at full speed (measured: one warp's compression takes 966 clocks in a
 * loop of one copy, 1007 of two, 2060 of three, 2420 of four to eight). */
__device__ __forceinline__ void lane_hash(const uint4 *smem, uint32_t msg, uint32_t (&cv)[8], uint32_t (&m)[16])
{
    uint32_t flags = kFlagsBlock1;
#pragma unroll 1
    for (uint32_t last = 0; last <= opaque_one(); last++) { /* twice; a known count would be unrolled */
        compress(cv, m, 64, flags);
        flags = kFlagsBlock2;
        put8(m, smem[msg], smem[msg + 1]);
        put8(m + 8, smem[msg + 2], smem[msg + 3]);
    }
}

/* A label of a directly loaded item: pool is the unit's shared-memory pool
 * (of this CTA, or of the cluster's rank 0). */
__device__ __forceinline__ void load_label(uint32_t *w, uint32_t ref, const uint4 *pool, uint32_t G2,
                                           const uint4 *gscr)
{
    const uint32_t slot = ref & PB_REF_SLOT_MASK;
    const uint4 *s = (ref & (PB_REF_PREV | PB_REF_SMEM)) == (PB_REF_PREV | PB_REF_SMEM) ? pool + (size_t)slot * G2
                                                                                        : gscr + (size_t)slot * 2;
    put8(w, s[0], s[1]);
}

__device__ __forceinline__ void lane_store(const uint32_t (&cv)[8], uint32_t x, uint32_t gslot, uint32_t sslot,
                                           uint32_t rank, uint4 *pool, uint32_t G2, const UnitCtx *cx)
{
    const uint4 o0 = make_uint4(cv[0], cv[1], cv[2], cv[3]);
    const uint4 o1 = make_uint4(cv[4], cv[5], cv[6], cv[7]);
    if (sslot != PB_NO_SLOT) {
        pool[(size_t)sslot * G2] = o0;
        pool[(size_t)sslot * G2 + 1] = o1;
    }
    if (gslot != PB_NO_SLOT) {
        uint4 *d = cx->gscr + (size_t)gslot * 2;
        d[0] = o0;
        d[1] = o1;
    }
    if ((x & PB_REC_OUT_BIT) && rank < cx->rank_lim) {
        uint4 *d = reinterpret_cast<uint4 *>(cx->out + (size_t)rank * 32);
        d[0] = o0;
        d[1] = o1;
    }
}

/* Record, block-0 value and predecessors of the node at level-order position
 * pos, loaded on the spot. */
template <class P>
__device__ __forceinline__ void load_direct(const P &p, uint32_t pos, const UnitCtx *cx, const uint4 *pool,
                                            uint32_t (&m)[16], uint32_t (&cv)[8], uint32_t &x, uint32_t &gslot,
                                            uint32_t &sslot, uint32_t &rank)
{
    const uint4 *rp = p.topo.recs2 + 2 * (size_t)pos;
    const uint4 r0 = __ldg(rp), r1 = __ldg(rp + 1);
    const uint32_t np = (r0.x >> PB_REC_NP_SHIFT) & 3u;
#pragma unroll
    for (int i = 0; i < 16; i++) m[i] = 0;
    if (np >= 1) load_label(m, r0.y, pool, 2 * p.units_per_cta, cx->gscr);
    if (np >= 2) load_label(m + 8, r0.z, pool, 2 * p.units_per_cta, cx->gscr);
    const uint4 *c = p.topo.cv0 + ((size_t)cx->copy * p.topo.S + pos) * 2;
    put8(cv, __ldg(c), __ldg(c + 1));
    x = r0.x; gslot = r0.w; sslot = r1.x; rank = r1.y;
}

/* What a quad does between the rounds of its block-1 compression: read the
 * next level's header and its own record there, both complete since before
 * this level began, and work out where its operands will be. */
struct NextLevel {
    const uint4 *smem;
    uint32_t G, quad_max, warp, j4, pool, lane4; /* the quad's item; lane4 = 4 * lane in the quad */
    bool ok;
    uint32_t hdr, rec, item; /* of the next level: ring header, record and data area (uint4 indices) */
    uint32_t ls, w, global;
    bool quads, busy;
    Desc d;
    uint4 h, r0, r1;

    template <int R>
    __device__ __forceinline__ void at()
    {
        if (R == 0) {
            h = smem[hdr];
        } else if (R == 1) {
            ls = h.x;
            w = uniform(h.y);
        } else if (R == 2) {
            quads = w * G <= quad_max;
            busy = quads && warp * 8 < w * G;
            const uint32_t from = ok && quads && j4 < w ? rec : Layout::empty;
            r0 = smem[from];
            r1 = smem[from + 1];
        } else if (R == 3) {
            d.x = r0.x;
            d.y = r0.y;
            d.z = r0.z;
            d.gslot = r0.w;
            d.sslot = r1.x;
            d.rank = r1.y;
        } else if (R == 4) {
            d.s0 = operand_at(r1.z, pool, item + 2, 2 * G) * 16;
            d.s1 = operand_at(r1.w, pool, item + 4, 2 * G) * 16;
            d.v = item * 16 + lane4;
            d.global = (r1.z | r1.w) & PB_PLACE_GLOBAL;
        } else if (R == 5) {
            global = __any_sync(0xFFFFFFFFu, d.global != 0);
        }
    }
};

/* All levels of one batch of cnt units, by the whole CTA (rank 0 of a cluster
 * when CLUSTER).  Shared memory is set up (setup_units) and a barrier has
 * passed. */
template <bool CLUSTER>
__device__ __forceinline__ void depth_levels(const pb_depth_params_t &p, uint4 *smem, const Layout &o, uint32_t cnt)
{
    const pb_topo_view2_t &tp = p.topo;
    const uint32_t L = tp.L, G = o.G, nthr = o.nthr;
    const uint32_t warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const uint32_t c = threadIdx.x;
    const uint32_t ginv = G > 1 ? (uint32_t)((0x100000000ull + G - 1) / G) : 0u;
    const UnitCtx *ctx = reinterpret_cast<const UnitCtx *>(smem + o.ctx);
    const uint32_t sw = CLUSTER ? p.split_width : 0xFFFFFFFFu;
    const uint32_t narrow_max = nthr / 4 < PB_NARROW_ITEMS ? nthr / 4 : PB_NARROW_ITEMS;
    const uint32_t narrow_threads = 32 * ((nthr / 32 < PB_NARROW_WARPS ? nthr / 32 : PB_NARROW_WARPS) + 1);
    /* A level that every hashing warp takes part in; the boundary between two
     * levels that both are not is a barrier of the narrow group alone. */
    const auto all_hands = [&](uint32_t wl) { return wl * G > narrow_max || (CLUSTER && wl > sw); };
    /* Boundary between a level of w nodes and the next, of wn. */
    const auto boundary = [&](uint32_t w, uint32_t wn) {
        if (CLUSTER && (w > sw || wn > sw)) cg::this_cluster().sync();
        else if (all_hands(w) || all_hands(wn)) __syncthreads();
        else narrow_sync(narrow_threads);
    };

    if (warp == nthr / 32) { /* the producer */
        uint32_t copies = 0;
        for (uint32_t u = 0; u < cnt; u++) copies |= 1u << ctx[u].copy;
        stage_records(p, smem, o, 0, lane, copies);
        stage_records(p, smem, o, 1, lane, copies);
        cp_async_commit();
        cp_async_wait_all();
        __syncwarp();
        stage_data(p, smem, o, cnt, 0, lane, ginv);
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
        uint32_t w = uniform(smem[Layout::hdr].y);
        if (CLUSTER && w > sw) cg::this_cluster().sync(); /* boundary 0 */
        __syncthreads(); /* every warp has read level 0 */
        for (uint32_t l = 0; l < L; l++) {
            const uint32_t wn = uniform(smem[Layout::hdr + (l + 1) % 3].y);
            stage_data(p, smem, o, cnt, l + 1, lane, ginv);
            stage_records(p, smem, o, l + 2, lane, copies);
            cp_async_commit();
            cp_async_wait_all();
            boundary(w, wn); /* l + 1 */
            w = wn;
        }
        return;
    }

    const QuadLane q(lane);
    /* this thread's item in the two modes: quad k4 or lane c; node j, unit u */
    const uint32_t k4 = c >> 2;
    const uint32_t j4 = G == 1 ? k4 : __umulhi(k4, ginv), u4 = k4 - j4 * G;
    const uint32_t j1 = G == 1 ? c : __umulhi(c, ginv), u1 = c - j1 * G;
    const bool ok4 = u4 < cnt, ok1 = u1 < cnt && c < o.slots * G;
    const uint32_t pool4 = o.upool(u4), pool1 = o.upool(u1);
    const uint32_t quad_max = nthr / 4;
    uint4 *const gscr4 = ok4 ? ctx[u4].gscr : nullptr;
    uint8_t *const out4 = ok4 ? ctx[u4].out : nullptr;
    const uint32_t lim4 = ok4 ? ctx[u4].rank_lim : 0;
    const uint4 *const tab4 = smem + o.tab + (ok4 ? u4 : 0) * 28 + q.i;
    const uint4 tab_first = *tab4;

    __syncthreads(); /* levels 0 and 1 are staged */
    const auto quad_desc = [&](uint32_t lv, uint32_t st, uint32_t wl) {
        Desc n = load_desc(smem, ok4 && j4 < wl, o.r(st, j4), o.d(lv & 1, k4), pool4, 2 * G);
        n.v += 4 * q.i;
        return n;
    };
    const auto lane_desc = [&](uint32_t lv, uint32_t st, uint32_t wl) {
        return load_desc(smem, ok1 && j1 < wl, o.r(st, j1), o.d(lv & 1, c), pool1, 2 * G);
    };
    /* The level's start and width, this warp's part in it, and the ring stage
     * of the next level. */
    uint32_t ls, w, st1, global;
    bool busy; /* this warp has a quad with an item */
    Desc d;
    const auto enter = [&](uint32_t lv) {
        const uint32_t st = lv % 3;
        ls = smem[Layout::hdr + st].x;
        w = uniform(smem[Layout::hdr + st].y);
        st1 = st == 2 ? 0 : st + 1;
        busy = w * G <= quad_max && warp * 8 < w * G;
        d = w * G <= quad_max ? quad_desc(lv, st, w) : lane_desc(lv, st, w);
        global = __any_sync(0xFFFFFFFFu, d.global != 0);
    };
    const bool skips = warp >= PB_NARROW_WARPS;
    if (CLUSTER && uniform(smem[Layout::hdr].y) > sw) cg::this_cluster().sync(); /* boundary 0 */
    enter(0);
    /* A warp reads the ring only at levels whose next boundary it passes: past
     * one that it skips the producer may already have refilled the stage
     * (level 0's in level 1).  Level 0 is read by all: the producer waits for
     * them.  (Its width read elsewhere by the warps that skip it, in place of
     * this barrier: 471.7 ms for 32 chunks of 2^17, 904 for 4 of 2^18, 709 for
     * 512 of 2^16; with it 470.4, 897 and 708.) */
    __syncthreads();
#pragma unroll 1
    for (uint32_t l = 0; l < L;) {
        if (skips && !all_hands(w)) {
            /* to the next level of all hands, found in the level offsets */
            for (bool found = false; l < L && !found;) {
                const uint32_t lv = l + lane;
                const bool hit = lv < L && all_hands(__ldg(tp.lstart + lv + 1) - __ldg(tp.lstart + lv));
                const uint32_t mask = __ballot_sync(0xFFFFFFFFu, hit);
                found = mask != 0;
                l += found ? __ffs(mask) - 1 : 32;
            }
            if (l >= L) break;
            boundary(uniform(__ldg(tp.lstart + l) - __ldg(tp.lstart + l - 1)),
                     uniform(__ldg(tp.lstart + l + 1) - __ldg(tp.lstart + l))); /* l */
            enter(l);
        }
        /* Every mode reads level l + 1's header, and its record when it has
         * one, while level l runs: they were complete before level l began. */
        if (busy) {
            /* a run of levels in which this warp has quads with items, in a
             * loop of its own: straight-line code with one jump a level */
#pragma unroll 1
            do {
                const uint32_t *v = reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(smem) + d.v);
                uint32_t va = v[0], vb = v[4];
                uint32_t m[16];
                put8(m, at16(smem, d.s0), at16(smem, d.s0 + 16));
                put8(m + 8, at16(smem, d.s1), at16(smem, d.s1 + 16));
                if (global) {
                    if (from_global(d.y)) load_label(m, d.y, nullptr, 0, gscr4);
                    if (from_global(d.z)) load_label(m + 8, d.z, nullptr, 0, gscr4);
                }
                NextLevel n;
                n.smem = smem; n.G = G; n.quad_max = quad_max; n.warp = warp; n.j4 = j4; n.pool = pool4;
                n.lane4 = 4 * q.i; n.ok = ok4; n.hdr = Layout::hdr + st1; n.rec = o.r(st1, j4);
                n.item = o.d((l + 1) & 1, k4);
                quad_compress(va, vb, m, kFlagsBlock1, q, n);
                quad_compress_table(va, vb, tab_first, tab4, kFlagsBlock2, q);
                if (d.sslot != PB_NO_SLOT) {
                    uint32_t *t = reinterpret_cast<uint32_t *>(smem + pool4 + d.sslot * 2 * G) + q.i;
                    t[0] = va;
                    t[4] = vb;
                }
                if (d.gslot != PB_NO_SLOT) {
                    uint32_t *t = reinterpret_cast<uint32_t *>(gscr4 + (size_t)d.gslot * 2) + q.i;
                    t[0] = va;
                    t[4] = vb;
                }
                if ((d.x & PB_REC_OUT_BIT) && d.rank < lim4) {
                    uint32_t *t = reinterpret_cast<uint32_t *>(out4 + (size_t)d.rank * 32) + q.i;
                    t[0] = va;
                    t[4] = vb;
                }
                d = n.d;
                global = n.global;
                busy = n.busy;
                boundary(w, n.w); /* l + 1 */
                ls = n.ls;
                w = n.w;
                st1 = st1 == 2 ? 0 : st1 + 1;
                l++;
            } while (busy && l < L);
            if (w * G > quad_max) d = lane_desc(l, st1 == 0 ? 2 : st1 - 1, w);
        } else {
            const uint4 h1 = smem[Layout::hdr + st1];
            const uint32_t w1 = uniform(h1.y);
            busy = w1 * G <= quad_max && warp * 8 < w1 * G;
            const Desc dl = d;
            if (w1 * G > quad_max) {
                d = lane_desc(l + 1, st1, w1);
            } else if (busy) {
                d = quad_desc(l + 1, st1, w1);
                global = __any_sync(0xFFFFFFFFu, d.global != 0);
            }
            if (w * G > quad_max) {
                uint32_t lim = ok1 ? w : 0;
                if (CLUSTER && w > sw) { /* split: rank 0 stops at ceil(w / C) nodes */
                    const uint32_t per = (w + p.cluster - 1) / p.cluster, a = per > nthr ? per - nthr : 0;
                    lim = nthr + a < w ? nthr + a : w;
                }
                const UnitCtx *cx = ctx + u1;
#pragma unroll 1
                for (uint32_t j = j1; j < lim; j += o.slots) {
                    uint32_t m[16], cv[8], x, gslot, sslot, rank;
                    if (j == j1) { /* staged */
                        put8(m, at16(smem, dl.s0), at16(smem, dl.s0 + 16));
                        put8(m + 8, at16(smem, dl.s1), at16(smem, dl.s1 + 16));
                        put8(cv, at16(smem, dl.v), at16(smem, dl.v + 16));
                        if (dl.global && from_global(dl.y)) load_label(m, dl.y, nullptr, 0, cx->gscr);
                        if (dl.global && from_global(dl.z)) load_label(m + 8, dl.z, nullptr, 0, cx->gscr);
                        x = dl.x; gslot = dl.gslot; sslot = dl.sslot; rank = dl.rank;
                    } else {
                        load_direct(p, ls + j, cx, smem + pool1, m, cv, x, gslot, sslot, rank);
                    }
                    lane_hash(smem, o.msg + u1 * 4, cv, m);
                    lane_store(cv, x, gslot, sslot, rank, smem + pool1, 2 * G, cx);
                }
            }
            boundary(w, w1); /* l + 1 */
            ls = h1.x;
            w = w1;
            st1 = st1 == 2 ? 0 : st1 + 1;
            l++;
        }
    }
}

} /* namespace */

/* G chunk copies per CTA; batches of G copies from a work counter. */
__global__ void __launch_bounds__(PB_CTA_THREADS, 1) k_label_ws(const __grid_constant__ pb_depth_params_t p)
{
    extern __shared__ uint4 smem[];
    __shared__ uint32_t s_batch;
    const uint32_t G = p.units_per_cta;
    const Layout o(p.team_warps * 32, G);
    for (;;) {
        if (threadIdx.x == 0) s_batch = atomicAdd(p.queue, 1u);
        __syncthreads();
        const uint32_t batch = uniform(s_batch);
        if (batch >= p.nbatches) break;
        const uint32_t left = p.nunits - batch * G, cnt = left < G ? left : G;
        setup_units(p, smem, o, batch, cnt, blockIdx.x * G, threadIdx.x, blockDim.x);
        __syncthreads();
        depth_levels<false>(p, smem, o, cnt);
    }
}

/* k_label_ws with a thread-block cluster of C CTAs per chunk copy (G = 1),
 * for launches with fewer copies than SMs.  CTA rank 0 runs the copy exactly
 * as k_label_ws does.  A level wider than split_width is shared: rank 0
 * hashes its staged nodes and as many of the rest as bring it to ceil(w / C)
 * nodes; the other ranks hash the remainder, striding over it, with direct
 * loads, and read and write rank 0's shared-memory pool through distributed
 * shared memory.  Every boundary between levels l - 1 and l where l - 1 or l
 * is split is a cluster barrier instead of rank 0's CTA barrier; the other
 * ranks walk only the split levels (split_levels, nsplit of them, ascending)
 * and meet rank 0 at exactly those barriers, so every CTA of the cluster
 * passes the same barrier sequence.  One copy per cluster: the grid is
 * nunits * C CTAs, and copy k's global pool is at scratch + k *
 * unit_scratch_bytes.  No spin-waits: only CTA and cluster barriers. */
__global__ void __launch_bounds__(PB_CTA_THREADS, 1) k_label_wsc(const __grid_constant__ pb_depth_params_t p)
{
    extern __shared__ uint4 smem[];
    cg::cluster_group cl = cg::this_cluster();
    const pb_topo_view2_t &tp = p.topo;
    const uint32_t C = p.cluster;
    const uint32_t rank = cl.block_rank();
    const uint32_t unit = blockIdx.x / C;
    const Layout o(p.team_warps * 32, 1);
    setup_units(p, smem, o, unit, 1, unit, threadIdx.x, blockDim.x);
    __syncthreads();
    if (rank == 0) {
        depth_levels<true>(p, smem, o, 1);
        return;
    }
    /* rank 0's pool, through distributed shared memory */
    uint4 *pool = cl.map_shared_rank(smem, 0) + o.pool;
    const UnitCtx *cx = reinterpret_cast<const UnitCtx *>(smem + o.ctx);
    const uint32_t nthr = o.nthr, c = threadIdx.x;
    for (uint32_t k = 0; k < p.nsplit; k++) {
        const uint32_t l = __ldg(p.split_levels + k);
        if (k == 0 || __ldg(p.split_levels + k - 1) + 1 != l) cl.sync(); /* boundary l */
        const uint32_t ls = __ldg(tp.lstart + l), w = __ldg(tp.lstart + l + 1) - ls;
        const uint32_t per = (w + C - 1) / C, a = per > nthr ? per - nthr : 0;
        if (c < nthr)
            for (uint32_t j = nthr + a + (rank - 1) * nthr + c; j < w; j += (C - 1) * nthr) {
                uint32_t m[16], cv[8], x, gslot, sslot, rk;
                load_direct(p, ls + j, cx, pool, m, cv, x, gslot, sslot, rk);
                lane_hash(smem, o.msg, cv, m);
                lane_store(cv, x, gslot, sslot, rk, pool, 2, cx);
            }
        cl.sync(); /* boundary l + 1 */
    }
}

} /* namespace pb */

extern "C" uint32_t pb_ws_smem_bytes(uint32_t units_per_cta, uint32_t team_warps)
{
    const uint32_t nthr = 32u * team_warps, slots = nthr / units_per_cta;
    return (5u + 34u * units_per_cta + 2u * units_per_cta * (PB_CSM + 1u) + 6u * slots + 12u * nthr) * 16u;
}

/* Allow a depth kernel the largest dynamic shared memory a CTA can have (the
 * device's opt-in limit less the kernel's static shared memory) and report
 * it.  The attribute is per function, not per launch, so every caller sets
 * this one value. */
template <class K>
static int allow_smem(K *kernel, uint32_t *max_smem_bytes)
{
    int dev = 0, optin = 0;
    cudaFuncAttributes fa;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, kernel) != cudaSuccess)
        return -1;
    const int lim = optin - (int)fa.sharedSizeBytes;
    if (lim <= 0 ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess)
        return -1;
    if (max_smem_bytes) *max_smem_bytes = (uint32_t)lim;
    return 0;
}

extern "C" int pb_dev_label_ws_prepare(uint32_t *max_smem_bytes) { return allow_smem(pb::k_label_ws, max_smem_bytes); }

extern "C" int pb_dev_label_ws(const pb_depth_params_t *params, uint32_t grid, uint32_t smem_bytes,
                               cudaStream_t stream)
{
    if (params->units_per_cta < 1 || params->units_per_cta > PB_WS_MAX_UNITS ||
        (params->team_warps != 7 && params->team_warps != 15) ||
        params->topo.csm > PB_CSM || smem_bytes < pb_ws_smem_bytes(params->units_per_cta, params->team_warps))
        return -1;
    cudaGetLastError(); /* report only this launch */
    pb::k_label_ws<<<grid, 32u * (params->team_warps + 1), smem_bytes, stream>>>(*params);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

extern "C" int pb_dev_label_ws_occupancy(uint32_t cta_threads, uint32_t smem_bytes, int *blocks_per_sm)
{
    uint32_t lim = 0;
    if (pb_dev_label_ws_prepare(&lim) != 0 || smem_bytes > lim) return -1;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, pb::k_label_ws, (int)cta_threads,
                                                         smem_bytes) == cudaSuccess
               ? 0
               : -1;
}

static int wsc_allow(uint32_t C)
{
    if (allow_smem(pb::k_label_wsc, nullptr) != 0) return -1;
    return C > 8 && cudaFuncSetAttribute(pb::k_label_wsc, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                        cudaSuccess
               ? -1
               : 0;
}

extern "C" int pb_dev_label_wsc(const pb_depth_params_t *params, uint32_t smem_bytes, cudaStream_t stream)
{
    const uint32_t C = params->cluster;
    if (C < 2 || C > 16 || (params->team_warps != 7 && params->team_warps != 15) || params->nunits == 0 ||
        params->units_per_cta != 1 || params->topo.csm > PB_CSM ||
        smem_bytes < pb_ws_smem_bytes(1, params->team_warps) ||
        wsc_allow(C) != 0)
        return -1;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(params->nunits * C);
    cfg.blockDim = dim3(32 * (params->team_warps + 1));
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaGetLastError(); /* report only this launch */
    if (cudaLaunchKernelEx(&cfg, pb::k_label_wsc, *params) != cudaSuccess) return -1;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

/* How many clusters of C CTAs (team_warps hashing warps + 1, smem_bytes of
 * dynamic shared memory each) the device holds at once. */
extern "C" int pb_dev_label_wsc_max_clusters(uint32_t C, uint32_t team_warps, uint32_t smem_bytes, int *clusters)
{
    *clusters = 0;
    if (C < 2 || C > 16 || wsc_allow(C) != 0) return -1;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(C * 148);
    cfg.blockDim = dim3(32 * (team_warps + 1));
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(clusters, pb::k_label_wsc, &cfg) == cudaSuccess ? 0 : -1;
}
