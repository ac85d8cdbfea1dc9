"""The depth kernels' per-level choices (label_ws.cu): which barrier ends a
level, and which of the two ways hashes it."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_topology import HostTopo, host  # noqa: F401  (the fixture)

NARROW_ITEMS = 64


def level_widths(lib, cb):
    t = HostTopo()
    assert lib.pb_topo_host_build(cb, C.byref(t)) == 0
    try:
        return np.diff(np.ctypeslib.as_array(t.lstart, shape=(t.L + 1,)).astype(np.int64))
    finally:
        lib.pb_topo_host_free(C.byref(t))


def full_barriers(w, warps, G, split_width):
    """The boundaries (b: between levels b - 1 and b) that end in a barrier of
    all hashing warps, restated for the narrow group and the producer, which
    walk every level, and for the other warps, which skip from one level of
    all hands to the next."""
    narrow = min(32 * warps // 4, NARROW_ITEMS)
    hands = (w * G > narrow) | (w > split_width)
    L = len(w)
    walk = [b for b in range(1, L + 1) if hands[b - 1] or (b < L and hands[b])]
    skip, l = [], 0
    while l < L:
        if not hands[l]:
            nxt = np.nonzero(hands[l:])[0]
            if len(nxt) == 0:
                break
            l += int(nxt[0])
            skip.append(l)
        skip.append(l + 1)
        l += 1
    return walk, skip


@pytest.mark.parametrize("cb", [2, 64, 300, 1024, 3000, 1 << 14])
def test_all_warps_pass_the_same_barriers(host, cb):  # noqa: F811
    w = level_widths(host, cb)
    for warps in (7, 15):
        for G in (1, 2, 3, 4):
            for sw in ((1 << 30,) if G > 1 else (1 << 30, 0, 10, 480)):
                walk, skip = full_barriers(w, warps, G, sw)
                assert walk == skip, (cb, warps, G, sw)


# level widths on both sides of 8 (one warp of quads), 64 (the narrow group),
# 120 or 56 (all quads) and 480 or 224 (one pass of lanes); one copy per chunk
# (chunk_blocks 1), ragged right copies
@pytest.mark.gpu
@pytest.mark.parametrize("cb,nsup", [(1, 5), (2, 3), (7, 2), (64, 3), (300, 2), (513, 3), (1500, 2), (2048, 2),
                                     (5000, 1)])
def test_depth_kernel_levels(pkg, cuda, oracle, cb, nsup):
    key, rbo = bytes(range(40)), 5 * cb
    want = oracle.label_region(key, cb, nsup, rbo, threads=8).tobytes()
    buf = cuda.zeros(nsup * cb * 32, dtype=cuda.uint8, device="cuda")
    with pkg.Topology(cb) as topo:
        for warps in (7, 15):
            for cluster in (1, 2):
                s = pkg.Sched()
                s.kernel, s.team_warps, s.cluster_ctas = 3, warps, cluster
                if cluster > 1 and (warps != 15 or topo.plan(nsup, s) is None):
                    continue  # the cluster form has 15 hashing warps and needs a level to share
                buf.zero_()
                rc, st = topo.label(key, buf.data_ptr(), buf.numel(), rbo, sched=s, stats=True)
                assert rc == 0, pkg.last_error()
                assert (st["kernel"], st["team_warps"], st["cluster_ctas"]) == (3, warps, cluster)
                assert buf.cpu().numpy().tobytes() == want, (cb, warps, cluster)


# units a team or CTA that are no power of two, the last batch ragged
@pytest.mark.gpu
@pytest.mark.parametrize("kernel,warps,nsup", [(1, 16, 1100), (1, 4, 1100), (1, 8, 3000), (3, 0, 500), (3, 0, 210),
                                               (3, 0, 700)])
def test_uneven_units(pkg, cuda, oracle, kernel, warps, nsup):
    key, cb, rbo = b"\x11" * 32, 33, 33 * 9
    want = oracle.label_region(key, cb, nsup, rbo, threads=8).tobytes()
    buf = cuda.zeros(nsup * cb * 32, dtype=cuda.uint8, device="cuda")
    with pkg.Topology(cb) as topo:
        s = pkg.Sched()
        s.kernel, s.team_warps = kernel, warps
        rc, st = topo.label(key, buf.data_ptr(), buf.numel(), rbo, sched=s, stats=True)
        assert rc == 0, pkg.last_error()
        assert st["kernel"] == kernel and st["units_per_team"] > 1
        assert buf.cpu().numpy().tobytes() == want, st
        assert topo.residue() == 0


# a multi-topology launch: all topologies with the block-0 table, some, none
@pytest.mark.gpu
@pytest.mark.parametrize("tables", [(True, True), (True, False), (False, False)])
def test_tables_in_one_launch(pkg, cuda, oracle, tables):
    sizes = [(33, 70), (300, 5)]
    topos = [pkg.Topology(cb, cv0_table=t) for (cb, _), t in zip(sizes, tables)]
    bufs = [cuda.zeros(n * cb * 32, dtype=cuda.uint8, device="cuda") for cb, n in sizes]
    with pkg.Batch([(t, b"\x22" * 32, b.data_ptr(), b.numel(), 3 * cb)
                    for t, b, (cb, _) in zip(topos, bufs, sizes)]) as batch:
        rc, st = batch.run()
    assert rc == 0, pkg.last_error()
    assert st["used_cv0_table"] == all(tables)
    for b, (cb, n) in zip(bufs, sizes):
        assert b.cpu().numpy().tobytes() == oracle.label_region(b"\x22" * 32, cb, n, 3 * cb, threads=8).tobytes()
    for t in topos:
        assert t.residue() == 0
        t.free()
