"""Scratch caps on batches: the same bytes with fewer CTAs, each of which then
runs several batches one after the other."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
KEY = b"\x33" * 32


def copy_bytes(pkg, topo, kernel):
    s = pkg.Sched()
    s.kernel, s.units_per_team, s.max_teams, s.cluster_ctas = kernel, 1, 1, 1 if kernel == 3 else 0
    return topo.plan(1, s).scratch_cap_bytes


# few copies (the depth kernel's plan), many small ones under a cap that leaves
# room for the lockstep kernel's, and a ragged last batch
@pytest.mark.parametrize("cb,n,copies", [(2048, 16, 3), (300, 211, 40), (64, 4096, 2820)])
def test_one_topology_batch_under_a_cap(pkg, cuda, oracle, cb, n, copies):
    rbo = 7 * cb
    want = oracle.label_region(KEY, cb, n, rbo, threads=8).tobytes()
    buf = cuda.zeros(n * cb * 32, dtype=cuda.uint8, device="cuda")
    with pkg.Topology(cb) as topo:
        s = pkg.Sched()
        s.scratch_cap_bytes = copies * max(copy_bytes(pkg, topo, k) for k in (1, 3))
        reqs = [(topo, KEY, buf.data_ptr() + i * cb * 32, cb * 32, rbo + i * cb) for i in range(n)]
        with pkg.Batch(reqs, s) as batch:
            for _ in range(2):
                buf.zero_()
                rc, st = batch.run()
                assert rc == 0 and st["scratch_bytes"] <= s.scratch_cap_bytes
                assert buf.cpu().numpy().tobytes() == want
        blocks = [rbo + i * cb + (37 * i) % cb for i in range(min(n, 64))]
        rc, labels, st = topo.challenge_blocks(KEY, blocks, s)
        assert rc == 0 and st["scratch_bytes"] <= s.scratch_cap_bytes
        assert labels == b"".join(want[32 * (x - rbo):32 * (x - rbo) + 32] for x in blocks)


# two deep parts and the rest under one cap, on the depth and the lockstep kernel
@pytest.mark.parametrize("kernel", ["1", "0"])
@pytest.mark.parametrize("copies", [0, 20])
def test_deep_parts_under_a_cap(pkg, cuda, oracle, monkeypatch, kernel, copies):
    monkeypatch.setenv("POSE_B200_DEEP_KERNEL", kernel)
    sizes = [(4096, 5), (2048, 9), (256, 20)]
    topos = [pkg.Topology(cb) for cb, _ in sizes]
    bufs = [cuda.zeros(n * cb * 32, dtype=cuda.uint8, device="cuda") for cb, n in sizes]
    lock, depth = ([copy_bytes(pkg, t, k) for t in topos] for k in (1, 3))
    s = pkg.Sched()
    least = depth[0] + depth[1] + lock[2] if kernel == "1" else lock[0] + max(lock[1:])
    s.scratch_cap_bytes = least + copies * lock[1]
    with pkg.Batch([(t, KEY, b.data_ptr(), b.numel(), 4 * cb) for t, b, (cb, _) in zip(topos, bufs, sizes)],
                   s) as batch:
        rc, st = batch.run()
    assert rc == 0 and st["scratch_bytes"] <= s.scratch_cap_bytes
    for b, (cb, n) in zip(bufs, sizes):
        assert b.cpu().numpy().tobytes() == oracle.label_region(KEY, cb, n, 4 * cb, threads=8).tobytes()
    for t in topos:
        t.free()
