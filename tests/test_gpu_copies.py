"""Copies per CTA of the depth kernel in batches and on the server, and the plan
that a topology keeps between calls."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
KEY = b"\x44" * 32


@pytest.mark.parametrize("units", [5, 6, 7, 8])
def test_batch_copies_per_cta(pkg, cuda, oracle, monkeypatch, units):
    monkeypatch.setenv("POSE_B200_DEEP_UNITS", str(units))
    monkeypatch.setenv("POSE_B200_DEEP2_UNITS", str(13 - units))
    sizes = [(4096, 7), (2048, 11), (256, 9)]  # ragged last batches
    topos = [pkg.Topology(cb) for cb, _ in sizes]
    bufs = [cuda.zeros(n * cb * 32, dtype=cuda.uint8, device="cuda") for cb, n in sizes]
    with pkg.Batch([(t, KEY, b.data_ptr(), b.numel(), 6 * cb) for t, b, (cb, _) in zip(topos, bufs, sizes)]) as batch:
        rc, st = batch.run()
    assert rc == 0 and st["kernel_launches"] == 6
    for b, (cb, n) in zip(bufs, sizes):
        assert b.cpu().numpy().tobytes() == oracle.label_region(KEY, cb, n, 6 * cb, threads=8).tobytes()
    for t in topos:
        t.free()


# by the load, and fixed; on few SMs the CTAs loop over their batches
@pytest.mark.parametrize("units", ["0", "1", "3", "4", "8"])
@pytest.mark.parametrize("sms", ["0", "4"])
def test_server_copies_per_cta(pkg, cuda, oracle, monkeypatch, units, sms):
    monkeypatch.setenv("POSE_B200_SERVER_DEEP_LEVELS", "5000")
    monkeypatch.setenv("POSE_B200_SERVER_DEEP_UNITS", units)
    monkeypatch.setenv("POSE_B200_SERVER_DEEP_SMS", sms)
    sizes = [(2048, 5), (4096, 1), (256, 6), (2048, 8), (4096, 3)]
    topos = {cb: pkg.Topology(cb) for cb in (256, 2048, 4096)}
    bufs = [cuda.zeros(n * cb * 32, dtype=cuda.uint8, device="cuda") for cb, n in sizes]
    cuda.cuda.synchronize()
    assert topos[2048].info()["levels"] >= 5000 > topos[256].info()["levels"]
    with pkg.Server(scratch_bytes=1 << 28) as srv:
        sid = srv.session(KEY)
        tickets = [srv.submit(topos[cb], sid, b.data_ptr(), b.numel(), (9 + i) * cb)
                   for i, ((cb, _), b) in enumerate(zip(sizes, bufs))]
        assert all(srv.wait(t)[0] == 0 for t in tickets)
    for i, ((cb, n), b) in enumerate(zip(sizes, bufs)):
        assert b.cpu().numpy().tobytes() == oracle.label_region(KEY, cb, n, (9 + i) * cb, threads=8).tobytes()
    for t in topos.values():
        t.free()


def test_kept_plan_across_sizes_caps_and_workspaces(pkg, cuda, oracle):
    cb, sizes = 512, [3, 90, 3, 700, 90, 1]
    want = oracle.label_region(KEY, cb, max(sizes), 0, threads=8).tobytes()
    buf = cuda.zeros(max(sizes) * cb * 32, dtype=cuda.uint8, device="cuda")
    with pkg.Topology(cb) as topo:
        for n in sizes:
            for cap in (0, 1 << 17, 0):  # automatic, under a cap, automatic again
                s = pkg.Sched()
                s.scratch_cap_bytes = cap
                buf.zero_()
                rc, st = topo.label(KEY, buf.data_ptr(), n * cb * 32, 0, sched=s if cap else None, stats=True)
                assert rc == 0 and st["units"] == 2 * n and (not cap or st["scratch_bytes"] <= cap)
                assert buf.cpu().numpy()[:n * cb * 32].tobytes() == want[:n * cb * 32]
                assert not buf[n * cb * 32:].any().item()
                assert topo.residue() == 0
