"""The host side's plans on a CUDA runtime that does nothing (fake_cuda.c): what
is allocated and what is launched, with which sizes."""
from __future__ import annotations

import ctypes as C
import importlib.util
import os
import subprocess
import time

import pytest

from conftest import PKG_DIR, ROOT

CSRC = os.path.join(PKG_DIR, "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
LABEL, MULTI, DEPTH, CLUSTER = 1, 2, 3, 4


class Launch(C.Structure):
    _fields_ = [("kind", C.c_uint32), ("grid", C.c_uint32), ("warps", C.c_uint32), ("units_per", C.c_uint32),
                ("nunits", C.c_uint32), ("nbatches", C.c_uint32), ("smem", C.c_uint32), ("scratch", C.c_uint64)]


class Fake:
    """The package on the fake library."""

    def __init__(self, path):
        spec = importlib.util.spec_from_file_location("pose_b200_fake", os.path.join(PKG_DIR, "__init__.py"),
                                                      submodule_search_locations=[PKG_DIR])
        self.pkg = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(self.pkg)
        self.pkg.LIB_PATH = path
        self.lib = self.pkg.load()
        self.lib.fake_set_free.argtypes = [C.c_uint64]
        self.lib.fake_live.restype = C.c_uint64
        self.topos = {}

    def topo(self, cb, **kw):
        key = (cb, tuple(kw.items()))
        if key not in self.topos:
            self.topos[key] = self.pkg.Topology(cb, **kw)
        return self.topos[key]

    def launches(self):
        a = (Launch * 4096)()
        n = self.lib.fake_launches(a, 4096)
        return [a[i] for i in range(n)]

    def copy_bytes(self, topo):
        """Scratch of one chunk copy on the lockstep kernel and on the depth kernel."""
        out = []
        for kernel in (1, 3):
            s = self.pkg.Sched()
            s.kernel, s.units_per_team, s.max_teams = kernel, 1, 1
            s.cluster_ctas = 1 if kernel == 3 else 0
            out.append(topo.plan(1, s).scratch_cap_bytes)
        return out

    def sched(self, **kw):
        s = self.pkg.Sched()
        for k, v in kw.items():
            setattr(s, k, v)
        return s


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("fake") / "libpose_fake.so")
    src = [os.path.join(CSRC, f) for f in ("label_api.c", "label_batch.c", "label_server.c", "label_stream.c",
                                           "label_verify.c", "topology.c", "b3_host.c")]
    src.append(os.path.join(ROOT, "tests", "fake_cuda.c"))
    subprocess.run(["gcc", "-O2", "-std=c11", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-D_GNU_SOURCE", "-I" + CUDA_INC,
                    "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-o", so, *src, "-lpthread", "-lm", "-ldl"],
                   check=True)
    return Fake(so)


def requests(topo, n, chunks=1, first=0):
    sb = topo.super_bytes
    return [(topo, b"k" * 32, 1 << 40, chunks * sb, (first + i) * topo.chunk_blocks * chunks) for i in range(n)]


def test_planning_only_reads_the_topology(fake):
    topo = fake.topo(2048)
    fake.lib.fake_reset()
    topo.plan(16)
    topo.plan(16, fake.sched(kernel=3, team_warps=7))
    with fake.pkg.Batch(requests(topo, 16)):
        pass
    assert fake.lib.fake_occupancy_queries() == 0


# a cap on the scratch of a batch of one topology: plans on the depth kernel
# (few copies) and on the lockstep kernel (many), and the challenge call
@pytest.mark.parametrize("cb,n,kind,copies", [(2048, 16, DEPTH, 3), (2048, 700, None, 10), (64, 4096, MULTI, 2820)])
def test_one_topology_batch_keeps_its_cap(fake, cb, n, kind, copies):
    topo = fake.topo(cb)
    cap = copies * max(fake.copy_bytes(topo))
    fake.lib.fake_reset()
    before = fake.lib.fake_live()
    with fake.pkg.Batch(requests(topo, n), fake.sched(scratch_cap_bytes=cap)) as b:
        rc, st = b.run()
        assert rc == 0 and st["scratch_bytes"] <= cap
        ran = fake.launches()
        assert kind is None or [x.kind for x in ran] == [kind]
        assert 0 < sum(x.scratch for x in ran) <= cap
    assert fake.lib.fake_live() == before
    rc, _, st = topo.challenge_blocks(b"k" * 32, [i * cb for i in range(n)], fake.sched(scratch_cap_bytes=cap))
    assert rc == 0 and 0 < st["scratch_bytes"] <= cap


def test_one_topology_batch_fits_free_memory(fake):
    topo = fake.topo(2048)
    copy = fake.copy_bytes(topo)[1]
    fake.lib.fake_set_free(fake.lib.fake_live() + (2 << 30) + 5 * copy)
    try:
        with fake.pkg.Batch(requests(topo, 16)) as b:
            rc, st = b.run()
            assert rc == 0 and st["scratch_bytes"] <= 5 * copy
    finally:
        fake.lib.fake_set_free(170 << 30)


# a cap below the scratch of the teams that the requests would otherwise be
# packed into: smaller teams
@pytest.mark.parametrize("copies", [1, 5, 40])
def test_mixed_batch_packs_within_its_cap(fake, copies):
    a, b = fake.topo(300), fake.topo(512)  # equally deep: one launch
    cap = copies * max(fake.copy_bytes(t)[0] for t in (a, b))
    with fake.pkg.Batch(requests(a, 2000) + requests(b, 2000), fake.sched(scratch_cap_bytes=cap)) as batch:
        rc, st = batch.run()
    assert rc == 0 and 0 < st["scratch_bytes"] <= cap


def wait_all(fake, server, tickets, seconds=20):
    """All tickets done; a server that holds some back for good is left alone
    (closing it would wait for them too)."""
    end = time.time() + seconds
    while time.time() < end and any(server.query(t) == 0 for t in tickets):
        time.sleep(0.01)
    left = [t for t in tickets if server.query(t) != 1]
    if left:
        server.handle = None
    return left


@pytest.mark.parametrize("copies", [1, 6])
def test_server_packs_within_its_arena(fake, copies):
    topo = fake.topo(512)
    arena = max(256, copies * fake.copy_bytes(topo)[0])
    server = fake.pkg.Server(scratch_bytes=arena)
    sid = server.session(b"k" * 32)
    # the first request holds the arena until the others are all pending
    fake.lib.fake_hold_events()
    tickets = [server.submit(topo, sid, 1 << 40, 4 * topo.super_bytes, 0)]
    while server.stats()["waves"] == 0:
        time.sleep(0.01)
    tickets += [server.submit(topo, sid, 1 << 40, 4 * topo.super_bytes, 0) for _ in range(600)]
    fake.lib.fake_finish_events()
    assert not wait_all(fake, server, tickets)
    server.close()


# more copies of the second deep part than the makespan search once took: the
# first part then ran one copy a CTA, eight times one after the other
def test_second_deep_part_of_any_size(fake):
    deep, second = fake.topo(4096), fake.topo(2048)
    fake.lib.fake_reset()
    with fake.pkg.Batch(requests(deep, 1, 600) + requests(second, 1, 12000)):
        pass
    first = fake.launches()[0]
    assert first.kind == DEPTH and first.nunits == 1200 and first.units_per > 1


# the deep parts, the second one's CTAs too, and the rest share the cap, down
# to one copy of each
@pytest.mark.parametrize("kernel", ["1", "0"])
@pytest.mark.parametrize("part", [2.0, 0.6, 0.3, 0.05, 0.02, 0])
def test_deep_parts_keep_the_cap(fake, monkeypatch, part, kernel):
    monkeypatch.setenv("POSE_B200_DEEP_KERNEL", kernel)
    deep, second, small = fake.topo(4096), fake.topo(2048), fake.topo(256)
    reqs = requests(deep, 40, 2) + requests(second, 60, 4) + requests(small, 20, 4)
    d, s, r = (fake.copy_bytes(t) for t in (deep, second, small))
    least = d[1] + s[1] + r[0] if kernel == "1" else d[0] + max(s[0], r[0])
    cap = max(least, int(part * (160 * d[1] + 480 * s[1])))
    fake.lib.fake_reset()
    with fake.pkg.Batch(reqs, fake.sched(scratch_cap_bytes=cap)) as batch:
        rc, st = batch.run()
    ran = fake.launches()
    assert rc == 0 and st["scratch_bytes"] == sum(x.scratch for x in ran) <= cap
    if kernel == "1":  # both deep parts on the depth kernel whenever both fit it
        assert [x.kind for x in ran] == [DEPTH, DEPTH, MULTI]


# a deep request that fits the free SMs at the most copies a CTA takes runs in
# one round of CTAs, whatever the load asks for; chunks of two copies each
@pytest.mark.parametrize("sizes", [(50, 50), (60, 20), (30, 10, 50), (64, 1)])
def test_served_depth_group_runs_in_one_round(fake, monkeypatch, sizes):
    monkeypatch.setenv("POSE_B200_SERVER_DEEP_LEVELS", "1")
    topo = fake.topo(512)
    fake.lib.fake_reset()
    fake.lib.fake_hold_events()
    server = fake.pkg.Server(scratch_bytes=1 << 28)
    sid, free, tickets = server.session(b"k" * 32), 148 - 148 // 8, []
    for chunks in sizes:
        assert 2 * chunks <= 4 * free
        tickets.append(server.submit(topo, sid, 1 << 40, chunks * topo.super_bytes, 0))
        end = time.time() + 20
        while len(fake.launches()) < len(tickets) and time.time() < end:
            time.sleep(0.01)
        ran = fake.launches()[-1]
        free -= ran.grid
        assert ran.kind == DEPTH and ran.nunits == 2 * chunks and free >= 0
        if ran.nbatches > ran.grid:
            fake.lib.fake_finish_events()
        assert ran.nbatches <= ran.grid, (ran.grid, ran.units_per, ran.nbatches)
    fake.lib.fake_finish_events()
    assert not wait_all(fake, server, tickets)
    server.close()


def test_served_depth_group_fits_the_arena(fake, monkeypatch):
    monkeypatch.setenv("POSE_B200_SERVER_DEEP_LEVELS", "1")
    topo = fake.topo(512)
    server = fake.pkg.Server(scratch_bytes=fake.copy_bytes(topo)[0])  # one copy on the lockstep kernel
    sid = server.session(b"k" * 32)
    assert not wait_all(fake, server, [server.submit(topo, sid, 1 << 40, 200 * topo.super_bytes, 0)])
    server.close()


# a graph's nodes keep the priority of the stream they were captured from only
# when it is instantiated so
def test_no_priority_that_the_graph_ignores(fake):
    fake.lib.fake_reset()
    with fake.pkg.Batch(requests(fake.topo(4096), 8) + requests(fake.topo(2048), 8) + requests(fake.topo(256), 8)):
        pass
    assert len(fake.launches()) == 3
    assert fake.lib.fake_priority_streams() == 0 or fake.lib.fake_node_priorities()


# k_label_multi's occupancy query also raises its shared memory limit: where it
# fails, launches keep to the default one (48 KB a CTA, 96 bytes a thread)
@pytest.mark.parametrize("mix", [(300, 256), (4096, 2048, 256), (512,)])
def test_default_shared_memory_limit(fake, mix):
    topos = [fake.topo(cb) for cb in mix]
    reqs = [r for t in topos for r in requests(t, 400)]
    fake.lib.fake_fail_multi_occupancy(1)
    try:
        fake.lib.fake_reset()
        with fake.pkg.Batch(reqs) as b:
            assert b.run()[0] == 0
        server = fake.pkg.Server(scratch_bytes=1 << 30)
        sid = server.session(b"k" * 32)
        assert not wait_all(fake, server, [server.submit(t, sid, 1 << 40, t.super_bytes, 0) for t in topos])
        server.close()
        ran = [x for x in fake.launches() if x.kind == MULTI]
        assert ran and all(x.warps <= 8 and x.smem <= 48 * 1024 - 1024 for x in ran)
    finally:
        fake.lib.fake_fail_multi_occupancy(0)


# windows labelled together: eight chunk copies an SM, of one or two copies a chunk
@pytest.mark.parametrize("cb,copies", [(1, 1), (64, 2)])
def test_stream_groups(fake, cb, copies):
    topo, window, n = fake.topo(cb), 16, 4096
    got = []
    fake.lib.fake_reset()
    rc, st = topo.label_stream(b"k" * 32, n * topo.super_bytes, lambda v, off: got.append((len(v), off)),
                               window_bytes=window * topo.super_bytes)
    wb = window * topo.super_bytes
    assert rc == 0 and got == [(wb, i * wb) for i in range(n // window)]
    per = -(-8 * 148 // (window * copies))  # windows a call
    assert [x.nunits for x in fake.launches()][0] == per * window * copies
    # a caller's schedule is for its own window
    fake.lib.fake_reset()
    rc, _ = topo.label_stream(b"k" * 32, 64 * topo.super_bytes, lambda v, off: 0, window_bytes=wb,
                              sched=fake.sched(kernel=1))
    assert rc == 0 and [x.nunits for x in fake.launches()] == [window * copies] * 4
