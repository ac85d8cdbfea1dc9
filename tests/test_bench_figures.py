"""The figures that bench.py derives from its measurements."""
from __future__ import annotations

import importlib.util
import os

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_traffic_of_the_kernel_that_ran(bench):
    lines = {}
    for fn in os.listdir(os.path.join(ROOT, "profiles")):
        for ln in open(os.path.join(ROOT, "profiles", fn)):
            f = ln.split()
            if len(f) == 4 and f[0] == "bench-traffic:":
                lines[f[1], f[2]] = float(f[3])
    # the headline runs the depth kernel, with or without clusters
    assert any(w == "plain_2e17" for w, _ in lines)
    for kernel, cluster, name in ((1, 0, "k_label"), (3, 1, "k_label_ws"), (3, 2, "k_label_wsc")):
        assert bench.profiled_traffic("plain_2e17", kernel, cluster) == lines.get(("plain_2e17", name))


def test_depth_bound_is_the_shortest_chain(bench):
    # narrow levels are hashed by four lanes a node where there is a block-0 table
    assert bench.chain_cycles(2, 995.5) == bench.FOUR_LANE_CYCLES < 964
    assert bench.chain_cycles(2, 700.0) == 700.0
    assert bench.chain_cycles(3, 995.5) == 995.5


def test_reference_arm_without_its_build(bench, monkeypatch, capsys):
    import types

    def missing(*_):
        raise FileNotFoundError("/somewhere/libposeref.so")
    monkeypatch.setattr(bench, "cpu_reference", missing)
    monkeypatch.delenv("RANK", raising=False)
    bench.run_reference_arm(types.SimpleNamespace(workload="plain_small", steps=1, warmup=0, gpus=1, no_aux=True))
    line = bench.json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libposeref.so" in line["unavailable"]
