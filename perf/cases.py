"""The calls that a program makes of this labeler, for timing them.

A case is one call pattern through the public entry points: labeling a device
window with a resident topology, the one-call form that builds its topology,
a captured batch of many sessions, a burst of requests to the server,
challenge answers, and labeling into host memory through the streaming sink.
All inputs of the path are keys and positions; they are drawn from the seed.
A program builds one topology per chunk size and keeps it, so topologies are
kept here across states, as are the batch and server handles of a state.
"""
from __future__ import annotations

import importlib
import os
import random

import numpy as np
import torch

os.environ.setdefault("POSE_GPU_QUIET", "1")  # as disk workers run it: no line per call
# a host that serves many requests raises the work queues before CUDA starts
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

pose = importlib.import_module("pose-memory-wiping_b200")
workloads = importlib.import_module("pose-memory-wiping_b200.workloads")

_topologies: dict = {}


def listed():
    return [
        # one small chunk: a spot relabel, where launches and the short chain count
        {"name": "label_256_x1", "kind": "label", "cb": 256, "chunks": 1, "tail": 0, "seed_len": 32},
        # the small configured region: one session, 64 chunks of 2^10 blocks
        {"name": "label_2e10_x64", "kind": "label", "cb": 1 << 10, "chunks": 64, "tail": 0, "seed_len": 32},
        # a chunk size that is no power of two, a buffer with a tail, a longer session seed
        {"name": "label_3000_x37", "kind": "label", "cb": 3000, "chunks": 37, "tail": 4777, "seed_len": 77},
        # a 256 MiB window at the default chunk size: many shallow chunks
        {"name": "label_4096_x2048", "kind": "label", "cb": 4096, "chunks": 2048, "tail": 0, "seed_len": 32},
        # a 1 GiB window of large chunks, as a disk worker labels one after another
        {"name": "label_2e16_x512", "kind": "label", "cb": 1 << 16, "chunks": 512, "tail": 0, "seed_len": 32},
        # the configured headline region: 32 chunks of 2^17 blocks
        {"name": "label_2e17_x32", "kind": "label", "cb": 1 << 17, "chunks": 32, "tail": 0, "seed_len": 32},
        # few chunks of the largest served size: the deepest graph
        {"name": "label_2e18_x4", "kind": "label", "cb": 1 << 18, "chunks": 4, "tail": 0, "seed_len": 32},
        # the one-call entry point: build the topology, label 64 default chunks, free it
        {"name": "oneshot_4096_x64", "kind": "oneshot", "cb": 4096, "chunks": 64, "seed_len": 32},
        # the configured batch: 256 sessions of 2^12 to 2^17 blocks, 1 to 8 chunks each
        {"name": "batch_256", "kind": "batch", "sessions": 256, "low": 12, "high": 17, "most": 8, "mix": 3},
        # a burst of served requests, shallow and deep together
        {"name": "served_48", "kind": "served", "requests": 48, "low": 10, "high": 17, "most": 8, "mix": 5},
        # a verifier's challenges on one region of default chunks
        {"name": "challenge_4096_x64", "kind": "challenge", "cb": 4096, "blocks": 64, "span": 1 << 16},
        # labels delivered to host memory window by window
        {"name": "stream_4096_x2048", "kind": "stream", "cb": 4096, "chunks": 2048, "window": 32 << 20},
    ]


def _log_uniform(rng, low, high):
    return max(low, min(high, int(round(low * (high / low) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["label", "label", "label", "label", "batch", "served", "challenge", "stream", "oneshot"])
    if kind == "batch":
        return {"kind": kind, "sessions": _log_uniform(rng, 12, 200), "low": rng.randint(10, 12),
                "high": rng.randint(13, 16), "most": rng.randint(1, 8), "mix": rng.randrange(1 << 30)}
    if kind == "served":
        return {"kind": kind, "requests": rng.randint(6, 48), "low": 10, "high": rng.randint(12, 16),
                "most": rng.randint(1, 8), "mix": rng.randrange(1 << 30)}
    if kind == "challenge":
        return {"kind": kind, "cb": _log_uniform(rng, 500, 16384), "blocks": _log_uniform(rng, 1, 200),
                "span": 1 << rng.randint(12, 18)}
    if kind == "oneshot":
        return {"kind": kind, "cb": _log_uniform(rng, 300, 8192), "chunks": _log_uniform(rng, 1, 128),
                "seed_len": 32}
    if kind == "stream":
        cb = _log_uniform(rng, 1000, 8192)
        return {"kind": kind, "cb": cb, "chunks": _log_uniform(rng, 32, (8 << 20) // cb),
                "window": rng.choice([8, 32, 64]) << 20}
    # label: chunk sizes over the whole range, odd ones among them, up to 2 G nodes
    cb = _log_uniform(rng, 128, 1 << 17)
    if rng.random() < 0.5:
        cb = 1 << (cb.bit_length() - 1)
    most = max(1, min(4096, (2 << 30) // workloads.chunk_nodes(cb)))
    return {"kind": "label", "cb": cb, "chunks": _log_uniform(rng, 1, most),
            "tail": rng.choice([0, 0, rng.randrange(cb * 32)]), "seed_len": rng.choice([32, 32, rng.randint(1, 200)])}


def _topology(cb):
    if cb not in _topologies:
        _topologies[cb] = pose.Topology(cb)
    return _topologies[cb]


def _requests(case, seed):
    """Sizes from the case, keys and positions from the seed."""
    sizes, rng = random.Random(case["mix"]), random.Random(seed)
    n = case["sessions"] if case["kind"] == "batch" else case["requests"]
    out = []
    for _ in range(n):
        cb, chunks = 1 << sizes.randint(case["low"], case["high"]), sizes.randint(1, case["most"])
        out.append((cb, chunks, rng.randbytes(32), rng.randrange(1 << 20) * cb))
    return out


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("label", "oneshot"):
        nbytes = case["chunks"] * case["cb"] * 32 + case.get("tail", 0)
        state.update(cb=case["cb"], key=rng.randbytes(case["seed_len"]), nbytes=nbytes,
                     rbo=rng.randrange(1 << 20) * case["cb"], out=torch.zeros(nbytes, dtype=torch.uint8, device="cuda"))
        if kind == "label":
            state["topo"] = _topology(case["cb"])
    elif kind in ("batch", "served"):
        reqs = _requests(case, seed)
        out = torch.zeros(sum(cb * chunks for cb, chunks, _, _ in reqs) * 32, dtype=torch.uint8, device="cuda")
        calls, at = [], out.data_ptr()
        for cb, chunks, key, rbo in reqs:
            nbytes = cb * chunks * 32
            calls.append((_topology(cb), key, at, nbytes, rbo))
            at += nbytes
        torch.cuda.synchronize()
        state["out"] = out
        if kind == "batch":
            state["batch"] = pose.Batch(calls)
        else:
            server = pose.Server(scratch_bytes=8 << 30)
            for topo in {id(c[0]): c[0] for c in calls}.values():
                server.prepare(topo)
            state["server"] = server
            state["calls"] = [(topo, server.session(key), ptr, nbytes, rbo) for topo, key, ptr, nbytes, rbo in calls]
    elif kind == "challenge":
        state.update(topo=_topology(case["cb"]), key=rng.randbytes(32),
                     blocks=[rng.randrange(case["span"]) for _ in range(case["blocks"])])
    else:
        nbytes = case["chunks"] * case["cb"] * 32
        out = np.zeros(nbytes, np.uint8)

        def sink(view, off):
            out[off:off + len(view)] = np.frombuffer(view, np.uint8)
            return 0

        state.update(topo=_topology(case["cb"]), key=rng.randbytes(32), rbo=rng.randrange(1 << 20) * case["cb"],
                     nbytes=nbytes, out=out, sink=sink, window=case["window"])
    torch.cuda.synchronize()
    return state


def _check(rc):
    if rc != 0:
        raise RuntimeError(pose.last_error())


def run(state):
    kind = state["kind"]
    if kind == "label":
        _check(state["topo"].label(state["key"], state["out"].data_ptr(), state["nbytes"], state["rbo"]))
    elif kind == "oneshot":
        _check(pose.label_hbm(state["key"], state["cb"], state["out"].data_ptr(), state["nbytes"], state["rbo"]))
    elif kind == "batch":
        _check(state["batch"].run()[0])
    elif kind == "served":
        server = state["server"]
        tickets = [server.submit(*call) for call in state["calls"]]
        for t in tickets:
            _check(server.wait(t)[0])
    elif kind == "challenge":
        rc, labels, _ = state["topo"].challenge_blocks(state["key"], state["blocks"])
        _check(rc)
        return np.frombuffer(labels, np.uint8)
    else:
        rc, _ = state["topo"].label_stream(state["key"], state["nbytes"], state["sink"], state["rbo"],
                                           window_bytes=state["window"])
        _check(rc)
    return state["out"]


def work(case):
    """Bytes of the labels that come out, and the 32-bit integer operations of
    the two seed-dependent compressions of every node (680 each; block 0 of a
    node depends on its index alone)."""
    kind = case["kind"]
    if kind in ("batch", "served"):
        parts = [(cb, chunks) for cb, chunks, _, _ in _requests(case, 0)]
    elif kind == "challenge":
        rng = random.Random(0)
        rng.randbytes(32)
        touched = {rng.randrange(case["span"]) // case["cb"] for _ in range(case["blocks"])}
        return {"bytes": 32 * case["blocks"], "flops": len(touched) * workloads.chunk_nodes(case["cb"]) * 1360}
    else:
        parts = [(case["cb"], case["chunks"])]
    return {"bytes": sum(cb * n * 32 for cb, n in parts),
            "flops": sum(workloads.chunk_nodes(cb) * n * 1360 for cb, n in parts)}
