"""Which levels' ring stages (records and header, three of them) a hashing warp
of the depth kernels reads between two of its barriers (label_ws.cu).  Every
warp reads level 0 before a barrier that the producer passes before its first
level.

The producer fills the stage of level m while level m - 2 runs, and passes
every boundary; a warp that skips narrow levels passes only the boundaries at
levels of all hands.  Between its boundaries b1 and b2 the producer may be in
any level of [b1, b2 - 1]: the stage of level r is complete when r <= b1 + 1
and not yet refilled (by level r + 3) when r >= b2 - 1."""
from __future__ import annotations

import numpy as np
import pytest

from test_depth_levels import NARROW_ITEMS, level_widths
from test_topology import host  # noqa: F401  (the fixture)


def skipping_warp(w, hands, barrier_0):
    """(level read, last boundary passed, next boundary) of a warp that skips
    levels that are not of all hands; barrier_0: a barrier follows the read of
    level 0."""
    L = len(w)
    first = -1 if barrier_0 else 0
    walk, passed = [(0, first)], sorted({first, 0})  # (level read, last boundary passed)
    for l in np.nonzero(hands)[0].tolist():
        if passed[-1] != l:  # after levels that it skipped
            passed.append(l)
            walk.append((l, l))
        walk.append((l + 1, l))  # the next level's header and record, while level l runs
        passed.append(l + 1)
    after = dict(zip(passed, passed[1:]))
    return [(r, b, after.get(b, L + 1)) for r, b in walk]


def unsafe(reads):
    # the prologue (boundary -1) fills the stages of levels 0 and 1
    return [(r, b1, b2) for r, b1, b2 in reads if not b2 - 1 <= r <= max(b1, 0) + 1]


@pytest.mark.parametrize("cb", [2, 64, 300, 1024, 3000, 1 << 14])
def test_ring_reads(host, cb):  # noqa: F811
    w = level_widths(host, cb)
    seen = 0
    for G in range(1, 9):
        for sw in ((1 << 30,) if G > 1 else (1 << 30, 0, 10, 480)):
            hands = (w * G > NARROW_ITEMS) | (w > sw)
            assert not unsafe(skipping_warp(w, hands, barrier_0=True)), (cb, G, sw)
            # level 0 is the graph's one source node: without the barrier a warp
            # that reads its stage and skips it may find a later level there
            seen += bool(unsafe(skipping_warp(w, hands, barrier_0=False)))
    if (w * 8 > NARROW_ITEMS).any():
        assert seen
