"""Where the pipelined records say the depth kernel finds a node's predecessors
as their level begins (topology.h, words 6 and 7)."""
from __future__ import annotations

import numpy as np
import pytest

from test_topology import NO_SLOT, PREV, SMEM, copy_edges, host, pipelined  # noqa: F401  (host: the fixture)

STAGED, GLOBAL, SLOT_MASK = 1 << 31, 1 << 30, 0xFFFF
POOL = 480  # the slots of the pool that the kernels run on; the entry after them is zero


@pytest.mark.parametrize("cb", [1, 2, 3, 100, 1024, 3000, 16384])
@pytest.mark.parametrize("csm", [4, POOL - 1, POOL, POOL + 1, 2048])
def test_places(host, cb, csm):  # noqa: F811
    info, lstart, _, recs = pipelined(host, cb, csm)
    np_, p0, p1, _ = copy_edges(host, cb)
    none = max(csm, POOL)
    ids = (recs[:, 0] & 0x0FFFFFFF).astype(np.int64)
    level, slot = np.zeros(info["S"], np.int64), np.zeros(info["S"], np.int64)
    level[ids] = np.repeat(np.arange(info["L"]), np.diff(lstart.astype(np.int64)))
    slot[ids] = recs[:, 4]
    assert (slot[slot != NO_SLOT] < min(csm, none)).all()
    for e, pred in ((0, p0), (1, p1)):
        q = pred[ids].astype(np.int64)
        has = np_[ids] > e
        late = has & (level[q] + 1 == level[ids])
        place, ref = recs[:, 6 + e].astype(np.int64), recs[:, 1 + e].astype(np.int64)
        assert (place[~has] == none).all()
        assert (place[has & ~late] == STAGED).all()
        pooled = late & (slot[q] != NO_SLOT)
        assert (place[pooled] == slot[q][pooled]).all()
        assert (ref[pooled] == (PREV | SMEM | slot[q][pooled])).all()
        assert (place[late & ~pooled] == (GLOBAL | none)).all()
