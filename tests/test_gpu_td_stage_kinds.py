"""Staged chunks (td_stage) on top-down levels above the touched-list limit:
marked in the bitmap, and found by the sweep.  Every vertex goes through the
chunk queue."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

_CACHE = {}


def graph(kind):
    if kind not in _CACHE:
        rng = np.random.default_rng(5)
        V, m = (3_100_003, 4_000_000) if kind == "bitmap" else (300_007, 1_500_000)
        u, v = rng.integers(0, V, (2, m)).astype(np.int32)
        if kind == "wide":
            # and a hub whose list has whole chunks, a partial one and an odd start
            hub = rng.choice(V, 7001, replace=False).astype(np.int32)
            u = np.concatenate([u, np.full(7001, 5, np.int32)])
            v = np.concatenate([v, hub])
        beg, col = ib.csr_from_edges(u, v, V)
        _CACHE[kind] = (beg, col, ib.Graph.from_csr(beg, col))
    return _CACHE[kind]


@pytest.mark.parametrize("kind,width,n", [("bitmap", 32, 6), ("wide", 64, 70), ("wide", 128, 128),
                                          ("wide", 256, 200)])
@pytest.mark.parametrize("mode", [ib.MODE_PLAIN, ib.MODE_DEVICE_LOOP])
@pytest.mark.parametrize("lrg_shed", [0, 512])
def test_staged_levels(kind, width, n, mode, lrg_shed):
    beg, col, g = graph(kind)
    V = len(beg) - 1
    src = ib.sample_sources(beg, col, n, seed=n)
    res = g.run(src, width=width, mode=mode, switch_level=1000, td_stage=1, sml_shed=1,
                lrg_shed=lrg_shed, levels_cap=256)
    ref, _ = oracle.bfs_auto(beg, col, src)
    assert np.array_equal(res.depth, ref)
    assert res.stats["traversed_edges"] == oracle.teps(beg, ref)
    mf = [r["frontier_edges"] for r in res.levels if r["dir"] in (-1, 0)]
    if kind == "wide":
        assert any(x * 2 >= V and x > 1 << 20 for x in mf)
    else:
        assert any(1 << 20 < x < V // 2 for x in mf)
