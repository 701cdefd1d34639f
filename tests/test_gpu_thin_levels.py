"""Top-down levels by frontier size: thin levels (touched list, queues built
by the inspect step) and the others (bitmap walk, queue build), which meet in
one traversal when the frontier grows past the thin limit (2^20 edges) and
shrinks below it again."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

MODES = [ib.MODE_PERSISTENT, ib.MODE_DEVICE_LOOP]
_CACHE = {}


def graph(kind):
    if kind not in _CACHE:
        if kind == "rmat16":  # 1.8 M edges: whole-graph frontiers are above the limit
            beg, col = ib.gen_rmat(16, 16, seed=3)
        else:  # grid: every level is thin, frontiers of up to ~20 k vertices
            beg, col = ib.gen_grid(403, 509, 0.05, 0.0, seed=6)
        _CACHE[kind] = (beg, col, ib.Graph.from_csr(beg, col))
    return _CACHE[kind]


@pytest.mark.parametrize("width", [32, 64, 128, 256])
@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("switch_level", [1000, 3, -1])
def test_thin_and_wide_levels(width, mode, switch_level):
    beg, col, g = graph("rmat16")
    src = ib.sample_sources(beg, col, width + 3, seed=width)
    res = g.run(src, width=width, mode=mode, switch_level=switch_level, levels_cap=64)
    ref, _ = oracle.bfs_auto(beg, col, src)
    assert np.array_equal(res.depth, ref)
    assert res.stats["traversed_edges"] == oracle.teps(beg, ref)
    edges = [r["frontier_edges"] for r in res.levels if r["dir"] in (-1, 0)]
    if switch_level == 1000:
        assert max(edges) > 1 << 20 > min(edges)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("groups,n", [(1, 128), (2, 250)])
def test_many_thin_levels(mode, groups, n):
    beg, col, g = graph("grid")
    src = ib.sample_sources(beg, col, n, seed=n)
    res = g.run(src, width=128, mode=mode, groups=groups, switch_level=10000)
    ref, _ = oracle.bfs_auto(beg, col, src)
    assert res.depth.dtype == ref.dtype and np.array_equal(res.depth, ref)
    assert res.stats["traversed_edges"] == oracle.teps(beg, ref)
