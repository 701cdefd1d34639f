"""Top-down levels whose frontier has more than 2^20 edges: marked in the
bitmap below one edge per two reachable vertices, found by a sweep (wide)
above it.  A sparse random graph has both, and thin levels, on its way out and
back."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

_CACHE = {}


def graph(kind):
    if kind not in _CACHE:
        rng = np.random.default_rng(5)
        if kind == "sparse":  # 3.1 M vertices, degree ~2.6: levels grow 2x
            V, m = 3_100_003, 4_000_000
        else:  # every wide level ends in a partial warp
            V, m = 300_007, 1_500_000
        u, v = rng.integers(0, V, (2, m)).astype(np.int32)
        beg, col = ib.csr_from_edges(u, v, V)
        _CACHE[kind] = (beg, col, ib.Graph.from_csr(beg, col))
    return _CACHE[kind]


@pytest.mark.parametrize("kind,width,n", [("sparse", 32, 6), ("dense", 64, 70),
                                          ("dense", 128, 128), ("dense", 256, 200)])
@pytest.mark.parametrize("mode", [ib.MODE_PERSISTENT, ib.MODE_DEVICE_LOOP])
@pytest.mark.parametrize("switch_level", [1000, 5, -1])
def test_all_kinds(kind, width, n, mode, switch_level):
    beg, col, g = graph(kind)
    src = ib.sample_sources(beg, col, n, seed=n)
    res = g.run(src, width=width, mode=mode, switch_level=switch_level, levels_cap=256)
    ref, _ = oracle.bfs_auto(beg, col, src)
    assert np.array_equal(res.depth, ref)
    assert res.stats["traversed_edges"] == oracle.teps(beg, ref)
    if switch_level == 1000:
        V = len(beg) - 1
        mf = [r["frontier_edges"] for r in res.levels if r["dir"] in (-1, 0)]
        assert any(x * 2 >= V and x > 1 << 20 for x in mf)
        if kind == "sparse":
            assert any(1 << 20 < x < V // 2 for x in mf)
