"""Graphs whose last, partial range of 32 vertices lies above the bottom-up
thread-path limit: the prefix of big vertices must end inside the graph."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu


def dense(V, deg, seed):
    rng = np.random.default_rng(seed)
    u, v = rng.integers(0, V, (2, V * deg // 2)).astype(np.int32)
    # a ring of 20 neighbours to each side keeps every degree at 40 or more
    i = np.repeat(np.arange(V, dtype=np.int32), 20)
    j = (i + np.tile(np.arange(1, 21, dtype=np.int32), V)) % V
    return ib.csr_from_edges(np.concatenate([u, i]), np.concatenate([v, j]).astype(np.int32), V)


@pytest.mark.parametrize("V,deg", [(63, 60), (65, 30), (1003, 100), (4001, 60), (1024, 60)])
@pytest.mark.parametrize("mode", [ib.MODE_PLAIN, ib.MODE_PERSISTENT, ib.MODE_DEVICE_LOOP])
def test_every_vertex_big(V, deg, mode):
    beg, col = dense(V, deg, seed=V)
    assert np.diff(beg).min() > 32
    src = ib.sample_sources(beg, col, 40, seed=3)
    ref, _ = oracle.bfs_auto(beg, col, src)
    with ib.Graph.from_csr(beg, col) as g:
        for switch_level in (0, 1, -1):
            for width in (32, 128):
                res = g.run(src, mode=mode, width=width, switch_level=switch_level)
                assert np.array_equal(res.depth, ref)
                assert res.stats["traversed_edges"] == oracle.teps(beg, ref)


@pytest.mark.parametrize("mode", [ib.MODE_PLAIN, ib.MODE_PERSISTENT, ib.MODE_DEVICE_LOOP])
@pytest.mark.parametrize("bu_thread_max", [1, 2, 8])
def test_small_thread_limit(mode, bu_thread_max):
    beg, col = ib.gen_grid(37, 27, seed=6)  # 999 vertices of degree 1 to 4
    src = ib.sample_sources(beg, col, 64, seed=5)
    ref, _ = oracle.bfs_auto(beg, col, src)
    with ib.Graph.from_csr(beg, col) as g:
        res = g.run(src, mode=mode, bu_thread_max=bu_thread_max, switch_level=1)
    assert np.array_equal(res.depth, ref)
