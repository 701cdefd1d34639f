"""Runs with fewer sources than the width keep only the status words their
batch needs: depths, edge counts and the reported width stay those of the
width asked for."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    beg, col = ib.gen_rmat(12, 12, seed=41)
    g = ib.Graph.from_csr(beg, col)
    yield beg, col, g
    g.close()


@pytest.mark.parametrize("n", [1, 32, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("mode", [ib.MODE_PLAIN, ib.MODE_PERSISTENT, ib.MODE_DEVICE_LOOP,
                                  ib.MODE_AUTO])
def test_words_follow_sources(graph, mode, n):
    beg, col, g = graph
    src = ib.sample_sources(beg, col, n, seed=n)
    res = g.run(src, width=256, mode=mode)
    ref, _ = oracle.bfs_auto(beg, col, src)
    assert np.array_equal(res.depth, ref)
    assert res.stats["traversed_edges"] == oracle.teps(beg, ref)
    assert res.stats["width"] == 256
