"""Host-buffer runs of the persistent schedule around the staging ring's
sizes: below 1 MB (one copy), from there through 4 MiB slots, with row lengths
that divide neither a slot nor a spread piece."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    beg, col = ib.gen_chung_lu(9973, 120000, 2.1, 900.0, seed=15)
    g = ib.Graph.from_csr(beg, col)
    yield beg, col, g
    g.close()


@pytest.mark.parametrize("layout", [ib.LAYOUT_SOURCE_MAJOR, ib.LAYOUT_VERTEX_MAJOR])
@pytest.mark.parametrize("n", [105, 106, 421, 1300])  # 1.04 MB is between 105 and 106 rows
def test_staged_rows(graph, n, layout):
    beg, col, g = graph
    src = ib.sample_sources(beg, col, n, seed=n)
    res = g.run(src, width=64, mode=ib.MODE_PERSISTENT, layout=layout)
    ref, _ = oracle.bfs_auto(beg, col, src)
    got = res.depth
    if layout == ib.LAYOUT_VERTEX_MAJOR:
        V, C = len(beg) - 1, 64
        got = np.concatenate([got[b * V:(b + min(C, n - b)) * V].reshape(V, -1).T
                              for b in range(0, n, C)])
    assert np.array_equal(got, ref)
