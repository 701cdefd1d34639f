"""Device-loop runs of mixed sizes on one resident graph replay a few built
graphs: one per status word count and group count, whatever the source count."""
import ctypes

import numpy as np
import pytest

import ibfs_b200 as ib
import oracle
from ibfs_b200 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def csr():
    return ib.gen_rmat(13, 16, seed=8)


def builds(g):
    f = api._lib().ibfs_internal_graph_builds
    f.argtypes, f.restype = [ctypes.c_void_p], ctypes.c_int64
    return f(g.handle)


@pytest.mark.parametrize("width,kinds", [(128, 6), (256, 7)])
def test_mixed_sizes_share_graphs(csr, width, kinds):
    import torch

    beg, col = csr
    V = len(beg) - 1
    out = torch.empty(1500 * V, dtype=torch.uint8, device="cuda:0")
    sizes = [1500, 100, 200, 300, 500, 1000, 20, 50, 1, 129, 257, 700, 60, 1500, 33]
    refs = {n: oracle.bfs_auto(beg, col, ib.sample_sources(beg, col, n, seed=n))[0]
            for n in set(sizes)}
    with ib.Graph.from_csr(beg, col) as g:
        def run(n):
            g.run(ib.sample_sources(beg, col, n, seed=n), mode=ib.MODE_DEVICE_LOOP, width=width,
                  on_device=True, out_ptr=out.data_ptr())
            got = out[:n * V].view(n, V).cpu().numpy()
            assert np.array_equal(got, refs[n])

        for n in sizes:
            run(n)
        first = builds(g)
        assert first <= kinds
        for n in sizes * 2 + sizes[::-1]:
            run(n)
        assert builds(g) == first


def test_growing_sizes_settle(csr):
    """Sizes that grow move the baked addresses a few times, then no more."""
    import torch

    beg, col = csr
    V = len(beg) - 1
    out = torch.empty(2000 * V, dtype=torch.uint8, device="cuda:0")
    sizes = [10, 100, 500, 1000, 2000]
    with ib.Graph.from_csr(beg, col) as g:
        for turn in range(4):
            before = builds(g)
            for n in sizes:
                g.run(ib.sample_sources(beg, col, n, seed=n), mode=ib.MODE_DEVICE_LOOP,
                      on_device=True, out_ptr=out.data_ptr())
            if turn >= 2:
                assert builds(g) == before
