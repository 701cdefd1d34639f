"""A graph or a server opened while the program's default stream is busy: nothing
of the open may be left to that stream, which is not ordered with theirs."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [8, 14])  # ordered on the host and on the GPU
def test_open_behind_busy_default_stream(scale):
    import torch

    beg, col = ib.gen_rmat(scale, 16, seed=3)
    src = ib.sample_sources(beg, col, 40, seed=7)
    ref, _ = oracle.bfs_auto(beg, col, src)
    torch.zeros(1, device="cuda:0")
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about 0.1 s on the default stream
    with ib.Graph.from_csr(beg, col) as g:
        torch.cuda.synchronize()
        for mode in (ib.MODE_PERSISTENT, ib.MODE_DEVICE_LOOP):
            assert np.array_equal(g.run(src, mode=mode).depth, ref)


def test_server_behind_busy_default_stream():
    import torch

    beg, col = ib.gen_rmat(12, 16, seed=5)
    src = ib.sample_sources(beg, col, 30, seed=2)
    ref, _ = oracle.bfs_auto(beg, col, src)
    with ib.Graph.from_csr(beg, col) as g:
        torch.zeros(1, device="cuda:0")
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)
        with ib.Server(g) as srv:
            depth, _ = srv.wait(srv.submit(src), len(src))
            assert np.array_equal(depth, ref)
