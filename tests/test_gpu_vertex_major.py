"""The vertex-major output on ragged shapes: batch blocks whose rows and whose
start are not aligned, word tails of every kind, vertex counts that leave a
partial step."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

_CACHE = {}


def graph(V):
    if V not in _CACHE:
        u, v = np.random.default_rng(V).integers(0, V, (2, 3 * V)).astype(np.int32)
        beg, col = ib.csr_from_edges(u, v, V)
        _CACHE[V] = (beg, col, ib.Graph.from_csr(beg, col))
    return _CACHE[V]


@pytest.mark.parametrize("width,conc", [(32, 0), (32, 7), (64, 33), (128, 97), (128, 128),
                                        (256, 250), (256, 255)])
@pytest.mark.parametrize("V", [31, 1003])
@pytest.mark.parametrize("shift", [0, 1, 2, 7, 12])
def test_ragged_blocks(width, conc, V, shift):
    import torch

    beg, col, g = graph(V)
    C = conc or width
    n = 2 * C + max(1, C // 3)
    src = np.random.default_rng(n).integers(0, V, n).astype(np.int32)
    ref, _ = oracle.bfs_auto(beg, col, src)
    for mode in (ib.MODE_PERSISTENT, ib.MODE_DEVICE_LOOP):
        out = torch.full((n * V + 64,), 77, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        g.run(src, width=width, concurrent=conc, layout=ib.LAYOUT_VERTEX_MAJOR, mode=mode,
              on_device=True, out_ptr=out.data_ptr() + shift)
        got = out.cpu().numpy()
        assert (got[:shift] == 77).all() and (got[shift + n * V:] == 77).all()
        got = got[shift:shift + n * V]
        for b in range(0, n, C):
            nb = min(C, n - b)
            assert np.array_equal(got[b * V:(b + nb) * V].reshape(V, nb).T, ref[b:b + nb])
