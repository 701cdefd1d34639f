"""The resident graph's internal order built on the GPU (8,192 edges and
more): vertices by degree, highest first, ties by caller id; every list
renamed and ascending, duplicates kept; GroupBy's hub table.  Against numpy,
around the sort's tile (4,096 keys), scan and digit sizes."""
import numpy as np
import pytest

import ibfs_b200 as ib

pytestmark = pytest.mark.gpu


def _csr(V, E, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "even":  # every vertex the same degree: ties only
        src = np.arange(E) % V
    elif kind == "hub":  # half the edges in one list, most vertices edgeless
        src = np.where(rng.random(E) < 0.5, V // 3, rng.integers(0, max(1, V // 5), E))
    else:
        src = np.minimum((V * rng.random(E) ** 3).astype(np.int64), V - 1)
    src = np.sort(src)
    col = rng.integers(0, V, E).astype(np.int32)  # directed, duplicates and loops
    beg = np.zeros(V + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=V), out=beg[1:])
    return beg, col


def _device_array(ptr, count, dtype):
    import torch

    t = torch.empty(count, dtype=dtype, device="cuda")
    from cuda.bindings import runtime as rt

    err, = rt.cudaMemcpy(t.data_ptr(), ptr, count * t.element_size(),
                         rt.cudaMemcpyKind.cudaMemcpyDeviceToDevice)
    assert err == rt.cudaError_t.cudaSuccess
    return t.cpu().numpy()


@pytest.mark.parametrize("kind", ["even", "hub", "skew"])
@pytest.mark.parametrize("V,E", [(2, 8192), (255, 8193), (257, 69631), (4097, 69633),
                                 (65536, 131072), (70001, 300007)])
def test_order_matches_numpy(V, E, kind):
    import torch

    beg, col = _csr(V, E, kind, V + E)
    with ib.Graph.from_csr(beg, col) as g:
        bp, cp = g.device_csr()
        nb = _device_array(bp, V + 1, torch.int64)
        nc = _device_array(cp, E, torch.int32)
        nm = _device_array(g.vertex_order(), V, torch.int32)
        src = np.random.default_rng(1).integers(0, V, 500).astype(np.int32)
        dsrc = torch.from_numpy(src).cuda()
        dout = torch.empty_like(dsrc)
        torch.cuda.synchronize()
        g.groupby_device(dsrc.data_ptr(), len(src), dout.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(dout.cpu().numpy(), ib.groupby_csr(beg, col, src))
        assert g.max_degree == int(np.diff(beg).max())
    deg = np.diff(beg)
    order = np.argsort(-deg, kind="stable")
    assert np.array_equal(nm[order], np.arange(V))
    assert np.array_equal(nb[1:], np.cumsum(deg[order]))
    new_src = np.repeat(nm, deg)
    at = np.lexsort((nm[col], new_src))
    assert np.array_equal(nc, nm[col][at])
