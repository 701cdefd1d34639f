"""A neighbour list with 2^31 entries and more (duplicates): positions inside
it do not fit 32 bits.  Run through the entry point that takes a device CSR,
which is filled on the GPU."""
import ctypes as C

import numpy as np
import pytest

from ibfs_b200 import api

pytestmark = pytest.mark.gpu


def test_list_beyond_32_bits():
    import torch

    # vertex 0: [4, 1, 1, ..., 2]; 4: [0, 2, 2, ...]; an edge that exists one
    # way exists the other way too
    n0, n4 = (1 << 31) + 77, 1 << 30
    lists = {1: [0], 2: [0, 3, 4], 3: [2]}
    deg = [n0, 1, 3, 1, n4]
    beg = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    V, E = 5, int(beg[-1])
    dev = torch.device("cuda", 0)
    if torch.cuda.mem_get_info()[0] < 4 * E + (2 << 30):
        pytest.skip("needs 15 GB of device memory")
    col = torch.empty(E, dtype=torch.int32, device=dev)
    col[:n0] = 1
    col[0], col[n0 - 1] = 4, 2
    for v, nb in lists.items():
        col[int(beg[v]):int(beg[v + 1])] = torch.tensor(nb, dtype=torch.int32, device=dev)
    col[int(beg[4]):] = 2
    col[int(beg[4])] = 0
    depth = np.array([[0, 1, 1, 2, 1], [1, 0, 2, 3, 2], [1, 2, 0, 1, 1], [2, 3, 1, 0, 2],
                      [1, 2, 1, 2, 0]], np.uint8)  # [source][vertex]
    beg_d = torch.from_numpy(beg).to(dev)
    stream = torch.cuda.current_stream(dev).cuda_stream
    try:
        for src in ([4], [3], [0, 1, 2, 3, 4]):
            src_d = torch.tensor(src, dtype=torch.int32, device=dev)
            out = torch.zeros(V * len(src), dtype=torch.uint8, device=dev)
            edges = C.c_int64(-1)
            st = api._lib().ibfs_run_static_scratch(
                C.c_void_p(beg_d.data_ptr()), C.c_void_p(col.data_ptr()), V, E,
                C.c_void_p(src_d.data_ptr()), len(src), 32, C.c_void_p(out.data_ptr()),
                C.c_void_p(stream), C.byref(edges))
            assert st == 0
            assert np.array_equal(out.cpu().numpy().reshape(V, len(src)).T, depth[src])
            assert edges.value == len(src) * E
    finally:
        del col
        torch.cuda.empty_cache()
