"""The group count yields to device memory, also when the groups' workspaces
exist already but have to grow: narrow batches first, wide ones after, with
little memory left."""
import numpy as np
import pytest

import ibfs_b200 as ib
import oracle

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_wider_run_with_little_memory():
    import torch

    # 2^20 vertices: 42 MB per group in 32-bit words, 340 MB in 256-bit words
    V = 1 << 20
    rng = np.random.default_rng(2)
    u, v = rng.integers(0, V, (2, 2 * V)).astype(np.int32)
    beg, col = ib.csr_from_edges(u, v, V)
    src = ib.sample_sources(beg, col, 4 * 256, seed=1)
    out = torch.empty(len(src) * V, dtype=torch.uint8, device="cuda:0")
    ref, _ = oracle.bfs_auto(beg, col, src[:8])
    with ib.Graph.from_csr(beg, col) as g:
        def run(n, concurrent):
            r = g.run(src[:n], mode=ib.MODE_DEVICE_LOOP, width=256, concurrent=concurrent, on_device=True,
                      out_ptr=out.data_ptr())
            assert np.array_equal(out[:8 * V].view(8, V).cpu().numpy(), ref)
            return r.stats["groups"]

        assert run(32, 8) == 4
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        filler = torch.empty(max(0, free - 900 * MB), dtype=torch.uint8, device="cuda:0")
        try:
            assert 1 <= run(1024, 256) < 4
        finally:
            del filler
            torch.cuda.empty_cache()
        run(32, 8)
        run(1024, 256)


def test_out_of_memory_leaves_no_error_behind():
    """A run that does not fit says so; the program's next CUDA call and a run
    that fits are not affected."""
    import torch

    V = 1 << 20
    rng = np.random.default_rng(3)
    u, v = rng.integers(0, V, (2, V)).astype(np.int32)
    beg, col = ib.csr_from_edges(u, v, V)
    src = ib.sample_sources(beg, col, 256, seed=1)
    out = torch.empty(len(src) * V, dtype=torch.uint8, device="cuda:0")
    ref, _ = oracle.bfs_auto(beg, col, src[:8])
    with ib.Graph.from_csr(beg, col) as g:
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        filler = torch.empty(max(0, free - 150 * MB), dtype=torch.uint8, device="cuda:0")
        try:
            with pytest.raises(ib.IbfsError, match="OOM"):
                g.run(src, width=256, on_device=True, out_ptr=out.data_ptr())
            out.zero_()
            g.run(src[:8], width=256, on_device=True, out_ptr=out.data_ptr())
            assert np.array_equal(out[:8 * V].view(8, V).cpu().numpy(), ref)
        finally:
            del filler
            torch.cuda.empty_cache()
