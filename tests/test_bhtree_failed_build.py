"""A rebuild that fails half-way (no device memory left) is reported once: the next build, of another tree,
succeeds."""
import numpy as np
import pytest

from conftest import gpu_available, pgb

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def test_a_failed_rebuild_leaves_the_library_usable():
    import torch
    n = 1 << 25
    rng = W.Rng(96)
    x = torch.zeros((n, 3), dtype=torch.float64).pin_memory()
    m = torch.full((n,), 1.0 / n, dtype=torch.float64).pin_memory()
    small = rng.uniform(3000).reshape(-1, 3)
    T = W.GpuTree(small, np.ones(len(small)))
    L = T.L
    L.pgbt_set_abort(0)
    try:
        nodes = L.pgbt_nnodes(T.h)
        # room for the uploads (the arrays' sizes rounded up to powers of two) and no more: the
        # permutation, 128 MB, is the first array that does not fit
        room = (1 << 30) + (1 << 28) + (48 << 20)
        torch.cuda.empty_cache()
        filler = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        left = torch.cuda.mem_get_info()[0]
        if not (1 << 30) + (1 << 28) < left < (1 << 30) + (1 << 28) + (100 << 20):
            pytest.skip(f"could not leave the room wanted ({left} bytes)")
        with pytest.raises(RuntimeError):
            T.rebuild(x.numpy(), m.numpy())
        del filler
        torch.cuda.empty_cache()
        T.close()
        T = W.GpuTree(small, np.ones(len(small)))
        assert L.pgbt_nnodes(T.h) == nodes
    finally:
        L.pgbt_clear_error()
        L.pgbt_set_abort(1)
        T.close()
        torch.cuda.empty_cache()
