"""The j-chunks that untuned Hermite launches take by default."""
import numpy as np
import pytest

from conftest import gpu_available, pgb

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _records(ni, nj, ff):
    import torch
    rng = W.Rng(104)
    x, v = rng.uniform(3 * nj).reshape(-1, 3), rng.uniform(3 * nj).reshape(-1, 3)
    ids = np.arange(nj, dtype=np.int32)
    put = lambda a: torch.from_numpy(a.view(np.uint8)).cuda()   # noqa: E731
    return (put(pgb.ffi.g6_irecords(x[:ni], v[:ni], ids[:ni], ff=ff)),
            put(pgb.ffi.g6_jrecords(x, v, np.full(nj, 1.0 / nj), ids, ff=ff)),
            torch.zeros(ni * pgb.ffi.G6OUT.itemsize, dtype=torch.uint8, device="cuda"))


def _us(f, n=10):
    import torch
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    f()
    best = 1e9
    for _ in range(4):
        torch.cuda.synchronize()
        a.record()
        for _ in range(n):
            f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / n * 1e3)
    return best


@pytest.mark.parametrize("ni,nj,lo,hi", [(4096, 65536, 20, 60), (4096, 4096, 8, 20)])
def test_fp64_positions_chunk_counts(ni, nj, lo, hi):
    """4096 i x 65536 j in 13 chunks take 496 us (one wave of tasks, the SMs unevenly filled), in 27 to 37 451;
    against 4096 j it is the other way: 13 chunks 44 us, 27 52."""
    g6 = pgb.ffi.G6()
    plan = g6.plan_create([[0, ni, 0, nj]], nn=True, f64=True)
    try:
        assert lo <= g6.L.pgb6_plan_chunks(plan) <= hi
    finally:
        g6.plan_destroy(plan)
