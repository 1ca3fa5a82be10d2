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


@pytest.mark.parametrize("ni,nj", [(777, 65536), (2048, 4096)])
def test_noalloc_takes_a_plan_s_time(ni, nj):
    """The allocation-free call runs the same kernels as an untuned plan (777 x 65536: 201 us in chunks of
    its own, 99 in a plan's), and returns the same forces up to the order of the sums."""
    import torch
    g6 = pgb.ffi.G6()
    f = pgb.ffi.bind_noalloc(g6)
    di, dj, do = _records(ni, nj, True)
    s = torch.cuda.current_stream().cuda_stream
    plan = g6.plan_create([[0, ni, 0, nj]], nn=True)
    try:
        t_plan = _us(lambda: g6.plan_launch(plan, di.data_ptr(), dj.data_ptr(), 1e-4, do.data_ptr(), s))
        want = do.cpu().numpy().view(pgb.ffi.G6OUT).copy()
        do.fill_(255)
        t = _us(lambda: f(di.data_ptr(), ni, dj.data_ptr(), nj, 1e-4, do.data_ptr(), g6.NN, s))
        got = do.cpu().numpy().view(pgb.ffi.G6OUT)
    finally:
        g6.plan_destroy(plan)
    assert t <= 1.4 * t_plan + 5.0   # and its two small launches more
    np.testing.assert_array_equal(got["jadr"], want["jadr"])
    for c in ("ax", "ay", "az", "jx", "jy", "jz", "pot"):
        # FP32 partial sums of at most 256 terms in other groups: some 1e-7 of the largest
        np.testing.assert_allclose(got[c], want[c], rtol=1e-6, atol=1e-6 * np.abs(want[c]).max())


@pytest.mark.parametrize("ni,nj", [(1, 1), (65, 129), (129, 127), (777, 1), (1000, 0), (3073, 300), (5000, 1031)])
def test_noalloc_ragged_sizes(ni, nj):
    import torch
    g6 = pgb.ffi.G6()
    f = pgb.ffi.bind_noalloc(g6)
    di, dj, do = _records(ni, max(nj, ni), True)
    s = torch.cuda.current_stream().cuda_stream
    plan = g6.plan_create([[0, ni, 0, nj]], nn=False)
    try:
        assert f(di.data_ptr(), ni, dj.data_ptr(), nj, 1e-4, do.data_ptr(), 0, s) == 0
        got = do.cpu().numpy().view(pgb.ffi.G6OUT).copy()
        g6.plan_launch(plan, di.data_ptr(), dj.data_ptr(), 1e-4, do.data_ptr(), s)
        want = do.cpu().numpy().view(pgb.ffi.G6OUT)
    finally:
        g6.plan_destroy(plan)
    for c in ("ax", "ay", "az", "jx", "jy", "jz", "pot"):
        np.testing.assert_allclose(got[c], want[c], rtol=1e-6, atol=1e-6 * max(np.abs(want[c]).max(), 1e-30))
