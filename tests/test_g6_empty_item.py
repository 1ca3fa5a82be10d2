"""Hermite plans of an item without j-records: no force, no neighbour, in every configuration."""
import numpy as np
import pytest

from conftest import gpu_available, pgb

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


@pytest.mark.parametrize("f64", [False, True])
@pytest.mark.parametrize("items", [[[0, 70, 0, 0]], [[0, 1, 0, 0]], [[0, 30, 0, 0], [30, 40, 0, 5]]])
def test_no_j(items, f64):
    import torch
    g6 = pgb.ffi.G6()
    x = np.linspace(0.0, 1.0, 210).reshape(70, 3)
    ids = np.arange(70, dtype=np.int32)
    put = lambda a: torch.from_numpy(a.view(np.uint8)).cuda()   # noqa: E731
    di = put(pgb.ffi.g6_irecords(x, x, ids + 100, ff=not f64))
    dj = put(pgb.ffi.g6_jrecords(x[:5], x[:5], np.ones(5), ids[:5], ff=not f64))
    plan = g6.plan_create(items, nn=True, f64=f64)
    try:
        for cfg in [None] + list(range(10)):
            if cfg is not None:
                assert g6.L.pgb6_plan_set_config(plan, cfg) == 0
            do = torch.full((70 * pgb.ffi.G6OUT.itemsize,), 255, dtype=torch.uint8, device="cuda")
            g6.plan_launch(plan, di.data_ptr(), dj.data_ptr(), 1e-4, do.data_ptr(), 0)
            torch.cuda.synchronize()
            o = do.cpu().numpy().view(pgb.ffi.G6OUT)[:items[0][1]]
            for c in ("ax", "ay", "az", "jx", "jy", "jz", "pot"):
                assert not o[c].any(), (cfg, c)
            assert np.all(o["jadr"] == -1)
    finally:
        g6.plan_destroy(plan)
