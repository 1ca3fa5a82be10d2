"""GRAPE-5 plans and calls of few j-records: the default configuration against the oracle at the sizes
where its rule changes (16 and 64 j, 64 i, 2^17 i in all), and against another configuration's time."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]
CFG_128x2, CFG_128x1, CFG_64x1, CFG_1024x1J = 5, 6, 7, 9


class _Plan:
    def __init__(self, kind, items, ni, nj):
        import torch
        rng = W.Rng(99)
        self.g5 = pgb.ffi.G5Sym() if kind == "symmetric" else pgb.ffi.G5()
        k = {"newton": self.g5.NEWTON, "symmetric": self.g5.SYMMETRIC_KIND, "quad": self.g5.QUAD}[kind]
        self.ip = np.concatenate([rng.uniform(3 * ni).reshape(-1, 3) - 0.5, np.full((ni, 1), 1e-3)], 1).astype(np.float32)
        self.jp = np.concatenate([rng.uniform(3 * nj).reshape(-1, 3) - 0.5, rng.uniform(nj)[:, None] + 0.5], 1).astype(np.float32)
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()   # noqa: E731
        self.di, self.dj = put(self.ip), put(self.jp)
        self.da = torch.zeros((nj, 8 if kind == "quad" else 4), device="cuda") if kind != "newton" else None
        self.out = torch.full((ni, 4), np.nan, dtype=torch.float64, device="cuda")
        self.h = self.g5.plan_create(k, items)

    def launch(self):
        import torch
        self.g5.plan_launch(self.h, self.di.data_ptr(), self.dj.data_ptr(), self.da.data_ptr() if self.da is not None else None,
                            self.out.data_ptr(), torch.cuda.current_stream().cuda_stream)

    def us(self):
        import torch
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = 1e9
        for _ in range(5):
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                self.launch()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) / 20 * 1e3)
        return best

    def close(self):
        self.g5.plan_destroy(self.h)


@pytest.mark.parametrize("kind", ["newton", "symmetric", "quad"])
@pytest.mark.parametrize("items,nj,cfg", [([(63, 16)], 16, CFG_64x1), ([(64, 16)], 16, CFG_128x1), ([(64, 17)], 17, CFG_64x1),
                                          ([(65, 1), (3, 16), (129, 7)], 16, CFG_128x1), ([(64, 0)], 1, CFG_64x1),
                                          ([(131072, 17)], 17, None), ([(131073, 64)], 64, CFG_128x1), ([(131073, 65)], 65, None)])
def test_default_at_the_edges_of_the_rule(kind, items, nj, cfg):
    ni = np.array([i[0] for i in items])
    io = np.concatenate([[0], np.cumsum(ni)])
    it = [[int(io[k]), i, 0, j] for k, (i, j) in enumerate(items)]
    P = _Plan(kind, it, int(io[-1]), nj)
    try:
        if cfg is None:
            cfg = CFG_1024x1J if kind == "newton" else CFG_64x1
        assert P.g5.L.pgb5_plan_config(P.h) == cfg
        P.launch()
        out = P.out.cpu().numpy()
    finally:
        P.close()
    for k, (i, j) in enumerate(items):
        s = np.unique(np.linspace(io[k], io[k + 1] - 1, 200).astype(int))   # enough of a large item
        if j == 0:
            assert not out[s].any()
            continue
        a, p = O.g5_newton(P.ip[s, :3].astype(np.float64), P.ip[s, 3], P.jp[:j, :3].astype(np.float64), P.jp[:j, 3].astype(np.float64))
        # a dozen FP32 operations a pair term, as in test_g5_slots.py
        np.testing.assert_allclose(out[s, :3], a, rtol=2e-6, atol=2e-6 * np.abs(a).max())
        np.testing.assert_allclose(np.abs(out[s, 3]), p, rtol=2e-6)


@pytest.mark.parametrize("kind", ["symmetric", "quad"])
def test_default_is_no_slower_than_the_scalar_form(kind):
    """262144 i against 4 j: 12 to 17 us in the slot kernel, 7 in the two-i form of 128 threads."""
    P = _Plan(kind, [[0, 262144, 0, 4]], 262144, 4)
    try:
        P.launch()
        default = P.us()
        assert P.g5.L.pgb5_plan_set_config(P.h, CFG_128x2) == 0
        P.launch()
        assert default <= 1.4 * P.us()
    finally:
        P.close()
