"""Untuned Hermite batches of small items: the default configuration's forces and nearest neighbours against
the oracle where its rule changes, and its time against configurations that may be set."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]
SMALL, MED = 0, 1


class _Batch:
    def __init__(self, shapes, nn=True):
        import torch
        self.shapes = shapes
        ni, nj = np.array([s[0] for s in shapes]), np.array([s[1] for s in shapes])
        self.io, self.jo = np.concatenate([[0], np.cumsum(ni)]), np.concatenate([[0], np.cumsum(nj)])
        rng = W.Rng(105)
        f32 = lambda a: a.astype(np.float32).astype(np.float64)   # noqa: E731
        n, m = int(self.io[-1]), int(self.jo[-1])
        self.xi, self.xj = rng.uniform(3 * n).reshape(-1, 3), rng.uniform(3 * m).reshape(-1, 3)
        self.vi, self.vj = f32(rng.uniform(3 * n).reshape(-1, 3)), f32(rng.uniform(3 * m).reshape(-1, 3))
        self.mj, self.idj = f32(rng.uniform(m) + 0.5), np.arange(m, dtype=np.int32)
        self.idi = np.concatenate([np.arange(a) + self.jo[k] if k % 2 and a <= b else np.full(a, -1)
                                   for k, (a, b) in enumerate(shapes)]).astype(np.int32)
        put = lambda a: torch.from_numpy(a.view(np.uint8)).cuda()   # noqa: E731
        self.di = put(pgb.ffi.g6_irecords(self.xi, self.vi, self.idi))
        self.dj = put(pgb.ffi.g6_jrecords(self.xj, self.vj, self.mj, self.idj))
        self.do = torch.full((n * pgb.ffi.G6OUT.itemsize,), 255, dtype=torch.uint8, device="cuda")
        self.g6 = pgb.ffi.G6()
        self.h = self.g6.plan_create(np.stack([self.io[:-1], ni, self.jo[:-1], nj], 1), nn=nn)

    def launch(self):
        import torch
        self.g6.plan_launch(self.h, self.di.data_ptr(), self.dj.data_ptr(), 1e-4, self.do.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)

    def us(self):
        import torch
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        self.launch()
        best = 1e9
        for _ in range(5):
            torch.cuda.synchronize()
            a.record()
            for _ in range(10):
                self.launch()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) / 10 * 1e3)
        return best

    def close(self):
        self.g6.plan_destroy(self.h)


@pytest.mark.parametrize("shapes,cfg", [
    ([(1, 1), (3, 128), (64, 200)], SMALL),                       # little work
    ([(16, 127), (30, 100)], MED),                                # under 128 j
    ([(1, 1800)] * 48, SMALL), ([(1, 700)] * 48, MED), ([(9, 5000)] * 47, MED),   # many items of few i
    ([(33, 9000), (64, 6000), (2, 12001), (7, 3000)], SMALL),     # up to four, more than 32 i
    ([(32, 9000), (5, 6000), (2, 12001), (7, 3000)], MED),
    ([(5, 33000), (30, 40000)], SMALL), ([(5, 33000), (30, 20000), (2, 33001), (7, 3000)], MED),
    ([(100, 16384), (129, 3001)], MED),                           # middle work: one i per thread
    ([(300, 9000), (4, 1), (257, 12001)], MED),
])
def test_default_forces(shapes, cfg):
    B = _Batch(shapes)
    try:
        assert B.g6.L.pgb6_plan_config(B.h) == cfg
        for _ in range(2):
            B.launch()
        out = B.do.cpu().numpy().view(pgb.ffi.G6OUT)
    finally:
        B.close()
    for q in range(len(shapes)):
        si, sj = slice(B.io[q], B.io[q + 1]), slice(B.jo[q], B.jo[q + 1])
        o = out[si]
        ref = O.g6_force(B.xi[si], B.vi[si], B.idi[si], np.float32(1e-4), B.xj[sj], B.vj[sj], B.mj[sj], B.idj[sj])
        # the tolerances of test_g6_quad_nn.py
        for f, cs, tol in (("acc", ("ax", "ay", "az"), 2e-6), ("jrk", ("jx", "jy", "jz"), 1e-5)):
            got = np.stack([o[c] for c in cs], 1)
            np.testing.assert_allclose(got, ref[f], rtol=tol, atol=tol * max(np.abs(ref[f]).max(), 1e-30), err_msg=str(shapes[q]))
        if shapes[q][1] > 1:
            clear = ref["r2nn2"] / ref["r2nn"] - 1.0 > 1e-5
            np.testing.assert_array_equal(o["jadr"][clear], ref["nnb"][clear])


@pytest.mark.parametrize("shapes,cfg,limit", [([(1, 1024)] * 256, SMALL, 1.2), ([(16, 4096)] * 4, SMALL, 1.1),
                                              ([(128, 4096)] * 4, MED, 0.9)])
def test_default_time(shapes, cfg, limit):
    """256 items of 1 i x 1024 j 55 us with two i per thread, 37 with SMALL; 4 of 16 x 4096 14.6 and 12.5; 4 of
    128 x 4096 23.8, with one i per thread 17.6."""
    B = _Batch(shapes)
    try:
        default = B.us()
        assert B.g6.L.pgb6_plan_set_config(B.h, cfg) == 0
        assert default <= limit * B.us()
    finally:
        B.close()


def test_a_tuned_plan_of_the_unlisted_form_is_kept():
    """The tuner tries the one-i form too; the plan reports MED for it and later plans of the shape take it."""
    import torch
    B = _Batch([(128, 4096)] * 4)
    try:
        untuned = B.us()
        cfg, _ = B.g6.plan_tune(B.h, B.di.data_ptr(), B.dj.data_ptr(), 1e-4, B.do.data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
        assert 0 <= cfg < 10 and B.g6.L.pgb6_plan_config(B.h) == cfg
        assert B.us() <= 1.1 * untuned
        assert B.g6.L.pgb6_plan_set_config(B.h, cfg) == 0
    finally:
        B.close()
