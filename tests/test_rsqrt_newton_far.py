"""The libraries with the reference's Newton-refined rsqrt, for a compact system far from the origin: every
pair's distance is moderate, the distance to the origin squares to more than FP32 holds.  There
the refined rsqrt of an overflowed r^2 is NaN (r^2 y with y = 0), so no kernel may evaluate a pair that
is not one of the caller's, not even a massless one."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]
BASE, STEP = 1.3e19, 2.0 ** 40   # FP32 holds BASE + k STEP: the spacing of floats there
MASS, EPS2 = 1e20, 1e24


def _points(rng, n):
    # a lattice of 4 x 4 x 4 sites: distances of 1e12 to 6e12, whose inverse cubes are normal FP32 numbers
    return np.float64(np.float32(BASE)) + STEP * np.floor(4 * rng.uniform(3 * n).reshape(-1, 3))


@pytest.mark.parametrize("kind,cfg", [("newton", 7), ("newton", 9), ("newton", 10), ("quad", 7), ("quad", 10)])
def test_g5_ragged_tiles(kind, cfg):
    import torch
    dev = torch.device("cuda")
    g5 = pgb.ffi.G5("libpg5_newton.so")
    rng = W.Rng(92)
    ni, nj = 70, np.array([1, 2, 3, 5, 6, 7, 8, 253, 258, 1027])
    jo = np.concatenate([[0], np.cumsum(nj)])
    x, m = _points(rng, jo[-1]).astype(np.float32), np.full(jo[-1], MASS, np.float32)
    xi = _points(rng, ni * len(nj)).astype(np.float32)
    items = np.stack([ni * np.arange(len(nj)), np.full(len(nj), ni), jo[:-1], nj], 1)
    ip = np.concatenate([xi, np.full((len(xi), 1), EPS2, np.float32)], 1)
    jp = np.concatenate([x, m[:, None]], 1)
    di, dj = torch.from_numpy(ip).to(dev), torch.from_numpy(jp).to(dev)
    da = torch.zeros((len(jp), 8), dtype=torch.float32, device=dev) if kind == "quad" else None
    out = torch.full((len(ip), 4), np.nan, dtype=torch.float64, device=dev)
    plan = g5.plan_create(g5.QUAD if kind == "quad" else g5.NEWTON, items)
    try:
        assert g5.L.pgb5_plan_set_config(plan, cfg) == 0
        assert g5.L.pgb5_plan_launch(plan, di.data_ptr(), dj.data_ptr(), da.data_ptr() if da is not None else None,
                                     out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        out = out.cpu().numpy()
    finally:
        g5.plan_destroy(plan)
    for q in range(len(nj)):
        si, sj = slice(ni * q, ni * (q + 1)), slice(jo[q], jo[q + 1])
        ao, po = O.g5_newton(xi[si].astype(np.float64), np.float32(EPS2), x[sj].astype(np.float64), m[sj].astype(np.float64))
        # a dozen FP32 operations a pair term, as in test_g5_slots.py
        np.testing.assert_allclose(out[si, :3], ao, rtol=2e-6, atol=2e-6 * np.abs(ao).max(), err_msg=f"nj {nj[q]}")
        np.testing.assert_allclose(np.abs(out[si, 3]), po, rtol=2e-6, err_msg=f"nj {nj[q]}")


@pytest.mark.parametrize("n", [2, 3, 5, 257, 513, 771])
def test_integrator_odd_chunks(n):
    """The step kernel's j-chunks of an odd number of particles: start-up forces of n particles."""
    g6 = pgb.ffi.G6("libpg6_newton.so")
    g6.L.g6_open(0)
    rng = W.Rng(93 + n)
    x = _points(rng, n)
    v = rng.uniform(3 * n).reshape(-1, 3) - 0.5
    m = np.full(n, MASS)
    H = pgb.ffi.Hermite(g6, m, x, v, EPS2, 0.2, 0.01, 0.125)
    try:
        s = H.get()
    finally:
        H.close()
    ref = O.g6_force(x, v.astype(np.float32).astype(np.float64), np.arange(n, dtype=np.int32), np.float32(EPS2), x,
                     v.astype(np.float32).astype(np.float64), m, np.arange(n, dtype=np.int32))
    # FP32 pair terms; the tolerances of test_g6_quad_nn.py (acc 2e-6, the cancelling jerk 1e-5 of the largest)
    np.testing.assert_allclose(s["acc"], ref["acc"], rtol=2e-6, atol=2e-6 * np.abs(ref["acc"]).max())
    np.testing.assert_allclose(s["jrk"], ref["jrk"], rtol=1e-5, atol=1e-5 * np.abs(ref["jrk"]).max())
