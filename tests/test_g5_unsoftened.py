"""Unsoftened point masses on top of a j-record, in the j-paired large CTAs (configurations 9: 1024x1J,
10: 256x1J, and the call that takes the former by default): the potential of such a pair is infinite,
and what pads a ragged j-tile to whole j-quads adds nothing to it."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _launch(g5, cfg, items, ip, jp):
    import torch
    dev = torch.device("cuda")
    di, dj = torch.from_numpy(ip).to(dev), torch.from_numpy(jp).to(dev)
    out = torch.full((len(ip), 4), np.nan, dtype=torch.float64, device=dev)
    plan = g5.plan_create(g5.NEWTON, items)
    try:
        assert g5.L.pgb5_plan_set_config(plan, cfg) == 0
        assert g5.L.pgb5_plan_launch(plan, di.data_ptr(), dj.data_ptr(), None, out.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        return out.cpu().numpy()
    finally:
        g5.plan_destroy(plan)


@pytest.mark.parametrize("cfg", [9, 10])
@pytest.mark.parametrize("nj", [1, 2, 3, 5, 255, 258, 1027, 2049])
def test_every_i_on_a_record_of_its_own(cfg, nj):
    """i = j and eps = 0: whichever record a tile starts with, one i lies on it.  One more i lies on no
    record: its force is the oracle's (2e-6 of a dozen FP32 operations a pair term)."""
    g5 = pgb.ffi.G5()
    rng = W.Rng(90 + nj)
    x = (rng.uniform(3 * nj).reshape(-1, 3) - 0.5).astype(np.float32)
    m = (rng.uniform(nj) + 0.5).astype(np.float32)
    free = np.array([[1.5, 1.25, -1.0]], np.float32)
    ip = np.concatenate([np.concatenate([x, free]), np.zeros((nj + 1, 1), np.float32)], 1)
    jp = np.concatenate([x, m[:, None]], 1)
    out = _launch(g5, cfg, [[0, nj + 1, 0, nj]], ip, jp)
    assert np.all(np.isneginf(out[:nj, 3]))
    ao, po = O.g5_newton(free.astype(np.float64), 0.0, x.astype(np.float64), m.astype(np.float64))
    np.testing.assert_allclose(out[nj:, :3], ao, rtol=2e-6, atol=2e-6 * np.abs(ao).max())
    np.testing.assert_allclose(-out[nj:, 3], po, rtol=2e-6)


def test_untuned_call_of_many_i():
    """More than 12288 i from host arrays, which run the 1024x1J configuration by default."""
    g5 = pgb.ffi.G5()
    g5.L.g5_open()
    rng = W.Rng(91)
    n, nj = 12291, 1027
    x = (rng.uniform(3 * n).reshape(-1, 3) - 0.5).astype(np.float32).astype(np.float64)
    g5.set_xmj(0, x[:nj], np.ones(nj))
    g5.L.g5_set_n(nj)
    g5.L.g5_set_eps_to_all(0.0)
    acc, pot = g5.calculate_force_on_x(x)
    assert np.all(np.isposinf(pot[:nj]))
    assert np.all(np.isfinite(pot[nj:])) and np.all(np.isfinite(acc[nj:]))
