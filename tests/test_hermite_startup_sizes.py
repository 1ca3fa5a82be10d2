"""The integrator's start-up step around 128 particles (more of them run in an instance of the step kernel of
their own) and where its force decomposition changes: the oracle's start-up given the GPU's forces, bit for bit,
and the forces against the FP64 oracle as in test_hermite_gpu.py."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O
from test_hermite_gpu import ForceCheck, _assert_state_equal

pytestmark = pytest.mark.gpu
W = pgb.workloads


@pytest.mark.parametrize("n", [16, 17, 33, 127, 128, 129, 2048, 2049])
def test_startup_step(n):
    if not gpu_available():
        pytest.skip("no GPU")
    g6 = pgb.ffi.G6()
    g6.L.g6_open(0)
    eps2, eta_s, dtmax = 1.0 / 64 ** 2, 0.01, 0.125
    x, v, m, _ = W.plummer_hermite(n, W.SEED0 + 7 * n)
    H = pgb.ffi.Hermite(g6, m, x, v, eps2, 0.2, eta_s, dtmax)
    try:
        assert H.counts() == (n, 1) and H.time == 0.0
        st = O.HermiteState(x, v, m, dtmax)
        act, acc, jrk, pot = H.last_step()
        np.testing.assert_array_equal(act, np.arange(n))
        xp, vp = O.hermite_predict(st, act, 0.0)
        fc = ForceCheck(st, eps2)
        fc.add(0.0, act, xp, vp, acc, jrk, pot)
        O.hermite_startup(st, act, acc, jrk, pot, eta_s, dtmax)
        _assert_state_equal(H, st, "start-up")
        fc.check()
        H.step()   # and the first step finds what it left
        assert H.counts()[1] == 2 and H.time > 0.0
    finally:
        H.close()
