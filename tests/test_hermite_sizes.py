"""GPU Hermite integrator at the sizes where its step kernel can go wrong, replayed step by step.

* n = 2, 3: chunks of one particle or none; 255, 257: a segment less one, one more; 600: an odd
  split of j over the chunks, every small and middle decomposition; 5001: two i per thread with a
  ragged last tile; 160001: more segments than two per CTA (those past the second keep no times in
  shared memory), tasks without a split j-range.

As in test_hermite_gpu.py the oracle replays every step with the GPU's force of that step: block
time, active set and new state are equal bit for bit, and the forces are within that file's
tolerances (rms 1e-6, largest 1e-4) of the FP64 oracle, here for up to 64 active particles a step.
"""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O
from test_hermite_gpu import ForceCheck, _assert_state_equal

pytestmark = pytest.mark.gpu

W = pgb.workloads


@pytest.mark.parametrize("n,nsteps", [(2, 40), (3, 40), (255, 80), (257, 80), (600, 120), (5001, 60), (160001, 10)])
def test_sizes_replay_bit_exact(n, nsteps):
    if not gpu_available():
        pytest.skip("no GPU")
    g6 = pgb.ffi.G6()
    g6.L.g6_open(0)
    eps2, eta, eta_s, dtmax = 1.0 / 64 ** 2, 0.2, 0.01, 0.125
    x, v, m, _ = W.plummer_hermite(n, W.SEED0 + n)
    H = pgb.ffi.Hermite(g6, m, x, v, eps2, eta, eta_s, dtmax)
    st = O.HermiteState(x, v, m, dtmax)
    fc = ForceCheck(st, eps2)

    def forces(t_gl, act, xp, vp, acc, jrk, pot):
        k = np.unique(np.linspace(0, len(act) - 1, min(len(act), 64)).astype(int))
        fc.add(t_gl, act[k], xp[k], vp[k], acc[k], jrk[k], pot[k])

    try:
        act, acc, jrk, pot = H.last_step()
        np.testing.assert_array_equal(act, np.arange(n))
        xp, vp = O.hermite_predict(st, act, 0.0)
        forces(0.0, act, xp, vp, acc, jrk, pot)
        O.hermite_startup(st, act, acc, jrk, pot, eta_s, dtmax)
        _assert_state_equal(H, st, "start-up")
        for k in range(nsteps):
            _, ni = H.step()
            t_gl, act_o = O.hermite_select(st)
            act, acc, jrk, pot = H.last_step()
            assert ni == len(act)
            np.testing.assert_array_equal(act, act_o, err_msg=f"step {k}")
            xp, vp = O.hermite_predict(st, act, t_gl)
            forces(t_gl, act, xp, vp, acc, jrk, pot)
            O.hermite_correct(st, act, t_gl, xp, vp, acc, jrk, pot, eta, dtmax)
            if t_gl - int(t_gl * (1.0 / dtmax)) * dtmax == 0.0:
                st.t[:] = 0.0
            _assert_state_equal(H, st, f"step {k} (t_gl {t_gl}, ni {ni})")
        fc.check()
    finally:
        H.close()
