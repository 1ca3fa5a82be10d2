"""GRAPE-5 calls of many i against few j: the results at the edge of the rule that chooses their way to
the host (words up to 256 i and 16 more for every j, a copy beyond)."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _set(g5, nj):
    rng = W.Rng(101)
    x = (rng.uniform(3 * nj).reshape(-1, 3) - 0.5).astype(np.float32).astype(np.float64)
    m = (rng.uniform(nj) + 0.5).astype(np.float32).astype(np.float64)
    g5.L.g5_open()
    g5.set_xmj(0, x, m)
    g5.L.g5_set_n(nj)
    g5.L.g5_set_eps_to_all(1.0 / 64)
    return x, m


@pytest.mark.parametrize("nj", [0, 1, 3, 17, 100, 240, 241])
def test_results_around_the_rule(nj):
    g5 = pgb.ffi.G5()
    x, m = _set(g5, max(nj, 1))
    g5.L.g5_set_n(nj)
    for ni in (256 + 16 * nj, 257 + 16 * nj, 256 + 16 * nj):
        xi = (W.Rng(102).uniform(3 * ni).reshape(-1, 3) - 0.5).astype(np.float32).astype(np.float64)
        acc, pot = g5.calculate_force_on_x(xi)
        if nj == 0:
            assert not acc.any() and not pot.any()
            continue
        a, p = O.g5_newton(xi, np.float32((1.0 / 64) ** 2), x, m)
        # a dozen FP32 operations a pair term, as in test_g5_slots.py
        np.testing.assert_allclose(acc, a, rtol=2e-6, atol=2e-6 * np.abs(a).max())
        np.testing.assert_allclose(pot, p, rtol=2e-6)
