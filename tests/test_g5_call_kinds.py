"""GRAPE-5 calls at the sizes where the results' way to the host changes (words up to 4096 i, a copy from
4097 on; test_g5_call_words.py covers the rest of those sizes), for the kinds and signs the libraries
return: point masses +sum m/r, symmetric softening the same, quadrupole cells -sum (phi_p + phi_q), the
table library no potential."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _f32(a):
    return np.asarray(a).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("ni", [1, 64, 65, 4096, 4097])
@pytest.mark.parametrize("kind", ["newton", "symmetric", "quad", "table"])
def test_every_kind_and_its_sign(kind, ni):
    rng = W.Rng(97 + ni)
    nj, eps = 777, 1.0 / 64
    xj, xi = _f32(rng.uniform(3 * nj).reshape(-1, 3) - 0.5), _f32(rng.uniform(3 * ni).reshape(-1, 3) - 0.5)
    m = _f32((rng.uniform(nj) + 0.5) / nj)
    if kind == "quad":
        g5 = pgb.ffi.G5()
        g5.L.g5_open()
        q = _f32(1e-5 * (rng.uniform(6 * nj).reshape(-1, 6) - 0.5))
        q[:, 5] = _f32(-(q[:, 0] + q[:, 3]))
        acc, pot = g5.quad_force(eps, xi, xj, m, q)
        a, p = O.g5_quad(xi, np.float32(eps * eps), xj, m, q)
        p = -p
    elif kind == "table":
        g5 = pgb.ffi.G5Table()
        g5.set_table(W.gaussian_split_force(0.05, 0.3, 0.01), 0.3, frc_bit=6)
        table, xs = g5.table()
        acc, pot = g5.force(xj, m, xi)
        # the library scales the i in FP64 and rounds once, the j in FP32 (as test_g5table.py has it)
        xjs = (xj.astype(np.float32) * np.float32(xs)).astype(np.float64) / xs
        a, p = O.g5_table(_f32(xi * xs) / xs, xjs, m, table, 4, 6, xs), np.zeros(ni)
    else:
        g5 = pgb.ffi.G5Sym() if kind == "symmetric" else pgb.ffi.G5()
        g5.L.g5_open()
        ej = _f32(eps ** 2 * (0.5 + rng.uniform(nj))) if kind == "symmetric" else None
        g5.set_xmj(0, xj, m, ej)
        g5.L.g5_set_n(nj)
        g5.L.g5_set_eps_to_all(eps)
        acc, pot = g5.calculate_force_on_x(xi)
        a, p = O.g5_newton(xi, np.float32(eps * eps), xj, m, ej) if ej is not None else O.g5_newton(xi, np.float32(eps * eps), xj, m)
    # tolerances of test_g5_slots.py: a dozen FP32 operations a pair term, the table's steep entries more
    tol = 8e-6 if kind == "table" else 2e-6
    np.testing.assert_allclose(acc, a, rtol=tol, atol=tol * np.abs(a).max())
    if kind == "quad":
        assert np.all(pot < 0)
    np.testing.assert_allclose(pot, p, rtol=2e-6, atol=2e-6 * np.abs(p).max())
