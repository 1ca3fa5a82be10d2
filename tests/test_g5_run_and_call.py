"""g5_run, a whole call, g5_get_force, in that order: a call is g5_set_xi, g5_run and g5_get_force
(PG5/newton/libpg5/phantom_g5.c:276-300), so the pipelines hold its results afterwards, whatever way
they took to the host (words up to 4096 i, a copy from 4097 on)."""
import numpy as np
import pytest

from conftest import gpu_available, pgb

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


@pytest.mark.parametrize("kind", ["newton", "table"])
@pytest.mark.parametrize("ni", [1, 3, 65, 4096, 4097])
def test_get_force_after_a_call(ni, kind):
    g5 = pgb.ffi.G5() if kind == "newton" else pgb.ffi.G5Table()
    L, ptr = g5.L, pgb.ffi.ptr
    if kind == "table":
        g5.set_table(W.gaussian_split_force(0.05, 0.3, 0.01), 0.3, frc_bit=6)
    L.g5_open()
    rng = W.Rng(98)
    xj, m = rng.uniform(3 * 500).reshape(-1, 3) - 0.5, rng.uniform(500) + 0.5
    xj, m = np.ascontiguousarray(xj), np.ascontiguousarray(m)
    if kind == "newton":
        L.g5_set_eps_to_all(0.01)
    L.g5_set_xmj(0, 500, ptr(xj), ptr(m))
    L.g5_set_n(500)
    npipe = L.g5_get_number_of_pipelines()
    xa = np.ascontiguousarray(rng.uniform(3 * npipe).reshape(-1, 3) - 0.5)
    xb = np.ascontiguousarray(rng.uniform(3 * ni).reshape(-1, 3) - 0.5)
    acc, pot = np.zeros((ni, 3)), np.zeros(ni)
    L.g5_set_xi(npipe, ptr(xa))
    L.g5_run()
    L.g5_calculate_force_on_x(ptr(xb), ptr(acc), ptr(pot), ni)
    n = min(ni, npipe)
    a, p = np.zeros((n, 3)), np.ones(n)
    L.g5_get_force(n, ptr(a), ptr(p))
    np.testing.assert_array_equal(a, acc[:n])
    np.testing.assert_array_equal(p, pot[:n])
    # and a run after it has its own again, the same bits as a call for them
    L.g5_set_xi(npipe, ptr(xa))
    L.g5_run()
    a, p = np.zeros((npipe, 3)), np.ones(npipe)
    L.g5_get_force(npipe, ptr(a), ptr(p))
    want, wpot = np.zeros((npipe, 3)), np.zeros(npipe)
    L.g5_calculate_force_on_x(ptr(xa), ptr(want), ptr(wpot), npipe)
    np.testing.assert_array_equal(a, want)
    np.testing.assert_array_equal(p, wpot)
