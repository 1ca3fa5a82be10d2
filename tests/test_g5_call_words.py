"""A GRAPE-5 call's results as numbered words (up to 4096 i) and as a copy (more): one i, i-tile edges, the
last size of the one and the first of the other; every kind; repeated calls (a word of the call before
must not be taken for one of this), a call without j-records, calls of different sizes in turn.
Against the FP64 oracle, tolerance as in test_g5_gpu.py (acc and potential rms 1e-6 relative)."""
import numpy as np
import pytest

from conftest import gpu_available, pgb

pytestmark = pytest.mark.gpu
W = pgb.workloads


def _rms(e):
    return float(np.sqrt(np.mean(e * e)))


@pytest.mark.parametrize("sym", [False, True])
@pytest.mark.parametrize("ni", [1, 63, 64, 65, 999, 4096, 4097])
def test_calls_of_every_size(ni, sym):
    if not gpu_available():
        pytest.skip("no GPU")
    g5 = pgb.ffi.G5Sym() if sym else pgb.ffi.G5()
    g5.L.g5_open()
    g = W.plummer_g5(1500, W.SEED0 + ni)
    xj, mj = g.x, g.m
    rng = np.random.RandomState(ni)
    xi = rng.normal(size=(ni, 3)).astype(np.float32).astype(np.float64)
    ej = (g.eps ** 2 * rng.uniform(0.5, 2.0, len(mj))).astype(np.float32).astype(np.float64) if sym else None
    ei = (g.eps ** 2 * rng.uniform(0.5, 2.0, ni)).astype(np.float32).astype(np.float64) if sym else None
    g5.set_xmj(0, xj, mj, ej)
    g5.L.g5_set_eps_to_all(g.eps)

    def exact(nj):
        # softened direct sum in FP64 of the float inputs
        f = lambda a: a.astype(np.float32).astype(np.float64)   # noqa: E731
        dx = f(xj[:nj])[None] - f(xi)[:, None]
        e2 = ej[None, :nj] + ei[:, None] if sym else np.float64(np.float32(g.eps ** 2))
        r2 = (dx * dx).sum(-1) + e2
        w = f(mj[:nj])[None] / (r2 * np.sqrt(r2))
        return (w[..., None] * dx).sum(1), -(f(mj[:nj])[None] / np.sqrt(r2)).sum(1)

    first = None
    for nj in (1500, 0, 700, 1500):
        g5.L.g5_set_n(nj)
        acc, pot = g5.calculate_force_on_x(xi, ei)
        if nj == 0:
            assert not acc.any() and not pot.any()
            continue
        a, p = exact(nj)
        assert _rms(np.linalg.norm(acc - a, axis=1) / np.linalg.norm(a, axis=1)) <= 1e-6
        assert _rms((pot - p) / p) <= 1e-6 or _rms((pot + p) / p) <= 1e-6
        if nj == 1500:
            if first is not None:
                np.testing.assert_array_equal(acc, first[0])
                np.testing.assert_array_equal(pot, first[1])
            first = acc, pot
        one, pone = g5.calculate_force_on_x(xi[:1], None if ei is None else ei[:1])   # another size in between
        np.testing.assert_allclose(one[0], acc[0], rtol=1e-5)
