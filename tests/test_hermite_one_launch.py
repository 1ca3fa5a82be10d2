"""Many block steps in one launch of the step kernel against the same steps launched one by one.

Within one launch a step starts from what the step before published (segment records kept for a few
steps, lists of active particles, chunk sums and flags tagged with the step's number, times kept
in shared memory); a launch of one step reads everything afresh from the state, and is itself
replayed by the oracle in test_hermite_sizes.py.  The two must agree in every step and count and in
every bit of the state.  n = 257: two segments, one of one particle; 5001: middle decompositions;
16384: large ones and halved tail tasks; 160001: more segments than two per CTA.  Every interval
crosses a reset of the times, and the single launch is repeated, since what it could get wrong
would depend on which CTA comes first.
"""
import numpy as np
import pytest

from conftest import gpu_available, pgb

pytestmark = pytest.mark.gpu
W = pgb.workloads


@pytest.mark.parametrize("n,dtmax,tend,repeats", [(257, 0.125, 0.3125, 6), (5001, 0.125, 0.1875, 4),
                                                  (16384, 0.03125, 0.046875, 4), (160001, 1 / 1024, 4.5 / 1024, 3)])
def test_one_launch_equals_single_steps(n, dtmax, tend, repeats):
    if not gpu_available():
        pytest.skip("no GPU")
    g6 = pgb.ffi.G6()
    g6.L.g6_open(0)
    x, v, m, _ = W.plummer_hermite(n, W.SEED0 + n)
    make = lambda: pgb.ffi.Hermite(g6, m, x, v, 1.0 / 64 ** 2, 0.2, 0.01, dtmax)   # noqa: E731
    H = make()
    try:
        steps = 0
        while H.time < tend:
            H.step()
            steps += 1
        want, counts, time, last = H.get(), H.counts(), H.time, H.last_step()
    finally:
        H.close()
    assert steps > 8 and time > dtmax
    for r in range(repeats):
        H = make()
        try:
            p, b = H.advance(tend)
            assert b == steps and H.counts() == counts and H.time == time
            got = H.get()
            for k in want:
                np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k}, launch {r}")
            for a, w in zip(H.last_step(), last):
                np.testing.assert_array_equal(a, w)
        finally:
            H.close()
