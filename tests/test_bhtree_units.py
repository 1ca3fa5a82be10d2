"""Interaction lists by work units and prefix sums of the GPU tree builder, bit for bit against the host
builder (as tests/test_bhtree_gpu.py): fewer nodes than units, the root taken as a cell or as
particles, an opening angle so wide that units start below cells taken whole, both unit counts
(ng theta^3 to both sides of 2500), and level and list sizes around a scan's tile of 2048."""
import numpy as np
import pytest

from conftest import pgb
from test_bhtree_gpu import check_same, hernquist, need_gpu  # noqa: F401

pytestmark = pytest.mark.gpu
W = pgb.workloads


@pytest.mark.parametrize("n,theta,nleaf,ncrit", [
    (2, 0.5, 1, 1), (16, 0.5, 16, 4), (17, 0.5, 16, 4), (300, 0.5, 4, 16), (300, 8.0, 4, 16), (300, 1e4, 4, 16), (2047, 2.5, 1, 8),
    (2049, 0.9, 1, 1), (9000, 1.5, 2, 8), (30000, 0.3, 4, 64), (30000, 1.2, 4, 8)])
def test_unit_lists_match_the_host_builder(n, theta, nleaf, ncrit):
    x, m = hernquist(n, W.SEED0 + n)
    check_same(x, m, theta, nleaf, ncrit)


def test_unit_lists_of_two_distant_clumps():
    a, m = hernquist(5000, W.SEED0 + 5)
    x = np.concatenate([a * 0.01 + 90.0, a * 0.01 - [90.0, -30.0, 0.0]])
    check_same(x, np.concatenate([m, m]), 0.5, 8, 64)
