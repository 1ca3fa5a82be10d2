"""Trees whose nodes outgrow the construction arrays' first allocation (a quarter of the particles):
small leaves, at sizes where the arrays' own rounding leaves the three-entry array (node centres)
the smallest.  Every array equals the host builder's."""
import pytest

from conftest import gpu_available, pgb
from test_bhtree_gpu import check_same, hernquist

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


# 58.9k nodes: within the 65536 of the one-entry arrays, above the 43690 of the centres; 71.5k: above
# both
@pytest.mark.parametrize("n", [140000, 170000])
def test_small_leaves_match_the_host_builder(n):
    x, m = hernquist(n, W.SEED0 + 61)
    host = check_same(x, m, 0.75, 8, 64)
    assert len(host.cmass) > 43690
