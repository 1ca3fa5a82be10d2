"""Unsoftened Hermite pairs at zero distance (two particles, two ids) in the j-paired configurations: the
potential is infinite and the nearest neighbour the record itself, whichever record a ragged j-tile
starts with; what pads the tile to whole j-quads adds nothing."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


@pytest.mark.parametrize("cfg", [0, 1, 2, 3, 6, 7, 8, 9])
@pytest.mark.parametrize("nj", [1, 2, 3, 5, 129, 258, 1027])
def test_every_i_on_a_record(cfg, nj):
    """i = j with other ids, eps = 0; one more i on no record, whose force is the oracle's."""
    import torch
    dev = torch.device("cuda")
    g6 = pgb.ffi.G6()
    rng = W.Rng(94 + nj)
    x = rng.uniform(3 * nj).reshape(-1, 3)
    v = (rng.uniform(3 * nj).reshape(-1, 3) - 0.5).astype(np.float32).astype(np.float64)
    m = (rng.uniform(nj) + 0.5).astype(np.float32).astype(np.float64)
    idj = np.arange(nj, dtype=np.int32)
    xi = np.concatenate([x, [[2.5, -1.25, 3.0]]])
    vi = np.concatenate([v, [[0.25, 0.5, -0.125]]])
    idi = (100000 + np.arange(nj + 1)).astype(np.int32)
    put = lambda a: torch.from_numpy(a.view(np.uint8)).to(dev)   # noqa: E731
    di, dj = put(pgb.ffi.g6_irecords(xi, vi, idi)), put(pgb.ffi.g6_jrecords(x, v, m, idj))
    out = torch.full((len(xi) * pgb.ffi.G6OUT.itemsize,), 255, dtype=torch.uint8, device=dev)
    plan = g6.plan_create([[0, nj + 1, 0, nj]], nn=True)
    try:
        assert g6.L.pgb6_plan_set_config(plan, cfg) == 0
        g6.plan_launch(plan, di.data_ptr(), dj.data_ptr(), 0.0, out.data_ptr(), 0)
        torch.cuda.synchronize()
        out = out.cpu().numpy().view(pgb.ffi.G6OUT)
    finally:
        g6.plan_destroy(plan)
    assert np.all(np.isneginf(out["pot"][:nj]))
    np.testing.assert_array_equal(out["jadr"][:nj], idj)
    ref = O.g6_force(xi[nj:], vi[nj:], idi[nj:], 0.0, x, v, m, idj)
    # the tolerances of test_g6_quad_nn.py
    for f, cs, tol in (("acc", ("ax", "ay", "az"), 2e-6), ("jrk", ("jx", "jy", "jz"), 1e-5)):
        got = np.stack([out[c][nj:] for c in cs], 1)
        np.testing.assert_allclose(got, ref[f], rtol=tol, atol=tol * np.abs(ref[f]).max())


@pytest.mark.parametrize("cfg", [1, 3, 6, 7, 8, 9])
@pytest.mark.parametrize("nj", [125, 126, 127, 253, 254, 255, 381, 511])
def test_tiles_of_a_quad_less_a_record(cfg, nj):
    """A j-tile that only its last quad keeps from being whole is a partial one: its padding is masked,
    also where no record can be one of the i."""
    import torch
    dev = torch.device("cuda")
    g6 = pgb.ffi.G6()
    rng = W.Rng(95 + nj)
    x, xi = rng.uniform(3 * nj).reshape(-1, 3), rng.uniform(3 * 70).reshape(-1, 3)
    v = (rng.uniform(3 * nj).reshape(-1, 3) - 0.5).astype(np.float32).astype(np.float64)
    vi = (rng.uniform(3 * 70).reshape(-1, 3) - 0.5).astype(np.float32).astype(np.float64)
    m = (rng.uniform(nj) + 0.5).astype(np.float32).astype(np.float64)
    idj, idi = np.arange(nj, dtype=np.int32), np.full(70, -1, np.int32)
    put = lambda a: torch.from_numpy(a.view(np.uint8)).to(dev)   # noqa: E731
    di, dj = put(pgb.ffi.g6_irecords(xi, vi, idi)), put(pgb.ffi.g6_jrecords(x, v, m, idj))
    out = torch.full((70 * pgb.ffi.G6OUT.itemsize,), 255, dtype=torch.uint8, device=dev)
    plan = g6.plan_create([[0, 70, 0, nj]], nn=True)
    try:
        assert g6.L.pgb6_plan_set_config(plan, cfg) == 0
        g6.plan_launch(plan, di.data_ptr(), dj.data_ptr(), 1e-3, out.data_ptr(), 0)
        torch.cuda.synchronize()
        out = out.cpu().numpy().view(pgb.ffi.G6OUT)
    finally:
        g6.plan_destroy(plan)
    ref = O.g6_force(xi, vi, idi, np.float32(1e-3), x, v, m, idj)
    # the tolerances of test_g6_quad_nn.py
    for f, cs, tol in (("acc", ("ax", "ay", "az"), 2e-6), ("jrk", ("jx", "jy", "jz"), 1e-5)):
        got = np.stack([out[c] for c in cs], 1)
        np.testing.assert_allclose(got, ref[f], rtol=tol, atol=tol * np.abs(ref[f]).max())
    np.testing.assert_allclose(out["pot"], ref["pot"], rtol=2e-6)
    clear = ref["r2nn2"] / ref["r2nn"] - 1.0 > 1e-5
    np.testing.assert_array_equal(out["jadr"][clear], ref["nnb"][clear])
