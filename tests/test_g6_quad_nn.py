"""The j-paired Hermite forms that keep the best j-quad (configurations 1: two j-lanes, tiles of 128 j,
and 3) at the edges of quads, tiles and i-tiles, and exact ties of the nearest neighbour."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]
NI = [1, 2, 63, 64, 65, 128, 129, 257]
NJ = [1, 2, 3, 4, 5, 127, 128, 129, 256, 259]


def _run(cfg, items, xi, vi, idi, xj, vj, mj, idj, eps2, nn=True):
    import torch
    g6 = pgb.ffi.G6()
    dev = torch.device("cuda")
    put = lambda a: torch.from_numpy(a.view(np.uint8)).to(dev)   # noqa: E731
    di, dj = put(pgb.ffi.g6_irecords(xi, vi, idi)), put(pgb.ffi.g6_jrecords(xj, vj, mj, idj))
    out = torch.full((len(xi) * pgb.ffi.G6OUT.itemsize,), 255, dtype=torch.uint8, device=dev)
    plan = g6.plan_create(items, nn=nn)
    try:
        assert g6.L.pgb6_plan_set_config(plan, cfg) == 0
        assert g6.L.pgb6_plan_kernels(plan) == 1   # no lookup kernel
        for _ in range(2):
            g6.plan_launch(plan, di.data_ptr(), dj.data_ptr(), eps2, out.data_ptr(), 0)
        torch.cuda.synchronize()
        return out.cpu().numpy().view(pgb.ffi.G6OUT)
    finally:
        g6.plan_destroy(plan)


@pytest.mark.parametrize("cfg", [1, 3])
def test_quad_and_tile_edges(cfg):
    shapes = [(a, b) for a in NI for b in NJ]
    ni, nj = np.array([s[0] for s in shapes]), np.array([s[1] for s in shapes])
    io, jo = np.concatenate([[0], np.cumsum(ni)]), np.concatenate([[0], np.cumsum(nj)])
    rng = W.Rng(5)
    f32 = lambda a: a.astype(np.float32).astype(np.float64)   # noqa: E731
    xi, xj = rng.uniform(3 * io[-1]).reshape(-1, 3), rng.uniform(3 * jo[-1]).reshape(-1, 3)
    vi, vj = f32(rng.uniform(3 * io[-1]).reshape(-1, 3)), f32(rng.uniform(3 * jo[-1]).reshape(-1, 3))
    mj = f32(rng.uniform(jo[-1]) + 0.5)
    idj = np.arange(jo[-1], dtype=np.int32)
    # every second item's i are ids of its own j-range where it is long enough (the self mask)
    idi = np.full(io[-1], -1, np.int32)
    for q, (a, b) in enumerate(shapes):
        if q % 2 and b > 1:
            idi[io[q]:io[q + 1]] = jo[q] + np.arange(a) % b
    eps2 = 1e-4
    out = _run(cfg, np.stack([io[:-1], ni, jo[:-1], nj], 1), xi, vi, idi, xj, vj, mj, idj, eps2)
    for q in range(len(shapes)):
        o, sj = out[io[q]:io[q + 1]], slice(jo[q], jo[q + 1])
        si = slice(io[q], io[q + 1])
        ref = O.g6_force(xi[si], vi[si], idi[si], np.float32(eps2), xj[sj], vj[sj], mj[sj], idj[sj])
        # FP32 pair terms of one sign of mass: 2e-6 of the largest term's size covers the sums, 1e-5 the
        # jerk's cancelling ones
        for k, (f, tol) in enumerate((("acc", 2e-6), ("jrk", 1e-5))):
            got = np.stack([o[c] for c in (("ax", "ay", "az"), ("jx", "jy", "jz"))[k]], 1)
            np.testing.assert_allclose(got, ref[f], rtol=tol, atol=tol * max(np.abs(ref[f]).max(), 1e-30), err_msg=str(shapes[q]))
        np.testing.assert_allclose(o["pot"], ref["pot"], rtol=2e-6)
        clear = ref["r2nn2"] / ref["r2nn"] - 1.0 > 1e-5 if nj[q] > 1 else np.ones(len(o), bool)
        assert np.all((o["jadr"] >= jo[q]) & (o["jadr"] < jo[q + 1])), shapes[q]
        assert np.array_equal(idj[o["jadr"]][clear], ref["nnb"][clear]), shapes[q]


@pytest.mark.parametrize("cfg", [1, 3])
@pytest.mark.parametrize("first,second", [(0, 1), (2, 3), (3, 4), (1, 5), (100, 228), (126, 127), (9, 4000), (4097, 6000)])
def test_ties_go_to_the_smallest_address(cfg, first, second):
    """Two j at one place, the nearest of every i: in one pair, quad, lane or chunk, and across them."""
    rng = W.Rng(6)
    n = 6001
    xj = rng.uniform(3 * n).reshape(-1, 3) + 2.0
    xj[first] = xj[second] = [0.1, 0.2, 0.3]
    xi = 0.01 * rng.uniform(3 * 70).reshape(-1, 3)
    z = np.zeros((n, 3))
    out = _run(cfg, [[0, 70, 0, n]], xi, z[:70], np.full(70, -1, np.int32), xj, z, np.full(n, 1.0 / n),
               np.arange(n, dtype=np.int32), 1e-4)
    assert np.all(out["jadr"] == first)
