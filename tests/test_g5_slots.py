"""The 64-thread PG5 configuration (16 i-slots over four j-lanes, one to four i per thread, j-tiles of
256 records) at the sizes where its task shapes and tiles change, against the FP64 oracle."""
import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

W = pgb.workloads
NI = [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 200]
NJ = [0, 1, 3, 4, 5, 255, 256, 257, 511, 1030]
CFG_64 = 7

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no GPU")]


def _launch(lib, kind, items, ip, jp, aux, jidx):
    import torch
    dev = torch.device("cuda")
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)   # noqa: E731
    di, dj = put(ip), put(jp)
    da = put(aux) if aux is not None else None
    dx = put(jidx) if jidx is not None else None
    out = torch.full((len(ip), 4), np.nan, dtype=torch.float64, device=dev)
    plan = lib.plan_create(items) if kind is None else lib.plan_create(kind, items)
    try:
        assert lib.L.pgb5_plan_set_config(plan, CFG_64) == 0
        pa = da.data_ptr() if da is not None else None
        s = torch.cuda.current_stream().cuda_stream
        for _ in range(2):   # the second launch finds the counters as the first left them
            if dx is not None:
                rc = lib.L.pgb5_plan_launch_indexed(plan, di.data_ptr(), dj.data_ptr(), pa, dx.data_ptr(), out.data_ptr(), s)
            else:
                rc = lib.L.pgb5_plan_launch(plan, di.data_ptr(), dj.data_ptr(), pa, out.data_ptr(), s)
            assert rc == 0
        torch.cuda.synchronize()
        return out.cpu().numpy()
    finally:
        lib.plan_destroy(plan)


@pytest.mark.parametrize("indexed", [False, True])
@pytest.mark.parametrize("kind", ["newton", "symmetric", "quad", "table"])
def test_task_and_tile_edges(kind, indexed):
    rng = W.Rng(77)
    shapes = [(a, b) for a in NI for b in NJ]
    ni, nj = np.array([s[0] for s in shapes]), np.array([s[1] for s in shapes])
    io, jo = np.concatenate([[0], np.cumsum(ni)]), np.concatenate([[0], np.cumsum(nj)])
    items = np.stack([io[:-1], ni, jo[:-1], nj], 1)
    f32 = lambda a: a.astype(np.float32)   # noqa: E731
    xi, xj = f32(rng.uniform(3 * io[-1]).reshape(-1, 3) - 0.5), f32(rng.uniform(3 * jo[-1]).reshape(-1, 3) - 0.5)
    mj = f32((rng.uniform(jo[-1]) + 0.5) / 1000.0)
    eps2 = np.float32(1e-3)
    e2j = f32(1e-3 * (0.5 + rng.uniform(jo[-1])))
    qj = f32(1e-5 * (rng.uniform(6 * jo[-1]).reshape(-1, 6) - 0.5))
    qj[:, 5] = -(qj[:, 0] + qj[:, 3])
    aux, xs = None, 1.0
    if kind == "table":
        lib, k = pgb.ffi.G5Table(), None
        lib.set_table(W.gaussian_split_force(0.05, 0.3, 0.01), 0.3, frc_bit=6)
        table, xs = lib.table()
    elif kind == "symmetric":
        lib = pgb.ffi.G5Sym()
        k = lib.SYMMETRIC_KIND
        aux = np.zeros((len(e2j), 4), np.float32)
        aux[:, 0] = e2j
    else:
        lib = pgb.ffi.G5()
        k = lib.QUAD if kind == "quad" else lib.NEWTON
        if kind == "quad":
            aux = np.zeros((len(qj), 8), np.float32)
            aux[:, :6] = qj
    ip = np.concatenate([f32(xi * np.float32(xs)), np.full((len(xi), 1), eps2, np.float32)], 1)
    jp = np.concatenate([f32(xj * np.float32(xs)), mj[:, None]], 1)
    jidx = None
    src_j, src_a = jp, aux
    if indexed:
        perm = rng.permutation(len(jp))
        jidx = np.empty(len(jp), np.int32)
        jidx[perm] = np.arange(len(jp))          # record k of the lists is row jidx[k] of the arrays
        jidx = np.ascontiguousarray(jidx)
        src_j = np.empty_like(jp)
        src_j[jidx] = jp
        if aux is not None:
            src_a = np.empty_like(aux)
            src_a[jidx] = aux
    out = _launch(lib, k, items, ip, src_j, src_a, jidx)
    d = np.float64
    for q, (a, b) in enumerate(shapes):
        si, sj = slice(io[q], io[q + 1]), slice(jo[q], jo[q + 1])
        if b == 0:
            assert np.all(out[si] == 0)
            continue
        po = None
        if kind == "table":
            ao = O.g5_table(ip[si, :3].astype(d) / xs, jp[sj, :3].astype(d) / xs, mj[sj].astype(d), table, 4, 6, xs)
        elif kind == "quad":
            ao, po = O.g5_quad(xi[si].astype(d), eps2, xj[sj].astype(d), mj[sj].astype(d), qj[sj].astype(d))
            po = po * np.sign(po[0] / out[si, 3][0])   # the sign conventions of the two are tested elsewhere
        elif kind == "symmetric":
            ao, po = O.g5_newton(xi[si].astype(d), eps2, xj[sj].astype(d), mj[sj].astype(d), e2j[sj].astype(d))
            po = -po
        else:
            ao, po = O.g5_newton(xi[si].astype(d), eps2, xj[sj].astype(d), mj[sj].astype(d))
            po = -po
        # a pair term is a dozen FP32 operations (6e-8 each), its coordinates' difference one more of
        # the box's size: 2e-6 of the largest force; the table's steep entries four times that
        tol = 8e-6 if kind == "table" else 2e-6
        np.testing.assert_allclose(out[si, :3], ao, rtol=tol, atol=tol * max(np.abs(ao).max(), 1e-30))
        if po is not None:
            np.testing.assert_allclose(out[si, 3], po, rtol=2e-6, atol=2e-6 * np.abs(po).max())


def test_one_split_item_equals_the_oracle():
    """One item of many j: its range is split over tasks whose partial sums are reduced."""
    rng = W.Rng(78)
    g5 = pgb.ffi.G5()
    x = (rng.uniform(3 * 20000).reshape(-1, 3) - 0.5).astype(np.float32)
    m = np.full((20000, 1), 1.0 / 20000, np.float32)
    ip = np.concatenate([x, np.full((20000, 1), 1e-4, np.float32)], 1)[:77]
    out = _launch(g5, g5.NEWTON, [[0, 77, 0, 20000]], ip, np.concatenate([x, m], 1), None, None)
    ao, po = O.g5_newton(x[:77].astype(np.float64), np.float32(1e-4), x.astype(np.float64), m[:, 0].astype(np.float64))
    np.testing.assert_allclose(out[:, :3], ao, rtol=2e-6, atol=2e-6 * np.abs(ao).max())
    np.testing.assert_allclose(-out[:, 3], po, rtol=2e-6)


def test_unsoftened_coincident_record_in_a_ragged_tile():
    """eps = 0 and an i-particle on the tile's first record: the potential is infinite (the padding
    of the ragged tile adds nothing to it), the other particle's force is finite."""
    g5 = pgb.ffi.G5()
    jp = np.array([[0, 0, 0, 1], [1, 0, 0, 1], [0, 2, 0, 1]], np.float32)
    ip = np.array([[0, 0, 0, 0], [3, 0, 0, 0]], np.float32)
    out = _launch(g5, g5.NEWTON, [[0, 2, 0, 3]], ip, jp, None, None)
    assert np.isneginf(out[0, 3])
    assert np.all(np.isfinite(out[1]))
