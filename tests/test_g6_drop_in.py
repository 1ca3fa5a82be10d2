"""The drop-in GRAPE-6 call: its update and prediction run behind g6calc_firsthalf, its results and
neighbour lists come back as numbered words.

Sizes at the edges of the kernel's shapes: one chunk (127 j), one cluster of eight chunks (1024, 1535 j),
several clusters (2049, 20011), i counts of each shape, and more than the pipes of one call (72 i).  Updates: those that ride in the prediction's launch (at most 64 records), a scatter (65, 300), a
dense range, and records beyond the call's nj.  Against the FP64 oracle, tolerances as in
test_g6_gpu.py (acc and potential rms 1e-6, jerk 1e-4 per particle); a list holds every neighbour
within h (1 - 1e-6) and none outside h (1 + 1e-6) (FP32 distances, 2^-22 relative), in j order.
"""
import ctypes as C

import numpy as np
import pytest

from conftest import gpu_available, pgb
from oracle import oracle as O

pytestmark = pytest.mark.gpu
W = pgb.workloads


def _field(x, v, m, eps2):
    n = len(m)
    k = np.arange(n, dtype=np.int32)
    f = O.g6_force(x, v, k, eps2, x, v, m, k)
    return f["acc"], f["jrk"]


def _check(st, res, act, t, nj, h2):
    xp, vp = O.g6_predict(t, st.pos[:nj], st.vel[:nj], st.acc2[:nj], st.jrk6[:nj], st.tj[:nj])
    f32 = lambda a: a.astype(np.float32).astype(np.float64)   # noqa: E731  (velocities and masses travel as float)
    args = (np.float32(st.eps2), xp, f32(vp), f32(st.mass[:nj]), st.idx[:nj])
    lists = [O.g6_force(res["xi"], f32(res["vi"]), act, *args, h2=h2 * (1.0 + s) ** 2, maxlen=4096) for s in (-1e-6, 1e-6)]
    ref = lists[0]
    rms = lambda e: float(np.sqrt(np.mean(e * e)))   # noqa: E731
    rel = lambda k: np.linalg.norm(res[k] - ref[k], axis=1) / np.linalg.norm(ref[k], axis=1)   # noqa: E731
    assert rms(rel("acc")) <= 1e-6 and rel("jrk").max() <= 1e-4
    assert rms((res["pot"] - ref["pot"]) / ref["pot"]) <= 1e-6
    clear = ref["r2nn2"] / ref["r2nn"] - 1.0 > 1e-5
    assert np.array_equal(res["nnb"][clear], ref["nnb"][clear])
    for i in range(len(act)):
        rc, err, got = res["nbl"][i]
        inner, outer = (set(r["nblist"][i, :r["nbcount"][i]].tolist()) for r in lists)
        assert rc == 0 and err == 0 and len(set(got.tolist())) == len(got)
        assert inner <= set(got.tolist()) <= outer
        where = np.argsort(st.idx)[got]    # the addresses of the ids
        assert np.all(np.diff(where) > 0)


@pytest.mark.parametrize("nj,ni,nupd", [(127, 1, 3), (128, 16, 31), (1024, 7, 7), (1535, 17, 64), (2049, 32, 65),
                                        (2049, 33, 1200), (20011, 48, 300), (4100, 72, 64)])
def test_updates_and_lists(nj, ni, nupd):
    if not gpu_available():
        pytest.skip("no GPU")
    g6 = pgb.ffi.G6()
    g6.L.g6_open(0)
    rng = np.random.RandomState(nj + ni)
    st = W.hermite_state(nj, seed=nj, force_fn=_field)
    st.idx[:] = rng.permutation(nj).astype(np.int32)   # ids that are not the addresses
    h2 = np.full(ni, (2.0 * nj ** (-1.0 / 3.0)) ** 2)

    def call(t, n, act, between=None):
        """One call of the API with neighbour lists, the i at their predicted positions."""
        xp, vp = O.g6_predict(t, st.pos, st.vel, st.acc2, st.jrk6, st.tj)
        ids = st.idx[act].copy()
        xi, vi = xp[act].copy(), vp[act].copy()
        if between is None:
            r = g6.calc(t, n, xi, vi, ids, st.eps2, h2=h2[:len(act)], variant="2np")
        else:
            p = pgb.ffi.ptr
            r = dict(acc=np.zeros((len(act), 3)), jrk=np.zeros((len(act), 3)), pot=np.zeros(len(act)),
                     nnb=np.zeros(len(act), np.int32), rnnb=np.zeros(len(act), np.float32), nbl={})
            head = [0, n, len(act), p(ids, C.c_int), p(xi), p(vi)]
            out = [p(r["acc"]), p(r["jrk"]), p(r["pot"])]
            g6.L.g6_set_ti(0, t)
            g6.L.g6calc_firsthalf(*head, *out, st.eps2, p(h2))
            between()
            g6.L.g6calc_lasthalf2np(*head, st.eps2, p(h2), *out, p(r["nnb"], C.c_int), p(r["rnnb"], C.c_float))
            err = g6.L.g6_read_neighbour_list(0)
            for k in range(len(act)):
                cnt, buf = C.c_int(), np.zeros(1024, np.int32)
                rc = g6.L.g6_get_neighbour_list(0, k, 1024, C.byref(cnt), p(buf, C.c_int))
                r["nbl"][k] = (rc, err, buf[:cnt.value].copy())
        return dict(r, xi=xi, vi=vi)

    def move(addr, d):
        st.pos[addr] += d
        g6.set_j(st.pos[addr], st.vel[addr], st.acc2[addr], st.jrk6[addr], st.mass[addr], st.tj[addr], st.idx[addr],
                 addr)

    act = np.sort(rng.permutation(nj)[:ni])
    npipe = g6.L.g6_npipes()
    g6.set_j(st.pos, st.vel, st.acc2, st.jrk6, st.mass, st.tj, st.idx)
    res = call(st.t_now, nj, act)
    _check(st, res, st.idx[act], st.t_now, nj, h2)
    upd = np.sort(rng.permutation(nj)[:nupd])
    move(upd, 1e-3)
    res = call(st.t_now, nj, act)
    _check(st, res, st.idx[act], st.t_now, nj, h2)
    again = call(st.t_now, nj, act)   # nothing sent: the same bits, the same lists
    for k in ("acc", "jrk", "pot", "nnb"):
        np.testing.assert_array_equal(res[k], again[k])
    for i in range(ni):
        np.testing.assert_array_equal(res["nbl"][i][2], again["nbl"][i][2])
    # a call over fewer j, with updates beyond them, and the full one after it
    n2, act2 = nj - 3, act[act < nj - 3]
    if len(act2):
        move(np.array([1, nj - 2]), -1e-3)
        _check(st, call(st.t_now, n2, act2), st.idx[act2], st.t_now, n2, h2[:len(act2)])
        _check(st, call(st.t_now, nj, act), st.idx[act], st.t_now, nj, h2)
    # a record sent between the halves of a call counts from the next call on
    if ni <= npipe:
        before = call(st.t_now, nj, act)
        old = st.pos[upd].copy()
        mid = call(st.t_now, nj, act, between=lambda: move(upd, 2e-3))
        for k in ("acc", "jrk", "pot", "nnb"):
            np.testing.assert_array_equal(before[k], mid[k])
        assert not np.array_equal(old, st.pos[upd])
        _check(st, call(st.t_now, nj, act), st.idx[act], st.t_now, nj, h2)
