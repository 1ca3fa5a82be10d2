"""The framework's work, as cases that can be timed and checked.

Each case is one pass that a simulation code has the libraries do, through their public entry
points (the C ABI as ``phantom-grape_b200/ffi.py`` and ``workloads.py`` bind it):

* ``call``      a GRAPE-6 force call of a block step, host arrays (g6_set_ti, g6calc_firsthalf,
                g6calc_lasthalf*), at most 48 active particles as the API has pipes
* ``block``     a large block step on the device (pgb6_predict + pgb6_plan_launch)
* ``clusters``  many independent Hermite systems in one launch (pgb6_plan_launch)
* ``direct``    a GRAPE-5 direct sum from host arrays (g5_set_xmj .. g5_calculate_force_on_x)
* ``treepm``    the short-range part of a TreePM step (pgb5_plan_launch of the table library)
* ``tree``      a Barnes-Hut step: tree, lists and both force launches (pgbt_*, pgb5_plan_*)
* ``integrate`` an interval of the device's Hermite block-time-step integrator (pgb6_hermite_*)

The batched and GRAPE-5 forces come back in float32, as a code keeps them beside its float32
particles: the records' FP64 words hold sums of FP32 pair terms.  The GRAPE-6 calls' FP64 arrays
and the integrator's FP64 state come back as they are.
"""
import ctypes as C
import importlib
import math

import numpy as np
import torch

pgb = importlib.import_module("phantom-grape_b200")
ffi, workloads = pgb.ffi, pgb.workloads

_LIBS = {}


def _lib(cls):
    """The one binding of a library that a program holds."""
    if cls not in _LIBS:
        _LIBS[cls] = cls()
    return _LIBS[cls]


class _Plan:
    """A plan handle, given back with the state that holds it."""

    def __init__(self, lib, h):
        self.lib, self.h = lib, h

    def __del__(self):
        self.lib.plan_destroy(self.h)


# ---- the cases ------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: a handful of particles of a small system, as most block steps are; the
        # particles advanced by the step before are sent again first
        dict(name="call 7 of 1024", kind="call", nj=1024, ni=7, variant="2p", resend=True),
        # a full call of a large system: 48 particles, the API's pipes
        dict(name="call 48 of 65536", kind="call", nj=65536, ni=48, variant="2p", resend=False),
        # the same with neighbour lists (an Ahmad-Cohen or collision code), odd sizes
        dict(name="call 33 of 20011 lists", kind="call", nj=20011, ni=33, variant="2np", resend=False),
        # a middle block step, an odd number of active particles
        dict(name="block 777 of 16384", kind="block", nj=16384, ni=777, nn=True, f64=False, tune=False),
        # the largest block step: every particle of the Hermite workload
        dict(name="block 65536 of 65536", kind="block", nj=65536, ni=65536, nn=True, f64=False, tune=False),
        # an ensemble of small clusters (the benchmark's size range, fewer of them), tuned once
        dict(name="clusters 96", kind="clusters", ncl=96, nmin=256, nmax=16384, tune=True),
        # a small direct sum, odd size: the latency of the host path
        dict(name="direct 999", kind="direct", n=999, sym=False),
        # the benchmark's direct sum
        dict(name="direct 16384", kind="direct", n=16384, sym=False),
        # a small TreePM step: odd size, the reference's 512-entry table, the plan as it is created
        dict(name="treepm 40003", kind="treepm", n=40003, group=200, bits=5, tune=False),
        # the benchmark's TreePM step, tuned once
        dict(name="treepm 1048576", kind="treepm", n=1 << 20, group=256, bits=6, tune=True),
        # a Barnes-Hut step from particles in host memory, plans tuned once
        dict(name="tree 1048576", kind="tree", n=1 << 20, theta=0.5, nleaf=16, ncrit=256, tune=True),
        # one interval of the integrator, from initial conditions to the state
        dict(name="integrate 16384", kind="integrate", n=16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "block", "clusters", "direct", "treepm", "tree", "integrate"])
    if kind == "call":
        ni = rng.randint(1, 48)
        return dict(kind=kind, nj=_log_int(rng, 512, 65536), ni=ni, variant=rng.choice(["plain", "2", "2p", "2p", "2np"]),
                    resend=ni <= 8)
    if kind == "block":
        nj = _log_int(rng, 2048, 65536)
        return dict(kind=kind, nj=nj, ni=_log_int(rng, 16, nj), nn=rng.random() < 0.8, f64=rng.random() < 0.15,
                    tune=rng.random() < 0.3)
    if kind == "clusters":
        return dict(kind=kind, ncl=_log_int(rng, 16, 96), nmin=rng.randint(64, 512), nmax=_log_int(rng, 2048, 16384),
                    tune=rng.random() < 0.5)
    if kind == "direct":
        return dict(kind=kind, n=_log_int(rng, 500, 20000), sym=rng.random() < 0.25)
    if kind == "treepm":
        return dict(kind=kind, n=_log_int(rng, 30000, 1 << 20), group=rng.randint(190, 400), bits=rng.choice([5, 6]),
                    tune=rng.random() < 0.5)
    if kind == "tree":
        return dict(kind=kind, n=_log_int(rng, 16384, 1 << 20), theta=rng.choice([0.5, 0.6, 0.75]),
                    nleaf=rng.choice([8, 16]), ncrit=rng.choice([64, 128, 256]), tune=rng.random() < 0.5)
    return dict(kind=kind, n=_log_int(rng, 512, 16384))


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return _KINDS[state["kind"]][1](state)


def exact(case, seed):
    return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


# flops of a pair as the reference counts them: 38 for a GRAPE-5 pair, 60 for a Hermite pair and
# for a quadrupole cell
_FLOP5, _FLOP6 = 38, 60
_DEV = "cuda"


def _bytes(rec):
    """A numpy record array as bytes on the device."""
    return torch.from_numpy(rec.view(np.uint8).reshape(len(rec), -1)).to(_DEV)


def _f64(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_DEV)


# ---- plain 64-bit forces --------------------------------------------------------------------

def _hermite_exact(xi, vi, idi, xj, vj, mj, idj, eps2):
    """acc, jerk and pot of the i-particles, the pair with equal ids left out (64-bit tensors)."""
    acc, jrk, pot = torch.empty_like(xi), torch.empty_like(xi), torch.empty_like(xi[:, 0])
    step = max(1, (1 << 24) // len(xj))
    for a in range(0, len(xi), step):
        b = slice(a, a + step)
        dx = xj[None] - xi[b, None]
        dv = vj[None] - vi[b, None]
        r2 = (dx * dx).sum(-1) + eps2
        w = torch.where(idi[b, None] == idj[None], 0.0, mj[None] / r2.sqrt())
        pot[b] = -w.sum(1)
        w = w / r2
        acc[b] = (w[..., None] * dx).sum(1)
        w2 = -3.0 * w * (dx * dv).sum(-1) / r2
        jrk[b] = (w[..., None] * dv + w2[..., None] * dx).sum(1)
    return acc, jrk, pot


def _gravity_exact(xi, xj, mj, eps2):
    """acc and sum m/r of the i-particles (64-bit tensors); eps2: a number, or one per j."""
    acc, pot = torch.empty_like(xi), torch.empty_like(xi[:, 0])
    step = max(1, (1 << 25) // len(xj))
    for a in range(0, len(xi), step):
        b = slice(a, a + step)
        dx = xj[None] - xi[b, None]
        w = mj[None] / ((dx * dx).sum(-1) + eps2).sqrt()
        pot[b] = w.sum(1)
        w = w / ((dx * dx).sum(-1) + eps2)
        acc[b] = (w[..., None] * dx).sum(1)
    return acc, pot


# ---- call: GRAPE-6 force calls with host arrays ---------------------------------------------

_LISTLEN = 1024


def _plummer_field(x, v, m, eps2):
    """The smooth model's acceleration and jerk: the predictor's terms have their usual sizes."""
    w = 1.0 + (x * x).sum(1, keepdims=True)
    a = -x * w ** -1.5
    return a, -v * w ** -1.5 + 3.0 * (x * v).sum(1, keepdims=True) * x * w ** -2.5


def _call_inputs(case, seed):
    n, ni = case["nj"], case["ni"]
    st = workloads.hermite_state(n, seed=seed, force_fn=_plummer_field)
    act = np.sort(np.random.RandomState(seed % (1 << 32)).permutation(n)[:ni]).astype(np.int32)
    dt = (st.t_now - st.tj)[:, None]
    xp = st.pos + st.vel * dt + st.acc2 * dt * dt + st.jrk6 * dt ** 3
    vp = st.vel + 2.0 * st.acc2 * dt + 3.0 * st.jrk6 * dt * dt
    return st, act, xp, vp


def _call_prepare(case, seed):
    g6 = _lib(ffi.G6)
    g6.L.g6_open(0)
    st, act, xp, vp = _call_inputs(case, seed)
    g6.set_j(st.pos, st.vel, st.acc2, st.jrk6, st.mass, st.tj, st.idx)   # the board's one j-memory
    ni = case["ni"]
    h2 = np.full(ni, (2.0 * case["nj"] ** (-1.0 / 3.0)) ** 2)   # ~ tens of neighbours near the centre
    a = dict(idi=act, xi=xp[act].copy(), vi=vp[act].copy(), h2=h2, acc=np.zeros((ni, 3)), jrk=np.zeros((ni, 3)),
             pot=np.zeros(ni), nnb=np.zeros(ni, np.int32), rnnb=np.zeros(ni, np.float32),
             count=np.zeros(ni, np.int32), lists=np.full((ni, _LISTLEN), -1, np.int32))
    p = lambda k, t=C.c_double: ffi.ptr(a[k], t)   # noqa: E731
    head = [0, case["nj"], ni, p("idi", C.c_int), p("xi"), p("vi")]
    v = case["variant"]
    last = head + [st.eps2, p("h2"), p("acc"), p("jrk"), p("pot")]
    if v != "plain":
        last.append(p("nnb", C.c_int))
    if v.endswith("p"):
        last.append(p("rnnb", C.c_float))
    again = []
    if case["resend"]:
        a["snp"] = np.zeros(3)
        a["j"] = [[np.ascontiguousarray(f[i]) for f in (st.jrk6, st.acc2, st.vel, st.pos)] for i in act]
        again = [[0, int(i), int(i), float(st.tj[i]), 0.0, float(st.mass[i]), ffi.ptr(a["snp"])] +
                 [ffi.ptr(f) for f in fs] for i, fs in zip(act, a["j"])]
    rows = [(k, ffi.ptr(a["count"][k:k + 1], C.c_int), ffi.ptr(a["lists"][k], C.c_int)) for k in range(ni)]
    return dict(kind="call", L=g6.L, arrays=a, variant=v, t=st.t_now, again=again, rows=rows,
                first=head + [p("acc"), p("jrk"), p("pot"), st.eps2, p("h2")], last=last,
                lasthalf=getattr(g6.L, "g6calc_lasthalf" + ("" if v == "plain" else v)))


def _call_run(s):
    L, a, v = s["L"], s["arrays"], s["variant"]
    for args in s["again"]:
        L.g6_set_j_particle(*args)
    L.g6_set_ti(0, s["t"])
    L.g6calc_firsthalf(*s["first"])
    s["lasthalf"](*s["last"])
    out = dict(acc=a["acc"], jrk=a["jrk"], pot=a["pot"])
    if v != "plain":
        out["nnb"] = a["nnb"]
    if v.endswith("p"):
        out["rnnb"] = a["rnnb"]
    if v == "2np":
        out["overflow"] = L.g6_read_neighbour_list(0)
        for k, c, row in s["rows"]:
            L.g6_get_neighbour_list(0, k, _LISTLEN, c, row)
        out["count"], out["lists"] = a["count"], a["lists"]
    return out


def _call_exact(case, seed):
    st, act, xp, vp = _call_inputs(case, seed)
    ids = torch.as_tensor(st.idx, device=_DEV)
    x, v, i = _f64(xp), _f64(vp), torch.as_tensor(act, device=_DEV).long()
    acc, jrk, pot = _hermite_exact(x[i], v[i], ids[i], x, v, _f64(st.mass), ids, st.eps2)
    return dict(acc=acc, jrk=jrk, pot=pot)


def _call_work(case):
    nj, ni = case["nj"], case["ni"]
    # the j-records read once (pos, vel, acc, jerk, mass, time, id), the i in and the results out
    return dict(bytes=nj * 116 + ni * (52 + 72), flops=_FLOP6 * nj * ni)


# ---- block: a block step on the device ------------------------------------------------------

def _block_inputs(case, seed):
    st, act, xp, vp = _call_inputs(case, seed)
    rec = np.zeros(len(st.mass), ffi.G6PTCL)
    rec["pos"], rec["vel"], rec["acc2"], rec["jrk6"] = st.pos, st.vel, st.acc2, st.jrk6
    rec["mass"], rec["tim"], rec["idx"] = st.mass, st.tj, st.idx
    return st, rec, ffi.g6_irecords(xp[act], vp[act], act, ff=not case["f64"])


def _hermite_outputs(out, nn):
    """acc, jerk and potential in float32, and the nearest neighbour's key and j address."""
    r = dict(force=out.view(torch.float64)[:, :7].float())
    if nn:
        r["key"], r["nearest"] = out.view(torch.float32)[:, 14], out.view(torch.int32)[:, 15]
    return r


def _block_prepare(case, seed):
    g6 = _lib(ffi.G6)
    st, jrec, irec = _block_inputs(case, seed)
    nj, ni = case["nj"], case["ni"]
    s = dict(kind="block", g6=g6, nj=nj, nn=case["nn"], t=st.t_now, eps2=st.eps2, flags=g6.POS_F64 if case["f64"] else 0,
             ptcl=_bytes(jrec), ipart=_bytes(irec), pred=torch.empty((nj, g6.sizes["predj"]), dtype=torch.uint8, device=_DEV),
             out=torch.zeros((ni, g6.sizes["out"]), dtype=torch.uint8, device=_DEV),
             plan=_Plan(g6, g6.plan_create([[0, ni, 0, nj]], nn=case["nn"], f64=case["f64"])))
    if case["tune"]:
        g6.L.pgb6_predict(s["ptcl"].data_ptr(), nj, s["t"], s["pred"].data_ptr(), s["flags"], None)
        g6.plan_tune(s["plan"].h, s["ipart"].data_ptr(), s["pred"].data_ptr(), s["eps2"], s["out"].data_ptr())
    return s


def _block_run(s):
    g6 = s["g6"]
    g6.L.pgb6_predict(s["ptcl"].data_ptr(), s["nj"], s["t"], s["pred"].data_ptr(), s["flags"], None)
    g6.plan_launch(s["plan"].h, s["ipart"].data_ptr(), s["pred"].data_ptr(), s["eps2"], s["out"].data_ptr())
    return _hermite_outputs(s["out"], s["nn"])


def _block_exact(case, seed):
    r = _call_exact(case, seed)
    return dict(force=torch.cat([r["acc"], r["jrk"], r["pot"][:, None]], 1))


def _block_work(case):
    nj, ni = case["nj"], case["ni"]
    return dict(bytes=nj * 116 + ni * (48 + 64), flops=_FLOP6 * nj * ni)


# ---- clusters: independent systems in one launch --------------------------------------------

def _clusters_sizes(case):
    """The clusters' particle counts, log-uniform: a property of the ensemble, not of its particles."""
    u = np.random.RandomState(case["ncl"]).uniform(size=case["ncl"])
    return np.rint(case["nmin"] * (case["nmax"] / case["nmin"]) ** u).astype(np.int64)


def _clusters_inputs(case, seed):
    sizes = _clusters_sizes(case)
    offs = np.concatenate([[0], np.cumsum(sizes)])
    x, v, m = np.empty((offs[-1], 3)), np.empty((offs[-1], 3)), np.empty(offs[-1])
    for c in range(case["ncl"]):
        s = slice(offs[c], offs[c + 1])
        x[s], v[s], m[s], _ = workloads.plummer_hermite(int(sizes[c]), seed * 7919 + c)
        x[s] += 64.0 * np.array([c % 8, c // 8 % 8, c // 64])
    return workloads.ClusterSet(offsets=offs, pos=x, vel=v, mass=m, eps2=1e-8, sizes=sizes)


def _clusters_prepare(case, seed):
    g6 = _lib(ffi.G6)
    cs = _clusters_inputs(case, seed)
    ids = np.arange(len(cs.mass), dtype=np.int32)
    items = np.stack([cs.offsets[:-1], cs.sizes, cs.offsets[:-1], cs.sizes], 1)
    s = dict(kind="clusters", g6=g6, eps2=cs.eps2, ipart=_bytes(ffi.g6_irecords(cs.pos, cs.vel, ids)),
             pred=_bytes(ffi.g6_jrecords(cs.pos, cs.vel, cs.mass, ids)),
             out=torch.zeros((len(ids), g6.sizes["out"]), dtype=torch.uint8, device=_DEV), plan=_Plan(g6, g6.plan_create(items)))
    if case["tune"]:
        g6.plan_tune(s["plan"].h, s["ipart"].data_ptr(), s["pred"].data_ptr(), s["eps2"], s["out"].data_ptr())
    return s


def _clusters_run(s):
    s["g6"].plan_launch(s["plan"].h, s["ipart"].data_ptr(), s["pred"].data_ptr(), s["eps2"], s["out"].data_ptr())
    return _hermite_outputs(s["out"], True)


def _clusters_exact(case, seed):
    cs = _clusters_inputs(case, seed)
    x, v, m = _f64(cs.pos), _f64(cs.vel), _f64(cs.mass)
    ids = torch.arange(len(m), device=_DEV)
    rows = []
    for a, b in zip(cs.offsets[:-1], cs.offsets[1:]):
        c = slice(int(a), int(b))
        acc, jrk, pot = _hermite_exact(x[c], v[c], ids[c], x[c], v[c], m[c], ids[c], cs.eps2)
        rows.append(torch.cat([acc, jrk, pot[:, None]], 1))
    return dict(force=torch.cat(rows))


def _clusters_work(case):
    n = _clusters_sizes(case).astype(float)
    return dict(bytes=float(n.sum()) * (48 + 48 + 64), flops=float((n * n).sum()) * _FLOP6)


# ---- direct: a GRAPE-5 direct sum from host arrays ------------------------------------------

def _direct_inputs(case, seed):
    g = workloads.plummer_g5(case["n"], seed)
    rng = np.random.RandomState(seed % (1 << 32))
    epsj2 = (g.eps * rng.uniform(0.5, 2.0, case["n"])) ** 2   # the symmetric form: a softening per particle
    return g, epsj2.astype(np.float32).astype(np.float64)


def _direct_prepare(case, seed):
    g5 = _lib(ffi.G5Sym if case["sym"] else ffi.G5)
    g5.L.g5_open()
    g, epsj2 = _direct_inputs(case, seed)
    return dict(kind="direct", g5=g5, x=g.x, m=g.m, eps=g.eps, epsj2=epsj2 if case["sym"] else None)


def _direct_run(s):
    g5, x, m = s["g5"], s["x"], s["m"]
    g5.set_xmj(0, x, m, s["epsj2"])
    g5.L.g5_set_eps_to_all(s["eps"])
    g5.L.g5_set_n(len(m))
    acc, pot = g5.calculate_force_on_x(x, s["epsj2"])
    return dict(acc=acc.astype(np.float32), pot=pot.astype(np.float32))


def _direct_exact(case, seed):
    g, epsj2 = _direct_inputs(case, seed)
    x, e = _f64(g.x), _f64(epsj2)
    if not case["sym"]:
        acc, pot = _gravity_exact(x, x, _f64(g.m), g.eps ** 2)
    else:
        acc, pot = torch.empty_like(x), torch.empty_like(e)
        for a in range(0, len(x), 512):
            b = slice(a, a + 512)
            dx = x[None] - x[b, None]
            r2 = (dx * dx).sum(-1) + e[None] + e[b, None]
            w = _f64(g.m)[None] / r2.sqrt()
            pot[b] = w.sum(1)
            acc[b] = ((w / r2)[..., None] * dx).sum(1)
    return dict(acc=acc, pot=pot)


def _direct_work(case):
    n = case["n"]
    return dict(bytes=n * (32 + 24 + 32), flops=_FLOP5 * n * n)


# ---- treepm: the short-range forces of a TreePM step ----------------------------------------

def _treepm_inputs(case, seed):
    """Uniform particles in the periodic unit box, sorted into nb^3 blocks (the i-groups); a
    group's j-list holds every particle or periodic image within rcut of its block."""
    n = case["n"]
    rs = 1.25 / n ** (1.0 / 3.0)
    rcut = 4.5 * rs
    nb = max(3, min(round((n / case["group"]) ** (1.0 / 3.0)), int(1.0 / rcut)))
    gen = torch.Generator(_DEV).manual_seed(seed)
    x = torch.rand((n, 3), generator=gen, device=_DEV)
    blk = (x * nb).long().clamp_(max=nb - 1)
    bid = (blk[:, 0] * nb + blk[:, 1]) * nb + blk[:, 2]
    order = torch.argsort(bid, stable=True)
    x, blk, bid = x[order], blk[order], bid[order]
    group, xj = [], []
    for o in range(27):
        off = torch.tensor([o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1], device=_DEV)
        to = blk + off                                # the block whose list this particle may enter
        wrap = torch.div(to, nb, rounding_mode="floor")
        y = x - wrap                                  # its image next to that block
        to = to - wrap * nb
        lo = to.float() / nb
        d = torch.maximum(lo - y, y - (lo + 1.0 / nb)).clamp_(min=0)
        keep = (d * d).sum(1) <= rcut * rcut
        group.append(((to[:, 0] * nb + to[:, 1]) * nb + to[:, 2])[keep])
        xj.append(y[keep])
    group, xj = torch.cat(group), torch.cat(xj)
    xj = xj[torch.argsort(group, stable=True)]
    ni = torch.bincount(bid, minlength=nb ** 3).cpu().numpy()
    nj = torch.bincount(group, minlength=nb ** 3).cpu().numpy()
    items = np.stack([np.cumsum(ni) - ni, ni, np.cumsum(nj) - nj, nj], 1).astype(np.int32)
    return x, xj, items, np.float32(1.0 / n), rs, rcut, 0.1 / n ** (1.0 / 3.0)


def _treepm_prepare(case, seed):
    tab = _lib(ffi.G5Table)
    x, xj, items, m, rs, rcut, eps = _treepm_inputs(case, seed)
    tab.set_table(workloads.gaussian_split_force(rs, rcut, eps), rcut, frc_bit=case["bits"])
    _, xs = tab.table()
    ipos = torch.zeros((len(x), 4), device=_DEV)
    ipos[:, :3] = (x.double() * xs).float()
    jpos = torch.full((len(xj), 4), float(m), device=_DEV)
    jpos[:, :3] = (xj.double() * xs).float()
    s = dict(kind="treepm", tab=tab, ipos=ipos, jpos=jpos, plan=_Plan(tab, tab.plan_create(items)),
             out=torch.zeros((len(x), 4), dtype=torch.float64, device=_DEV))
    torch.cuda.synchronize()
    if case["tune"]:
        tab.plan_tune(s["plan"].h, ipos.data_ptr(), jpos.data_ptr(), s["out"].data_ptr())
    return s


def _treepm_run(s):
    s["tab"].plan_launch(s["plan"].h, s["ipos"].data_ptr(), s["jpos"].data_ptr(), s["out"].data_ptr())
    return s["out"][:, :3].float()


def _treepm_exact(case, seed):
    """The table's force -- linear in 2 + |dx|^2 (table units) between the nodes, which are the
    floats with `bits` leading mantissa bits -- in 64 bits on the same float32 table coordinates."""
    x, xj, items, m, rs, rcut, eps = _treepm_inputs(case, seed)
    if int((items[:, 1].astype(np.int64) * items[:, 3]).sum()) > 6e9:
        return None
    size, tick = 1 << (4 + case["bits"]), 1 << (23 - case["bits"])
    node32 = (np.arange(size, dtype=np.uint32) * np.uint32(tick) + np.uint32(0x40000000)).view(np.float32)
    top = float(1 << 16) * (2.0 - 1.0 / (1 << case["bits"]))
    scale = float(np.float32(top - 2.0) / np.float32(rcut * rcut))
    f = workloads.gaussian_split_force(rs, rcut, eps)
    node = node32.astype(np.float64)
    # the nodes' radii are floats, as the table's generation has them
    val = np.array([f(float(np.sqrt(np.float32((s - 2.0) / scale)))) for s in node])
    slope = np.append(np.diff(val) / np.diff(node), 0.0)
    node, val, slope = _f64(node), _f64(val), _f64(slope)
    xs = float(np.float32(math.sqrt(scale)))
    xi, y = (x.double() * xs).float().double(), (xj.double() * xs).float().double()
    out = torch.zeros_like(xi)
    for i0, ni, j0, nj in items.tolist():
        if ni == 0:
            continue
        dx = y[None, j0:j0 + nj] - xi[i0:i0 + ni, None]
        s = (2.0 + (dx * dx).sum(-1)).clamp_(max=float(node[-1]))
        # the node's index: the exponent (from 1) and the leading mantissa bits of s
        b = torch.log2(s).floor_()
        b = torch.where(torch.exp2(b) > s, b - 1, b)
        k = ((b - 1) * (1 << case["bits"]) + ((s * torch.exp2(-b) - 1.0) * (1 << case["bits"])).floor()).long()
        w = float(m) * (val[k] + (s - node[k]) * slope[k])
        out[i0:i0 + ni] = (w[..., None] * dx).sum(1)
    return out / xs


def _treepm_work(case):
    n = case["n"]
    rcut = 4.5 * 1.25 / n ** (1.0 / 3.0)
    nb = max(3, min(round((n / case["group"]) ** (1.0 / 3.0)), int(1.0 / rcut)))
    b = 1.0 / nb
    # the volume within rcut of a block: the block, its sides, its edges, its corners
    vol = b ** 3 + 6 * b * b * rcut + 3 * math.pi * b * rcut ** 2 + 4.0 / 3.0 * math.pi * rcut ** 3
    per = n * vol
    return dict(bytes=nb ** 3 * per * 16 + n * (16 + 32), flops=_FLOP5 * n * per)


# ---- tree: a Barnes-Hut step ----------------------------------------------------------------

def _tree_inputs(case, seed):
    """A Hernquist sphere (a = 1, within 100 a), float32 positions, in pinned host memory."""
    n = case["n"]
    gen = torch.Generator(_DEV).manual_seed(seed)
    q = torch.rand(n, generator=gen, device=_DEV, dtype=torch.float64) * (100.0 / 101.0) ** 2
    r = q.sqrt() / (1.0 - q.sqrt())
    d = torch.randn((n, 3), generator=gen, device=_DEV, dtype=torch.float64)
    x = (d / d.norm(dim=1, keepdim=True) * r[:, None]).float().double()
    return x, float(np.float32(1.0 / n)), 1e-3


def _tree_prepare(case, seed):
    g5 = _lib(ffi.G5)
    x, m, eps = _tree_inputs(case, seed)
    n = case["n"]
    xh = x.cpu().pin_memory().numpy()
    mh = torch.full((n,), m, dtype=torch.float64).pin_memory().numpy()
    tree = workloads.GpuTree(xh, mh, case["theta"], case["nleaf"], case["ncrit"], eps)
    s = dict(kind="tree", g5=g5, x=xh, m=mh, eps2=eps * eps, tree=tree, irec=torch.zeros((n, 4), device=_DEV),
             perm=np.empty(n, np.int32), out=[torch.zeros((n, 4), dtype=torch.float64, device=_DEV) for _ in range(2)])
    s["plans"] = [_Plan(g5, g5.plan_create(k, items)) for k, items in zip((g5.NEWTON, g5.QUAD), tree.items())]
    torch.cuda.synchronize()
    if case["tune"]:
        tree.irecords(s["eps2"], s["irec"].data_ptr())
        for plan, args in zip(s["plans"], _tree_args(s)):
            g5.plan_tune_indexed(plan.h, *args)
    return s


def _tree_args(s):
    d, i = s["tree"].device(), s["irec"].data_ptr()
    return ((i, d["part"], None, d["pidx"], s["out"][0].data_ptr()),
            (i, d["cell"], d["cquad"], d["cidx"], s["out"][1].data_ptr()))


def _tree_run(s):
    g5, tree = s["g5"], s["tree"]
    tree.rebuild(s["x"], s["m"])
    items = tree.items()
    tree.irecords(s["eps2"], s["irec"].data_ptr())
    for plan, it, args in zip(s["plans"], items, _tree_args(s)):
        g5.plan_update(plan.h, it)
        g5.plan_launch_indexed(plan.h, *args)
    tree.L.pgbt_perm(C.c_void_p(tree.h), ffi.ptr(s["perm"], C.c_int))   # tree order -> the program's order
    p, c = s["out"]
    return dict(acc=(p[:, :3] + c[:, :3]).float(), pot=(p[:, 3] - c[:, 3]).float(), perm=s["perm"])


def _tree_exact(case, seed):
    """The direct sum (which the multipole expansion differs from too), in tree order."""
    if case["n"] > 70000:
        return None
    x, m, eps = _tree_inputs(case, seed)
    tree = workloads.GpuTree(x.cpu().numpy(), np.full(case["n"], m), case["theta"], case["nleaf"], case["ncrit"], eps)
    perm = torch.as_tensor(tree.set().perm, device=_DEV).long()   # only where each particle goes
    tree.close()
    x = x[perm]
    acc, pot = _gravity_exact(x, x, torch.full_like(x[:, 0], m), eps * eps)
    return dict(acc=acc, pot=-pot, perm=None)


def _tree_work(case):
    # list entries a particle, as counted on these spheres (3050 at 2^14, 4250 at 2^20 for theta = 0.5
    # and ncrit = 256): a third of them particles, the rest cells
    n = case["n"]
    per = (3050.0 + 200.0 * math.log2(n / 16384.0)) * (0.5 / case["theta"]) ** 2.4 * (0.73 + 0.27 * case["ncrit"] / 256.0)
    return dict(bytes=n * (32 + 16 + 16 + 4), flops=n * per * (_FLOP5 + 2 * _FLOP6) / 3)


# ---- integrate: an interval of the device integrator ----------------------------------------

_EPS, _ETA, _ETA_S, _DTMAX = 0.0, 0.2, 0.01, 0.125   # the reference's sample parameters


def _integrate_prepare(case, seed):
    x, v, m = workloads.plummer_henon(case["n"], seed)
    return dict(kind="integrate", g6=_lib(ffi.G6), x=x, v=v, m=m)


def _integrate_run(s):
    h = ffi.Hermite(s["g6"], s["m"], s["x"], s["v"], _EPS ** 2, _ETA, _ETA_S, _DTMAX)
    h.advance(_DTMAX)
    state = h.get()
    state["steps"], state["blocks"] = h.counts()
    h.close()
    return state


def _integrate_exact(case, seed):
    return None   # two trajectories part where a particle's step is halved in one of them only


def _integrate_work(case):
    n = case["n"]
    steps = 26.0 * (n / 16384.0) ** 0.33   # particle steps a particle and interval, as measured
    return dict(bytes=n * 16 * 8 * 2, flops=_FLOP6 * n * n * (steps + 1))


_KINDS = dict(
    call=(_call_prepare, _call_run, _call_exact, _call_work),
    block=(_block_prepare, _block_run, _block_exact, _block_work),
    clusters=(_clusters_prepare, _clusters_run, _clusters_exact, _clusters_work),
    direct=(_direct_prepare, _direct_run, _direct_exact, _direct_work),
    treepm=(_treepm_prepare, _treepm_run, _treepm_exact, _treepm_work),
    tree=(_tree_prepare, _tree_run, _tree_exact, _tree_work),
    integrate=(_integrate_prepare, _integrate_run, _integrate_exact, _integrate_work),
)
