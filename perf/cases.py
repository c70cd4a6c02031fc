"""Workloads of the external-mode solver, each a call sequence a host program makes.

``listed()`` gives the workloads, ``draw(rng)`` another one of the same ranges,
``prepare(case, seed)`` what the host program has in hand (grids, state, a
context), ``run(state)`` one pass through the public entry points, ``work(case)``
the bytes and operations a pass cannot do without, and ``exact(case, seed)`` the
first pass's results from a plain torch FP64 evaluation of the same formulas
with the linear systems solved to rounding.

Kinds of workloads:

* ``host``: one CALPUV2C call on host arrays, as EFDC+'s time loop makes it
  (hdmt2t.f90:509): everything goes up, one step, everything comes back.
* ``resident``: a few steps with the state kept on the GPU, then the surface,
  depths and discharges downloaded (an output interval of a hydrodynamic run);
  one basin or an ensemble of basins of uneven sizes.
* ``batch``: one step of an ensemble on page-locked host arrays, the arrays the
  driver does not touch declared unchanged.
* ``flat``: wetting and drying tidal flats (ISDRY = 99), state on the GPU.
* ``levels``: CALPUV9C calls in the order of the three-time-level time loop.
* ``producers``: the explicit momentum terms (CALEXP2T), a step that reads them
  and the bottom stresses (CALTBXY) of one coupled time step, on host arrays.
* ``calib``: the gradient of a gauge misfit, by torch.autograd over the adjoint.
* ``congrad``: the CONGRAD solve alone on arrays that are already on the device.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parent.parent / "efdcplus8.5_b200"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import efdc_xm as X  # noqa: E402
import scenario as S  # noqa: E402
from calib import CalibLoss, CalibProblem  # noqa: E402

OUT = ("p", "hp", "uhdye", "vhdxe")  # what a run writes out at an output interval
DRY = ("lmaskdry", "iscdry", "lopenbcdry", "natdry", "qdwaste", "vdwaste")
PREC = {"fp64": X.PREC_FP64, "mixed": X.PREC_MIXED}


def listed():
    return [
        # an EFDC+ sample-model-sized lake (about 1,100 cells), coupled step by
        # step with a Fortran host: the smallest call, where latency counts
        dict(name="host_lake", kind="host", nx=44, ny=28, prec="fp64"),
        # the 100x60 basin of the CPU-runnable configuration, the same way
        dict(name="host_100x60", kind="host", nx=100, ny=60, prec="fp64"),
        # a regional model of 240,000 cells in mixed precision, output every 10 steps
        dict(name="regional_mixed", kind="resident", members=1, nx=512, ny=512, prec="mixed",
             steps=10),
        # a million-cell model in the reference's precision, output every 5 steps
        dict(name="million_fp64", kind="resident", members=1, nx=1024, ny=1024, prec="fp64",
             steps=5),
        # the large single domain: 2048x2048, curvilinear metrics
        dict(name="large_mixed", kind="resident", members=1, nx=2048, ny=2048, prec="mixed",
             steps=4),
        # an ensemble of uneven basins (10k to 400k cells), output every 5 steps
        dict(name="ensemble_mixed", kind="resident", members=24, lo=10000, hi=400000,
             prec="mixed", steps=5),
        # the same kind of ensemble stepped on the host program's own arrays
        dict(name="ensemble_host", kind="batch", members=12, lo=10000, hi=200000, prec="mixed"),
        # wetting and drying flats: three or four solves per step
        dict(name="flats_mixed", kind="flat", members=4, nx=384, ny=384, prec="mixed", steps=4),
        # the three-time-level scheme: five leapfrog steps and their correction
        dict(name="levels_fp64", kind="levels", nx=317, ny=203, prec="fp64", every=5),
        # one coupled time step of a four-layer model with its upstream producers
        dict(name="producers_4layers", kind="producers", nx=300, ny=200, layers=4),
        # calibration: forward and adjoint of 20 steps with a snapshot every 5
        dict(name="calib_gradient", kind="calib", nx=128, ny=96, steps=20, every=5),
        # CONGRAD alone on device arrays, ragged size
        dict(name="congrad_device", kind="congrad", nx=403, ny=299),
    ]


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("host", "host", "resident", "resident", "resident", "ensemble", "batch",
                       "flat", "levels", "producers", "calib", "congrad"))
    prec = rng.choice(("fp64", "mixed"))
    if kind == "ensemble":
        return dict(kind="resident", members=rng.randint(2, 24), lo=10000,
                    hi=_loguniform(rng, 20000, 200000), prec=prec, steps=rng.randint(2, 5))
    if kind == "batch":
        return dict(kind="batch", members=rng.randint(2, 12), lo=10000,
                    hi=_loguniform(rng, 20000, 200000), prec=prec)
    lo, hi = {"host": (24, 400), "resident": (60, 1024), "flat": (48, 384),
              "levels": (40, 512), "producers": (40, 320), "calib": (40, 160),
              "congrad": (30, 560)}[kind]
    nx = _loguniform(rng, lo, hi)
    ny = min(hi, max(lo, int(nx * rng.uniform(0.5, 1.6)) | 1))
    c = dict(kind=kind, nx=nx, ny=ny)
    if kind == "host":
        c["prec"] = prec
    elif kind == "resident":
        c.update(members=1, prec=prec, steps=rng.randint(3, 10))
    elif kind == "flat":
        c.update(members=rng.randint(1, 4), prec=prec, steps=rng.randint(2, 4))
    elif kind == "levels":
        c.update(prec=prec, every=rng.randint(3, 6))
    elif kind == "producers":
        c.update(layers=rng.choice((1, 2, 4, 8)))
    elif kind == "calib":
        c.update(steps=rng.randint(8, 24), every=rng.randint(3, 6))
    return c


# ---------------------------------------------------------------- inputs
def _smooth(rng, shape, cells):
    """A smooth random field in [0, 1]: seeded noise at a coarse spacing,
    interpolated."""
    ny, nx = shape
    coarse = torch.from_numpy(rng.random((1, 1, max(3, ny // cells + 2), max(3, nx // cells + 2))))
    f = torch.nn.functional.interpolate(coarse, size=(ny, nx), mode="bicubic",
                                        align_corners=True)[0, 0].numpy()
    lo, hi = f.min(), f.max()
    return (f - lo) / (hi - lo)


def _basin(nx, ny, seed, *, curvilinear=False, depth=(4.0, 30.0)):
    """A tidal basin: the islands of its model grid (the same for every seed), and
    seeded smooth bathymetry, M2 tide on the west side, a surface that is already
    moving, wind and river inflows."""
    rng = np.random.default_rng(seed)
    jc, ic = ny + 2, nx + 2
    land = np.random.default_rng((nx, ny)).random((ny, nx)) < 0.07
    belv = -(depth[0] + (depth[1] - depth[0]) * _smooth(rng, (jc, ic), 10))
    amp = rng.uniform(0.2, 0.5)
    scn = S.make_scenario(nx, ny, seed=seed, dx=100.0, dy=100.0, land_mask=land, belv2d=belv,
                          curvilinear=(60.0, 180.0) if curvilinear else None,
                          obc_sides=("W",), amp=amp, u0=0.0, dt=10.0, rsqm=1e-10, iterm=500,
                          fill_dead_ends=True)
    g, st, la = scn.grid, scn.state, scn.la
    i0 = np.arange(1, la)
    x = g["il"][i0] / nx
    y = g["jl"][i0] / ny
    eta = rng.uniform(0.05, 0.2) * np.cos(math.pi * x) * np.cos(math.pi * y)
    st["hp"][i0] = eta - g["belv"][i0]
    st["h1p"][:] = st["hp"]
    st["p"][i0] = S.G * (st["hp"][i0] + g["belv"][i0])
    st["hu"], st["hv"], st["hpi"], st["hui"], st["hvi"] = S.face_depths(g, st["hp"])
    st["tsx"][i0] = rng.uniform(-1e-4, 1e-4)
    st["tsy"][i0] = rng.uniform(-1e-4, 1e-4)
    rivers = rng.choice(i0, size=max(1, (la - 1) // 2000), replace=False)
    st["qsume"][rivers] = rng.uniform(1.0, 20.0, rivers.size)
    return scn


def _scenarios(case, seed):
    """The basins of a case, from the seed alone."""
    kind = case["kind"]
    if "lo" in case:
        rng = np.random.default_rng(case["members"])  # the basins' sizes are the ensemble's
        cells = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["members"]))
        # scaled to the mean of the range, so that the work follows from the case
        cells *= case["members"] * (case["hi"] - case["lo"]) / math.log(
            case["hi"] / case["lo"]) / cells.sum()
        cells = np.clip(cells, case["lo"], case["hi"])
        out = []
        for k, n in enumerate(cells):
            side = math.sqrt(n / 0.93)
            nx = max(8, int(side * rng.uniform(0.7, 1.4)))
            out.append(_basin(nx, max(8, int(n / 0.93 / nx)), seed * 1009 + k))
        return out
    nx, ny = case["nx"], case["ny"]
    if kind == "flat":  # a rising 2 m tide that starts at mean level
        out = []
        for k in range(case["members"]):
            rng = np.random.default_rng(seed * 1009 + k)
            x = np.linspace(0.0, 1.0, nx + 2)[None, :]
            belv = -2.0 + 5.75 * x + 0.3 * rng.standard_normal((ny + 2, nx + 2))
            belv[:, :3] = np.minimum(belv[:, :3], -2.0)
            out.append(S.make_scenario(nx, ny, seed=seed + k, land_frac=0.0, belv2d=belv, dx=50.0,
                                       dy=50.0, obc_sides=("W",), amp=2.0,
                                       phase=S.M2_PERIOD / 4, dt=5.0, isdry=99, hdry=0.05,
                                       ndrystp=-10, rsqm=1e-10, iterm=500, u0=0.0))
        return out
    scn = _basin(nx, ny, seed, curvilinear=nx >= 2000 or ny >= 2000)
    if kind == "levels":
        S.add_three_levels(scn)
    if kind == "producers":
        S.add_momentum(scn, kc=case["layers"], seed=seed)
    return [scn]


def _joined(scns, pinned, without=()):
    """One array per field with the members back to back (as an ensemble driver
    holds them), page-locked or not, and the members' states as views of it;
    the fields in `without` are not given."""
    sizes = [s.lc + 1 for s in scns]
    total, states = sum(sizes), [dict() for _ in scns]
    joined = {}
    for k, v in scns[0].state.items():
        if k in without:
            continue
        if not isinstance(v, np.ndarray) or v.shape != (sizes[0],):
            for s, st in zip(scns, states):
                st[k] = s.state[k]
            continue
        t = torch.empty(total, dtype=torch.float64 if v.dtype == np.float64 else torch.int32,
                        pin_memory=pinned)
        a, o = t.numpy(), 0
        joined[k] = a
        for s, st, n in zip(scns, states, sizes):
            a[o:o + n] = s.state[k]
            st[k] = a[o:o + n]
            o += n
    return joined, states


class _State:
    pass


def prepare(case, seed):
    kind = case["kind"]
    s = _State()
    s.case, s.kind, s.n = case, kind, 0
    s.scns = _scenarios(case, seed)
    s.prec = PREC[case.get("prec", "fp64")]
    scn = s.scns[0]
    if kind == "congrad":
        s.sys = {k: torch.from_numpy(v).cuda() for k, v in _system(scn, seed).items()}
        s.p0 = torch.from_numpy(scn.state["p"]).cuda()
        s.p = s.p0.clone()
        return s
    if kind == "calib":
        truth, s.log_n, s.amps, gauges = _calib_inputs(case, scn, seed)
        s.pb = CalibProblem(scn, gauges, case["steps"], every=case["every"])
        s.pb.obs = s.pb.forward(truth, np.array([0.45, 0.55, 0.5, 0.6]), keep=False)
        return s
    # the batch driver's basins neither dry nor flood: it holds no wet/dry arrays
    s.joined, s.states = _joined(s.scns, pinned=kind not in ("host", "producers"),
                                 without=DRY if kind == "batch" else ())
    if kind in ("host", "producers"):
        s.sol = X.Solver(scn.grid)
    else:
        s.sol = X.BatchSolver([q.grid for q in s.scns])
    if kind == "producers":
        s.sol.set_momentum(scn.momentum)
        s.bed = S.make_bed(scn, seed=seed, kc=case["layers"])
        s.sol.set_bed(s.bed)
        s.mom, s.drag = _producer_inputs(scn, seed)
        s.step_in = {k: v for k, v in s.states[0].items()
                     if k not in ("fcaxe", "fcaye", "fxe", "fye", "tbx", "tby")}
        s.sol.upload(s.states[0])
    elif kind == "batch":
        # the driver rewrites the forcing before each step and leaves the state alone
        names = ("p", "hp", "hu", "hv", "uhdye", "vhdxe", "sub", "svb", "sbx", "sby")
        s.first = s.sol.prepare(s.states)
        s.later = s.sol.prepare(s.states, unchanged=X.same_bits(names))
    elif kind != "host":
        s.sol.upload(s.states)
        s.out = [{k: st[k] for k in OUT} for st in s.states]
        if kind == "flat":
            for o, st in zip(s.out, s.states):
                o["lmaskdry"] = st["lmaskdry"]
    return s


def _system(scn, seed):
    """The scaled system of a CALPUV2C step of a basin (calpuv2c.f90:306-399),
    with the boundary rows clamped, and its neighbour maps."""
    g, st, la = scn.grid, scn.state, scn.la
    i0 = np.arange(1, la)
    n = scn.lc + 1
    D2, G = 5.0, S.G
    rng = np.random.default_rng(seed + 1)
    wx, wy = st["sub"] * g["hruo"] * st["hu"], st["svb"] * g["hrvo"] * st["hv"]
    bc = g["obc"]["W"]["l"] - 1
    for b in bc:  # the boundary values enter the right-hand side
        wx[g["lec"][b] - 1] = 0.0
    c = {k: np.zeros(n) for k in ("ccc", "ccs", "ccn", "ccw", "cce", "fptmp")}
    C1 = -0.5 * D2 * G
    c["ccw"][i0] = C1 * wx[i0]
    c["cce"][i0] = C1 * wx[g["lec"][i0] - 1]
    c["ccs"][i0] = C1 * wy[i0]
    c["ccn"][i0] = C1 * wy[g["lnc"][i0] - 1]
    for k in ("ccw", "cce", "ccs", "ccn"):
        c[k][bc] = 0.0
    c["ccc"][i0] = 0.1 * g["dxyp"][i0] - sum(c[k][i0] for k in ("ccw", "cce", "ccs", "ccn"))
    c["fptmp"][i0] = 0.1 * g["dxyp"][i0] * (st["p"][i0] + rng.normal(0.0, 0.05, la - 1))
    scale = 1.0 / c["ccc"][i0].min()
    for k in c:
        c[k][i0] *= scale
    c["ccc"][0] = c["ccc"][la:] = 1.0
    for k in ("lnc", "lsc", "lec", "lwc"):
        c[k] = g[k].copy()
    return c


def _calib_inputs(case, scn, seed):
    rng = np.random.default_rng(seed + 2)
    log_n = np.full(scn.lc + 1, math.log(0.025))
    truth = log_n.copy()
    truth[1:scn.la] = rng.normal(math.log(0.025), 0.2, scn.la - 1)
    gauges = np.sort(rng.choice(np.arange(scn.la // 4, scn.la), size=20, replace=False))
    return (truth, torch.from_numpy(log_n).requires_grad_(),
            torch.full((4,), 0.48, dtype=torch.float64, requires_grad=True),
            gauges.astype(np.int32))


def _producer_inputs(scn, seed):
    """The internal mode's layer velocities and transports, and the bottom
    layer's velocities, of one time step."""
    mom = S.momentum_fields(scn, seed=seed)
    st = scn.state
    rng = np.random.default_rng(seed + 3)
    n = scn.lc + 1
    drag = dict(ub=mom["u"][0].copy(), vb=mom["v"][0].copy(), vu=0.2 * rng.standard_normal(n),
                uv=0.2 * rng.standard_normal(n), h1u=st["hu"].copy(), h1v=st["hv"].copy())
    for k in ("stbx", "stby", "tbx", "tby"):
        drag[k] = np.zeros(n)
    return mom, drag


# ---------------------------------------------------------------- passes
def _prm(s, scn, **kw):
    p = dict(scn.params, **kw) if kw else scn.params
    return X.make_params(p, n=s.n, tn=scn.tn(s.n), precision=s.prec)


def _stats(sts):
    return np.array([[t.status, t.solves] for t in sts], dtype=np.int32)


def run(s):
    kind = s.kind
    if kind == "host":
        s.n += 1
        t = s.sol.step(_prm(s, s.scns[0]), s.states[0])
        st = s.states[0]
        return [st[k] for k in OUT + ("hu", "hv", "uhe", "vhe")] + [_stats([t])]
    if kind == "batch":
        s.n += 1
        first = s.n == 1
        t = s.sol.step_prepared([_prm(s, q) for q in s.scns], s.first if first else s.later)
        return [s.joined[k] for k in OUT + ("hu", "hv", "uhe", "vhe")] + [_stats(t)]
    if kind in ("resident", "flat"):
        for _ in range(s.case["steps"]):
            s.n += 1
            t = s.sol.step_device([_prm(s, q) for q in s.scns])
        s.sol.download(s.out)
        out = [s.joined[k] for k in OUT] + [_stats(t)]
        return out + [s.joined["lmaskdry"]] if kind == "flat" else out
    if kind == "levels":
        every = s.case["every"]
        for k in range(every + 1):
            istl = 3 if k < every else 2
            s.n += istl == 3
            t = s.sol.step_device([_prm(s, s.scns[0], **_level(k, every))])
        s.sol.download(s.out)
        return [s.joined[k] for k in OUT] + [_stats(t)]
    if kind == "producers":
        s.n += 1
        s.sol.explicit(X.make_explicit_params(1.0, 1, 0), s.mom)
        t = s.sol.step(_prm(s, s.scns[0]), s.step_in)
        s.sol.bottom_stress(X.make_drag_params(s.scns[0].params, n=s.n), s.drag)
        st = s.step_in
        return [s.mom[k] for k in ("fcaxe", "fcaye", "fxe", "fye", "fcax", "fcay", "fx", "fy",
                                   "cac")] + [st[k] for k in OUT] + \
            [s.drag[k] for k in ("stbx", "stby", "tbx", "tby")] + [_stats([t])]
    if kind == "calib":
        s.log_n.grad = s.amps.grad = None
        loss = CalibLoss.apply(s.log_n, s.amps, s.pb)
        loss.backward()
        return [loss.detach(), s.log_n.grad, s.amps.grad]
    # congrad
    s.p.copy_(s.p0)
    C = X.C
    it, rsq = C.c_int32(0), C.c_double(0.0)
    q = s.sys
    rc = X.load().efdc_xm_congrad_noalloc(
        s.scns[0].la, *[C.c_void_p(q[k].data_ptr()) for k in
                        ("lnc", "lsc", "lec", "lwc", "ccc", "ccs", "ccn", "ccw", "cce", "fptmp")],
        C.c_void_p(s.p.data_ptr()), 1e-10, 500, C.c_void_p(torch.cuda.current_stream().cuda_stream),
        C.byref(it), C.byref(rsq))
    return [s.p, rc, it.value]


def _level(k, every):
    """Call k of the three-time-level loop's block of `every` leapfrog steps and
    their correction (hdmt.f90:1009-1029)."""
    if k < every:
        return dict(tl3_istl=3, nctbc=k + 1, rold=0.0, rnew=1.0)
    return dict(tl3_istl=2, nctbc=0, rold=0.5, rnew=0.5)


# ---------------------------------------------------------------- work
def _cells(case):
    if "lo" in case:
        return case["members"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    return case.get("members", 1) * case["nx"] * case["ny"] * (1.0 if case["kind"] == "flat"
                                                               else 0.92)


def work(case):
    """Per step and cell: 28 arrays of metrics, state and forcing read and 9
    written, 150 operations around the solve and 20 in each of about 15
    iterations of it."""
    n, kind = _cells(case), case["kind"]
    if kind == "congrad":
        return {"bytes": n * (7 * 8 + 4 * 4 + 8), "flops": n * 20.0 * 15}
    steps = {"levels": case.get("every", 0) + 1, "calib": 3.0 * case.get("steps", 0)}.get(
        kind, case.get("steps", 1))
    byt, ops = n * steps * 37 * 8.0, n * steps * (150.0 + 20 * 15)
    if kind == "producers":
        byt += n * (case["layers"] * (4 + 5 + 4) + 30) * 8.0
        ops += n * case["layers"] * 70.0
    return {"bytes": byt, "flops": ops}


# ---------------------------------------------------------------- exact
class _Solve(torch.autograd.Function):
    """x with A x = b on the water cells, A = (cc, cs, cw, ce, cn) symmetric, by
    Jacobi-preconditioned CG taken to rounding."""

    @staticmethod
    def _cg(m, c, b):
        cc, cs, cw, ce, cn = c
        mul = lambda v: torch.where(m.water, cc * v + cs * v[m.ls] + cw * v[m.lw] +  # noqa: E731
                                    ce * v[m.le] + cn * v[m.ln], m.zero)
        inv = torch.where(m.water, 1.0 / torch.where(m.water, cc, m.one), m.zero)
        b = torch.where(m.water, b, m.zero)
        x = b * inv
        stop = 1e-31 * float((b * b * inv).sum())
        for _ in range(2):  # restarted once from the true residual
            r = b - mul(x)
            z = r * inv
            p = z.clone()
            rz = (r * z).sum()
            for k in range(1000):
                if k % 8 == 0 and float(rz) <= stop:
                    break
                q = mul(p)
                a = rz / (p * q).sum()
                x = x + a * p
                r = r - a * q
                z = r * inv
                new = (r * z).sum()
                p = z + (new / rz) * p
                rz = new
        return x

    @staticmethod
    def forward(ctx, m, cc, cs, cw, ce, cn, b):
        x = _Solve._cg(m, (cc, cs, cw, ce, cn), b)
        ctx.m = m
        ctx.save_for_backward(cc, cs, cw, ce, cn, x)
        return x

    @staticmethod
    def backward(ctx, g):
        m = ctx.m
        *c, x = ctx.saved_tensors
        v = _Solve._cg(m, c, g)
        return (None, -v * x, -v * x[m.ls], -v * x[m.lw], -v * x[m.le], -v * x[m.ln], v)


class _Model:
    """The basins of a case as one set of L-indexed arrays, one after another."""

    def __init__(self, scns):
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        off = np.cumsum([0] + [s.lc + 1 for s in scns])
        cat = lambda f: torch.from_numpy(  # noqa: E731
            np.concatenate([f(s) for s in scns])).to(dev)
        ix = lambda k: torch.from_numpy(np.concatenate(  # noqa: E731
            [np.maximum(s.grid[k].astype(np.int64) - 1, 0) + o for s, o in zip(scns, off)])).to(dev)
        self.le, self.lw, self.ln, self.ls = ix("lec"), ix("lwc"), ix("lnc"), ix("lsc")
        self.water = cat(lambda s: (np.arange(s.lc + 1) >= 1) & (np.arange(s.lc + 1) < s.la))
        self.zero = torch.zeros((), dtype=torch.float64, device=dev)
        self.one = self.zero + 1.0
        for k in ("dxyp", "dxyip", "dxiu", "dyiu", "dxiv", "dyiv", "dxyu", "dxyv", "hruo", "hrvo",
                  "subo", "svbo", "belv"):
            setattr(self, k, cat(lambda s, k=k: s.grid[k]))
        self.st = {k: cat(lambda s, k=k: s.state[k]) for k, v in scns[0].state.items()
                   if isinstance(v, np.ndarray) and v.dtype == np.float64 and
                   v.shape == (scns[0].lc + 1,)}
        self.sub, self.svb = self.st["sub"], self.st["svb"]
        w = self.water
        self.fu = torch.where(w, 0.5 / torch.where(w, self.dxyu, self.one), self.zero)
        self.fv = torch.where(w, 0.5 / torch.where(w, self.dxyv, self.one), self.zero)
        self.prm = scns[0].params
        ob = [s.grid["obc"]["W"] for s in scns]
        self.bc = torch.from_numpy(np.concatenate([o["l"] - 1 + f for o, f in zip(ob, off)])).to(dev)
        self.isbc = torch.zeros_like(w)
        self.isbc[self.bc] = True
        self.pcb = torch.from_numpy(np.concatenate([o["pcb"][0] for o in ob])).to(dev)
        self.psb = torch.from_numpy(np.concatenate([o["psb"][0] for o in ob])).to(dev)
        self.tcp = float(scns[0].grid["tcp"][0])
        self.off = off

    def step(self, st, n, *, istl=0, nctbc=0, pcb=None, log_n=None):
        """One CALPUV2C (istl = 0) or CALPUV9C(istl) step of every basin."""
        w, le, lw, ln, ls = self.water, self.le, self.lw, self.ln, self.ls
        G, dt = float(self.prm["g"]), float(self.prm["dt"])
        delt = 2.0 * dt if istl == 3 else dt
        D2, delti = 0.5 * delt, 1.0 / delt
        on = lambda a: torch.where(w, a, self.zero)  # noqa: E731
        sub, svb = self.sub, self.svb
        st = dict(st)
        tbx, tby = self._manning(st, log_n) if log_n is not None else (st["tbx"], st["tby"])
        tsx, tsy = st["tsx"], st["tsy"]
        if istl:
            u0, v0, p0 = st["uhdy1e"], st["vhdx1e"], st["p1"]
            tsx, tsy, tbx, tby = st["tsx1"], st["tsy1"], st["tbx1"], st["tby1"]
            hu, hv = (st["hu"], st["hv"]) if istl == 3 else \
                (0.5 * (st["hu"] + st["h1u"]), 0.5 * (st["hv"] + st["h1v"]))
        else:
            u0, v0, p0, hu, hv = st["uhdye"], st["vhdxe"], st["p"], st["hu"], st["hv"]
        snlt, ritb1 = float(self.prm["snlt"]), float(self.prm["ritb1"])
        fu = on(u0 - D2 * sub * self.hruo * hu * (p0 - p0[lw]) + sub * delt * self.dxiu *
                (self.dxyu * (tsx - ritb1 * tbx) + st["fcaxe"] - snlt * st["fxe"]))
        fv = on(v0 - D2 * svb * self.hrvo * hv * (p0 - p0[ls]) + svb * delt * self.dyiv *
                (self.dxyv * (tsy - ritb1 * tby) - st["fcaye"] - snlt * st["fye"]))
        fp = delti * self.dxyp * p0 - 0.5 * G * (u0[le] - u0 + v0[ln] - v0)
        if istl == 3:
            h = 0.5 if nctbc == 1 else 1.0
            st.update(uhdy2e=st["uhdy1e"], vhdx2e=st["vhdx1e"], uhdy1e=h * st["uhdye"],
                      vhdx1e=h * st["vhdxe"], p1=st["p"], h1u=st["hu"], h1v=st["hv"],
                      h2p=st["h1p"], h1p=st["hp"])
        elif not istl:
            st["h1p"] = st["hp"]
        fp = on(fp - 0.5 * G * ((sub * fu)[le] - sub * fu + (svb * fv)[ln] - svb * fv -
                                2.0 * st["qsume"]))
        kx, ky = on(self.hruo * hu), on(self.hrvo * hv)
        c1 = -0.5 * D2 * G
        cw, cs = c1 * sub * kx, c1 * svb * ky
        ce, cn = cw[le], cs[ln]
        cc = on(delti * self.dxyp - cs - cw - ce - cn)
        # clamped cells: their value goes to the right-hand side of the cell to
        # the east (setopenbc.f90:32-74, setopenbc2.f90:17-22)
        ph = float(self.prm["pi2"]) * math.fmod(dt * n, self.tcp) / self.tcp
        amp = self.pcb if pcb is None else pcb
        f = amp * math.cos(ph) + (self.psb * math.sin(ph) if pcb is None else 0.0)
        east = le[self.bc]
        off = self.isbc
        gone = torch.zeros_like(off)
        gone[east] = True
        fp = fp.index_add(0, east, 0.5 * D2 * G * self.hruo[east] * hu[east] * f)
        cc = torch.where(off, delti * self.dxyp, cc)
        cw, cs, ce, cn = (torch.where(off, self.zero, on(a)) for a in (cw, cs, ce, cn))
        cw = torch.where(gone, self.zero, cw)
        fp = fp.index_put((self.bc,), delti * self.dxyp[self.bc] * f)
        p = _Solve.apply(self, cc, cs, cw, ce, cn, fp)
        un = on(sub * (fu - D2 * kx * (p - p[lw])))
        vn = on(svb * (fv - D2 * ky * (p - p[ls])))
        q = st["qsume"]
        if istl:
            hb, ub, vb = (st["h2p"], st["uhdy2e"], st["vhdx2e"]) if istl == 3 else \
                (st["h1p"], st["uhdy1e"], st["vhdx1e"])
        else:
            hb, ub, vb = st["h1p"], u0, v0
        su, sv = un + ub, vn + vb
        hp = hb + delt * self.dxyip * (q - 0.5 * (su[le] - su + sv[ln] - sv))
        hp = torch.where(off, p / G - self.belv, hp)
        hp = torch.where(w, hp, st["hp"])
        a = self.dxyp * hp
        st.update(uhdye=un, vhdxe=vn, hp=hp, p=torch.where(w, G * (hp + self.belv), st["p"]),
                  hu=on((a + a[lw]) * self.fu), hv=on((a + a[ls]) * self.fv),
                  uhe=on(un * self.dyiu), vhe=on(vn * self.dxiv))
        return st

    def _manning(self, st, log_n):
        """The calibration model's bottom drag (see include/efdc_xm.h)."""
        w, lw, ls, le, ln = self.water, self.lw, self.ls, self.le, self.ln
        hu = torch.where(w, st["hu"], self.one)
        hv = torch.where(w, st["hv"], self.one)
        u = torch.where(w, st["uhdye"] * self.dyiu / hu, self.zero)
        v = torch.where(w, st["vhdxe"] * self.dxiv / hv, self.zero)
        vu = 0.25 * (v + v[ln] + v[lw] + v[ln[lw]])
        uv = 0.25 * (u + u[le] + u[ls] + u[le[ls]])
        en = torch.exp(log_n)
        nu, nv = 0.5 * (en + en[lw]), 0.5 * (en + en[ls])
        G = float(self.prm["g"])
        tiny = 1e-300
        su = torch.sqrt(torch.clamp(vu * vu + u * u, min=tiny))
        sv = torch.sqrt(torch.clamp(uv * uv + v * v, min=tiny))
        bx = w & (self.subo > 0.5)
        by = w & (self.svbo > 0.5)
        return (torch.where(bx, G * nu * nu / hu ** (1.0 / 3.0) * su * u, self.zero),
                torch.where(by, G * nv * nv / hv ** (1.0 / 3.0) * sv * v, self.zero))


def exact(case, seed):
    kind = case["kind"]
    if kind == "flat":
        return None  # cells decide in serial order, sweep after sweep: a loop over them takes long
    scns = _scenarios(case, seed)
    m = _Model(scns)
    if kind == "congrad":
        return _exact_congrad(scns[0], m, seed)
    if kind == "calib":
        return _exact_calib(case, scns[0], m, seed)
    if kind == "producers":
        return _exact_producers(case, scns[0], m, seed)
    st = m.st
    if kind == "levels":
        n = 0
        for k in range(case["every"] + 1):
            c = _level(k, case["every"])
            n += c["tl3_istl"] == 3
            st = m.step(st, n, istl=c["tl3_istl"], nctbc=c["nctbc"])
    else:
        for n in range(1, case.get("steps", 1) + 1):
            st = m.step(st, n)
    names = OUT if kind in ("resident", "levels") else OUT + ("hu", "hv", "uhe", "vhe")
    return [st[k].cpu() for k in names] + [None]


def _exact_congrad(scn, m, seed):
    c = {k: torch.from_numpy(v).to(m.dev) for k, v in _system(scn, seed).items()}
    x = _Solve.apply(m, c["ccc"], c["ccs"], c["ccw"], c["cce"], c["ccn"], c["fptmp"])
    return [torch.where(m.water, x, m.st["p"]).cpu(), None, None]


def _exact_calib(case, scn, m, seed):
    truth, log_n, amps, gauges = _calib_inputs(case, scn, seed)
    groups = torch.from_numpy((np.arange(len(m.bc)) * 4) // len(m.bc)).to(m.dev)
    gi = torch.from_numpy(gauges.astype(np.int64) - 1).to(m.dev)

    def etas(logn, a):
        st, out = m.st, []
        for n in range(1, case["steps"] + 1):
            st = m.step(st, n, pcb=a[groups] * S.G, log_n=logn)
            out.append(st["p"][gi] / S.G)
        return torch.stack(out)

    with torch.no_grad():
        obs = etas(torch.from_numpy(truth).to(m.dev),
                   torch.tensor([0.45, 0.55, 0.5, 0.6], dtype=torch.float64, device=m.dev))
    k = log_n.detach().to(m.dev).requires_grad_()
    a = amps.detach().to(m.dev).requires_grad_()
    loss = ((etas(k, a) - obs) ** 2).sum()
    loss.backward()
    return [loss.detach().cpu(), k.grad.cpu(), a.grad.cpu()]


def _exact_producers(case, scn, m, seed):
    """calexp2t.f90:205-237, 481-562, 648-689, 940-956, the step, and
    caltbxy.f90:476-537 with hdmt2t.f90:670-684."""
    mom, drag = _producer_inputs(scn, seed)
    mo, dev, w = scn.momentum, m.dev, m.water
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    u, v, uh, vh = (T(mom[k]) for k in ("u", "v", "uhdy", "vhdx"))
    on = lambda x: torch.where(w, x, m.zero)  # noqa: E731
    le, lw, ln, ls = m.le, m.lw, m.ln, m.ls
    up = lambda t, a, b: t.clamp(min=0.0) * a + t.clamp(max=0.0) * b  # noqa: E731
    uhb, vhc = 0.5 * (uh + uh[:, le]), 0.5 * (vh + vh[:, lw])
    vhb, uhc = 0.5 * (vh + vh[:, ln]), 0.5 * (uh + uh[:, ls])
    fuhu, fvhu = on(up(uhb, u, u[:, le])), on(up(vhc, u[:, ls], u))
    fvhv, fuhv = on(up(vhb, v, v[:, ln])), on(up(uhc, v[:, lw], v))
    c = {k: T(mo[k]) for k in ("fcorc", "dydi", "dxdj", "scax", "scay", "saax", "saay", "sgzu",
                               "sgzv", "fsgzu", "fsgzv")}
    lnw, lse = (T(np.maximum(mo[k].astype(np.int64) - 1, 0)) for k in ("lnwc", "lsec"))
    cac = on((c["fcorc"] * m.dxyp + 0.5 * (v[:, ln] + v) * c["dydi"] -
              0.5 * (u[:, le] + u) * c["dxdj"]) * T(mom["hp"]))
    fcax = on(0.25 * c["scax"] * (cac * (v[:, ln] + v) + cac[:, lw] * (v[:, lnw] + v[:, lw])))
    fcay = on(0.25 * c["scay"] * (cac * (u[:, le] + u) + cac[:, ls] * (u[:, lse] + u[:, ls])))
    fx = on(c["fsgzu"] * (fuhu - fuhu[:, lw] + fvhu[:, ln] - fvhu))
    fy = on(c["fsgzv"] * (fvhv - fvhv[:, ls] + fuhv[:, le] - fuhv))
    for L, E, N in zip(mo["lbcs"], mo["lberc"], mo["lbnrc"]):
        for a, sa, other in ((fx, c["saax"], E), (fy, c["saay"], N)):
            for q in (int(L) - 1, max(int(other), 1) - 1):
                a[:, q] = sa[q] * a[:, q]
    st = dict(m.st)
    st.update(fcaxe=(fcax * c["sgzu"]).sum(0), fcaye=(fcay * c["sgzv"]).sum(0),
              fxe=(fx * c["sgzu"]).sum(0), fye=(fy * c["sgzv"]).sum(0))
    new = m.step(st, 1)
    bed = S.make_bed(scn, seed=seed, kc=case["layers"])
    ub, vb, vu, uv = (T(drag[k]) for k in ("ub", "vb", "vu", "uv"))
    zbr = T(bed["zbr"])
    hus, hvs = (torch.where(w, new[k], m.one) for k in ("hu", "hv"))
    stress = []
    for a, b, h, h1, nb, width, inv, lay in (
            (ub, vu, hus, "h1u", lw, "dxp", m.dxiu, "sgzu1"),
            (vb, uv, hvs, "h1v", ls, "dyp", m.dyiv, "sgzv1")):
        dz = T(bed[width]) * zbr
        zb = torch.where(w, 0.5 * (dz[nb] + dz) * inv, m.one)
        mag = torch.sqrt(a * a + b * b + 1e-12)
        ratio = torch.maximum(zb, T(drag[h1])) / zb
        if case["layers"] == 1:
            rough = 0.16 / (torch.log((0.5 * ratio).clamp(min=7.5)) - 1.0) ** 2
        else:
            frac = 0.5 * torch.maximum(T(bed["dzc1"]), T(bed[lay]))
            rough = bed["avcon"] * 0.16 / torch.log((1.0 + frac * ratio).clamp(min=7.5)) ** 2
        smooth = 0.0258 * bed["coeftsbl"] ** (2.0 / 7.0) * bed["avcon"] * \
            (bed["vismud"] / h / mag) * (2.0 / 7.0)
        cd = torch.minimum(0.5 * h / (float(scn.params["dt"]) * mag),
                           torch.where(zbr <= 1e-6, smooth, rough))
        stress.append((on(cd), on(cd * torch.sqrt(a * a + b * b) * a)))
    (stbx, tbx), (stby, tby) = stress
    return [x.cpu() for x in (st["fcaxe"], st["fcaye"], st["fxe"], st["fye"], fcax, fcay, fx, fy,
                              cac)] + [new[k].cpu() for k in OUT] + \
        [x.cpu() for x in (stbx, stby, tbx, tby)] + [None]
