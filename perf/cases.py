"""The work a user of this framework has it do, as measurable cases.

A case is a dict of plain values; `prepare` makes what a program holds before
the call, `run` makes one pass through the public entry points
(regcm_gb300.moloch and the C ABI behind it) and returns the updated state,
`work` counts what a pass cannot do without, and `exact` restates the step in
64-bit torch, from the equations of the MOLOCH core and without this
package's code.

Forms (the `form` of a case):

  segment  one domain between two output times: the prognostic state goes in
           from pinned host memory, `steps` steps run on the GPU, the updated
           prognostic state comes back
  coupled  the step split at the physics: every step the host reads the state
           the physics needs and hands its tendencies back
  batch    an ensemble, or domains of different extents, advanced together
  serve    requests that join a pool, run, are read back and leave
  budget   the mass budget of arrays that the caller keeps on the GPU

Members' state comes back in double precision from an FP64 domain; a mixed
domain holds FP32 fields, and its state is written to single-precision
records, as RegCM's output files hold it.
"""
from __future__ import annotations

import ctypes as C
import dataclasses
import functools
import math

import numpy as np
import torch

from regcm_gb300 import abi
from regcm_gb300 import case as cs
from regcm_gb300.moloch import MolochBatch, MolochPool, domain_from_case

# What a segment reads and writes: the prognostic state.
STATE = ("u", "v", "w", "pai", "tetav", "qx", "trac", "tke", "ps")


def listed():
    """Sizes follow regcm_gb300.case's benchmark configurations, the parity
    tests' option sets and odd extents between them."""
    return [
        # plain dry dynamics at the small benchmark size: launch-bound
        {"name": "fp64 dry 64x64x30", "form": "segment", "recipe": "dry", "nx": 64, "ny": 64, "kz": 30,
         "steps": 40, "precision": "fp64"},
        {"name": "mixed dry 64x64x30", "form": "segment", "recipe": "dry", "nx": 64, "ny": 64, "kz": 30,
         "steps": 24, "precision": "mixed"},
        # a small nest that the host's physics drives step by step
        {"name": "fp64 coupled 47x33x23", "form": "coupled", "recipe": "moist", "nx": 47, "ny": 33, "kz": 23,
         "steps": 4, "precision": "fp64"},
        # the convection-permitting benchmark domain, both precisions
        {"name": "fp64 moist 512x512x41", "form": "segment", "recipe": "moist", "nx": 512, "ny": 512, "kz": 41,
         "steps": 10, "precision": "fp64"},
        {"name": "mixed moist 512x512x41", "form": "segment", "recipe": "moist", "nx": 512, "ny": 512, "kz": 41,
         "steps": 18, "precision": "mixed"},
        # a drop-in call per step: state in, one step, state out
        {"name": "fp64 one step 256x256x41", "form": "segment", "recipe": "moist", "nx": 256, "ny": 256, "kz": 41,
         "steps": 1, "precision": "fp64"},
        # double-moment microphysics, TKE and the reference's exponential nudging, odd extents
        {"name": "fp64 ipptls5 tke 201x157x35", "form": "segment", "recipe": "moist", "nx": 201, "ny": 157,
         "kz": 35, "steps": 10, "precision": "fp64", "ipptls": 5, "tke": True, "lehmann": False},
        # rotated pole with the reference's default splitting (2 advection rounds of 5 substeps)
        {"name": "mixed rotated 150x187x40", "form": "segment", "recipe": "dry", "nx": 150, "ny": 187, "kz": 40,
         "steps": 8, "precision": "mixed", "rotated": True, "nadv": 2, "nsound": 5},
        # an initial-condition ensemble over one region
        {"name": "mixed ensemble 32x128x128x30", "form": "batch", "recipe": "dry", "nx": 128, "ny": 128, "kz": 30,
         "members": 32, "steps": 20, "precision": "mixed"},
        # domains of different extents (regcm_gb300.case.config3_dims) in one context
        {"name": "mixed uneven 12 domains", "form": "batch", "recipe": "moist", "nx": 0, "ny": 0, "kz": 0,
         "members": 12, "first": 0, "steps": 12, "precision": "mixed"},
        # continuous batching: requests of different sizes join, run and leave
        {"name": "mixed serving 4 requests", "form": "serve", "recipe": "moist", "nx": 0, "ny": 0, "kz": 30,
         "members": 4, "first": 0, "steps": 24, "precision": "mixed"},
        # the budget check of a host model that owns its device memory
        {"name": "budget 512x512x41", "form": "budget", "recipe": "moist", "nx": 512, "ny": 512, "kz": 41,
         "precision": "fp64"},
    ]


def _log(rng, lo, hi):
    return cs.log_uniform_int(rng.random(), lo, hi)


def draw(rng):
    """One more case of the same ranges, extents odd as often as even; the
    steps keep a pass below the largest listed one's work."""
    form = rng.choice(("segment", "segment", "segment", "segment", "coupled", "batch", "serve", "budget"))
    prec = rng.choice(("fp64", "mixed"))
    c = {"form": form, "recipe": rng.choice(("dry", "moist")), "precision": prec}
    if form == "batch" and rng.random() < 0.5 or form == "serve":
        c.update(recipe="moist", nx=0, ny=0, kz=30 if form == "serve" else 0, members=rng.randint(2, 6),
                 first=rng.randint(16, 190), precision="mixed", steps=rng.randint(4, 16))
        return c
    if form == "budget":
        c.update(recipe="moist", nx=_log(rng, 40, 500), ny=_log(rng, 40, 500), kz=rng.randint(18, 45),
                 precision="fp64")
        return c
    hi = 160 if form == "coupled" else 420
    c.update(nx=_log(rng, 32, hi), ny=_log(rng, 32, hi), kz=rng.randint(18, 45))
    if form == "batch":
        c.update(nx=_log(rng, 32, 130), ny=_log(rng, 32, 130), members=rng.randint(2, 12), precision="mixed")
    pts = c["nx"] * c["ny"] * c["kz"] * c.get("members", 1)
    most = (6e7 if c["precision"] == "fp64" else 2e8) / (4 if form == "coupled" else 1)
    c["steps"] = max(1, min(rng.choice((1, 4, 10, 24) if prec == "fp64" else (1, 4, 8, 16)), int(most / pts),
                            4 if form == "coupled" else 24))
    if form == "segment":
        if c["recipe"] == "moist":
            c["ipptls"] = rng.choice((2, 2, 3, 4, 5))
        c["tke"] = rng.random() < 0.25
        c["lehmann"] = rng.random() < 0.5 or c["recipe"] == "dry"  # a tracer's weights are Lehmann's
        c["rotated"] = c["recipe"] == "dry" and rng.random() < 0.25
        if rng.random() < 0.25:
            c.update(nadv=2, nsound=rng.choice((2, 3)), steps=min(8, c["steps"]))
    return c


# ---- inputs ------------------------------------------------------------------

def _extents(case):
    """(nx, ny, kz) of every member."""
    n = case.get("members", 1)
    if case["nx"]:
        return [(case["nx"], case["ny"], case["kz"])] * n
    if case["form"] == "serve":  # the serving configuration's sizes, up to 256
        sizes = [min(256, cs.config4_shape(case["first"] + m)[0]) for m in range(n)]
        return [(x, x, case["kz"]) for x in sizes]
    return [cs.config3_dims(case["first"] + m) for m in range(n)]


@functools.lru_cache(maxsize=16)
def _base(nx, ny, kz, recipe, precision, ipptls, tke, lehmann, rotated, nadv, nsound, coarse):
    """The region: terrain, metric, boundary data and mean state of a domain
    (regcm_gb300.case's recipes).  Initial conditions of a seed perturb it."""
    moist = recipe == "moist"
    dx, dt, ns = (3000.0, 20.0, 4) if moist and not coarse else (12000.0, 60.0, 3)
    hills = ([(0.3 * nx * dx, 0.4 * ny * dx, 1500.0), (0.7 * nx * dx, 0.65 * ny * dx, 700.0)] if moist
             else [(0.5 * nx * dx, 0.5 * ny * dx, 500.0)])
    c = cs.build(nx, ny, kz, dx=dx, dt=dt, nsound=nsound or ns, nadv=nadv, moist=moist, seed=nx + ny,
                 hills=hills, wind=10.0, jet=moist, theta_noise=0.0, tracer=not moist, lrotllr=rotated,
                 precision=abi.MLC_PREC_FP64 if precision == "fp64" else abi.MLC_PREC_MIXED,
                 ipptls=ipptls, tke=tke, lehmann=lehmann, name=f"{recipe}_{nx}x{ny}x{kz}")
    if rotated:  # the map factor and latitude of a rotated grid about its equator
        jx, iy = c.dims.jx, c.dims.iy
        lat = np.degrees((np.arange(1, iy + 1) - 0.5 * iy) * dx / 6.371229e6)
        c.static["rlat"][:] = lat
        c.static["msfx"][:] = 1.0 / np.cos(np.radians(lat))[None, :]
        c.static["msfu"][:] = c.static["msfx"]
    return c


def _base_of(case, ext):
    return _base(*ext, case["recipe"], case["precision"], case.get("ipptls"), case.get("tke", False),
                 case.get("lehmann", True), case.get("rotated", False), case.get("nadv", 1),
                 case.get("nsound", 0), case["form"] == "batch")


def _host(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available())


def _initial(base, seed, m, buf):
    """The seed's initial conditions of member m in `buf` (C order, the
    reversed extents of the Fortran arrays)."""
    gen = torch.Generator().manual_seed(1000003 * seed + m)
    for n, b in buf.items():
        b.copy_(torch.from_numpy(base.state[n].T))
    rand = lambda shape: torch.rand(shape, generator=gen, dtype=torch.float64)
    amp = 0.1 if base.params.ipptls else 0.4
    inner = buf["tetav"][..., 1:-1, 1:-1]
    inner += amp * (2.0 * rand(inner.shape) - 1.0)
    buf["u"] *= 1.0 + 0.1 * (rand((1,)) - 0.5)
    qv = buf["qx"][0]
    qv *= 1.0 + 0.05 * (rand(qv.shape) - 0.5)


def _numpy_state(buf):
    return {n: b.numpy().T for n, b in buf.items()}


def _members(case, seed, out=True):
    """Per member (base, initial state), both as slices of one host buffer per
    field, and the buffers the results are read into."""
    ext = _extents(case)
    bases = [_base_of(case, e) for e in ext]
    names = [n for n in STATE if n in bases[0].state]
    shapes = {n: [b.state[n].T.shape for b in bases] for n in names}

    def carve():
        whole, parts = {}, [{} for _ in bases]
        for n in names:
            sizes = [math.prod(s) for s in shapes[n]]
            whole[n] = _host((sum(sizes),))
            at = 0
            for p, s, z in zip(parts, shapes[n], sizes):
                p[n] = whole[n][at:at + z].view(s)
                at += z
        return whole, parts

    _, start = carve()
    for m, (b, s) in enumerate(zip(bases, start)):
        _initial(b, seed, m, s)
    whole, parts = carve() if out else (None, None)
    return bases, start, whole, parts


def _tendencies(base, seed):
    """What the host's physics leaves (a few K a day, small species sources)."""
    gen = torch.Generator().manual_seed(7 * seed + 5)
    d = base.dims
    shape = (d.kz, d.iy - 3, d.jx - 3)
    rand = lambda shape, s: s * torch.randn(shape, generator=gen, dtype=torch.float64)
    t = {"tten": rand(shape, 1e-4), "uten": rand(shape, 3e-4), "vten": rand(shape, 3e-4),
         "qxten": rand((d.nqx, *shape), 1e-9)}
    if d.ntr:
        t["chiten"] = rand((d.ntr, *shape), 1e-7)
    return t


def prepare(case, seed):
    form = case["form"]
    if form == "budget":
        return _prepare_budget(case, seed)
    bases, start, whole, parts = _members(case, seed)
    cases = [dataclasses.replace(b, state={**b.state, **_numpy_state(s)}) for b, s in zip(bases, start)]
    ins = [cs.Case.state_ptrs_of(_numpy_state({k: v for k, v in s.items() if k != "ps"})) for s in start]
    outs = [cs.Case.state_ptrs_of(_numpy_state(p)) for p in parts]
    st = {"form": form, "steps": case["steps"], "cases": cases, "keep": (start, parts), "ins": ins, "outs": outs,
          "whole": whole, "record": None}
    if case["precision"] == "mixed":
        st["record"] = {n: torch.empty(b.shape, dtype=torch.float32) for n, b in whole.items()}
    if form in ("segment", "coupled"):
        st["dom"] = domain_from_case(cases[0])
    elif form == "batch":
        st["batch"] = MolochBatch(cases)
    else:
        st["pool"] = MolochPool(cases[0].params, capacity=len(cases))
    if form == "coupled":
        st["tend"] = _tendencies(bases[0], seed)
        st["tend_ptrs"] = cs.Case.tend_ptrs_of(_numpy_state(st["tend"]))
        d = bases[0].dims
        st["seen"] = {n: _host((d.kz, d.iy - 1, d.jx - 1)) for n in ("t", "p", "rho", "qsat", "ux", "vx")}
        st["seen"]["qx"] = _host((d.nqx, d.kz, d.iy - 1, d.jx - 1))
        st["seen_ptrs"] = cs.Case.state_ptrs_of(_numpy_state(st["seen"]))
    return st


def _prepare_budget(case, seed):
    base = _base_of(case, _extents(case)[0])
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    put = lambda a: torch.from_numpy(a.T.copy()).to(dev)
    wobble = lambda a: a * (1.0 + 0.02 * (torch.rand(a.shape, generator=gen, device=dev, dtype=torch.float64) - 0.5))
    a = {n: wobble(put(base.state[n])) for n in ("rho", "qx", "u", "ps")}
    a["dz"] = put(base.static["dz"])
    a["v"] = torch.randn(base.state["v"].T.shape, generator=gen, device=dev, dtype=torch.float64)
    fn = abi.load().mlc_mass_budget_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.POINTER(abi.mlc_dims), C.c_double, C.c_double] + [C.c_void_p] * 8
    return {"form": "budget", "fn": fn, "dims": base.dims, "dx": base.params.dx, "dt": base.params.dtsec, "a": a,
            "out": torch.zeros(7, dtype=torch.float64, device=dev)}


# ---- one pass ----------------------------------------------------------------

def run(state):
    form = state["form"]
    if form == "budget":
        a = state["a"]
        abi.check(state["fn"](C.byref(state["dims"]), state["dx"], state["dt"],
                              *[a[n].data_ptr() for n in ("rho", "dz", "qx", "u", "v", "ps")],
                              state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream), "mass budget")
        return state["out"]
    if form == "segment":
        dom = state["dom"]
        dom.upload(state["ins"][0])
        dom.step(state["steps"])
        dom.download(state["outs"][0])
    elif form == "coupled":
        dom = state["dom"]
        dom.upload(state["ins"][0])
        for _ in range(state["steps"]):
            dom.step_dynamics()
            dom.download(state["seen_ptrs"])  # the state the host's physics reads
            dom.set_tendencies(state["tend_ptrs"])
            dom.step_finish()
        dom.download(state["outs"][0])
    elif form == "batch":
        batch = state["batch"]
        for m, p in enumerate(state["ins"]):
            batch.upload(m, p)
        batch.step(state["steps"])
        for m, p in enumerate(state["outs"]):
            batch.download(m, p)
    else:
        pool = state["pool"]
        slots = [pool.join(c) for c in state["cases"]]
        pool.step(state["steps"])
        for slot, p in zip(slots, state["outs"]):
            pool.download(slot, p)
            pool.leave(slot)
    if state["record"] is None:
        return state["whole"]
    for n, r in state["record"].items():
        r.copy_(state["whole"][n])
    return state["record"]


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """Bytes: per step every prognostic, metric and boundary-independent field
    of the path once in and the updated state once out.  Operations: the
    scheme's own arithmetic (WAF fluxes and updates of each field in three
    directions, the acoustic substeps), a multiply-add counting two."""
    if case["form"] == "budget":
        pts = case["nx"] * case["ny"] * case["kz"]
        return {"bytes": 8.0 * pts * 7, "flops": 14.0 * pts}
    moist = case["recipe"] == "moist"
    nqx = {2: 5, 3: 5, 4: 7, 5: 10}[case.get("ipptls") or 2] if moist else 2
    nf = 5 + (nqx if moist else 1) + (0 if moist else 1) + (1 if case.get("tke") else 0)
    coarse = case["form"] == "batch" or not moist
    nsound, nadv = case.get("nsound") or (3 if coarse else 4), case.get("nadv", 1)
    word = 8 if case["precision"] == "fp64" else 4
    pts = float(sum(x * y * k for x, y, k in _extents(case)))
    fields = 2 * nf + 2 * nqx + 18       # state in and out, metric, diagnostics
    flops = nadv * (98 * nf + 42 + nsound * 105) + 80
    return {"bytes": pts * case["steps"] * word * fields, "flops": pts * case["steps"] * flops}


# ---- the same in 64 bits, in plain torch -------------------------------------

GRAV, DEG, RADIUS = 9.80665, math.pi / 180.0, 6.371229e6
RGAS = ((6.02214076e23 * 1.3806490e-23) / 28.96454) * 1000.0
CPD, CVD, EP1, P00 = 3.5 * RGAS, 2.5 * RGAS, 28.96454 / 18.01528 - 1.0, 1.0e5
QCHECK = {0: 1.0e-8, 7: 1.0e10, 8: 100.0, 9: 0.01}  # floors of qv and of number concentrations


def exact(case, seed):
    if case["form"] == "budget":
        return _exact_budget(_prepare_budget(case, seed))
    points = sum(x * y * k for x, y, k in _extents(case)) * case["steps"]
    if points > (4e8 if torch.cuda.is_available() else 4e7) or case["form"] == "batch" and case["members"] > 16:
        return None  # more than some 20 seconds
    dev = torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")
    bases, start, _, _ = _members(case, seed, out=False)
    got = []
    for b, s in zip(bases, start):
        tend = _tendencies(b, seed) if case["form"] == "coupled" else None
        got.append(_Step(b, s, tend, dev).advance(case["steps"]))
    return {n: torch.cat([g[n].reshape(-1) for g in got]).cpu() for n in got[0]}


def _exact_budget(s):
    """Dry and water mass over the interior, their lateral fluxes over dt, and
    the extrema of surface pressure."""
    a, dx, dt = s["a"], s["dx"], s["dt"]
    m = a["dz"] * a["rho"]
    inner = m[:, 1:-1, 1:-1]
    q = a["qx"].sum(0)
    f = dt * dx * m
    west, east = a["u"][..., 0] * f[..., 0], a["u"][..., -1] * f[..., -1]
    south, north = a["v"][:, 0, 1:-1] * f[:, 0, 1:-1], a["v"][:, -1, 1:-1] * f[:, -1, 1:-1]
    qadv = ((q[..., 0] * west).sum() - (q[..., -1] * east).sum() + (q[:, 0, 1:-1] * south).sum()
            - (q[:, -1, 1:-1] * north).sum())
    ps = a["ps"][1:-1, 1:-1]
    return torch.stack([dx * dx * inner.sum(), west.sum() - east.sum() + south.sum() - north.sum(),
                        dx * dx * (q[:, 1:-1, 1:-1] * inner).sum(), qadv, ps.max(), ps.min(),
                        torch.zeros((), dtype=torch.float64, device=ps.device)])


def _to_cross(x, dim):
    """Staggered points to cross points: fourth order, second at the edges."""
    n = x.shape[dim] - 1
    at = lambda lo, num: x.narrow(dim, lo, num)
    mid = 0.5625 * (at(2, n - 2) + at(1, n - 2)) - 0.0625 * (at(3, n - 2) + at(0, n - 2))
    return torch.cat([0.5 * (at(0, 1) + at(1, 1)), mid, 0.5 * (at(n - 1, 1) + at(n, 1))], dim)


def _to_stag(x, dim):
    """Cross points to the staggered points between them."""
    n = x.shape[dim]
    at = lambda lo, num: x.narrow(dim, lo, num)
    mid = 0.5625 * (at(2, n - 3) + at(1, n - 3)) - 0.0625 * (at(3, n - 3) + at(0, n - 3))
    return torch.cat([0.5 * (at(0, 1) + at(1, 1)), mid, 0.5 * (at(n - 2, 1) + at(n - 1, 1))], dim)


def _waf(vel, zamu, up, a, c, num):
    """The weighted average flux of an interface with values a and c either
    side, Courant number zamu and upwind difference num."""
    den = c - a
    tiny = den.abs() < 1.0e-30
    r = torch.where(tiny, (num.abs() < 1.0e-30).double(), num / torch.where(tiny, torch.ones_like(den), den))
    b = torch.maximum(r, torch.minimum(2.0 * r, torch.ones_like(r))).clamp(0.0, 2.0)
    s = torch.where(up, 1.0, -1.0).to(den)
    phi = s + (zamu - s) * b
    return 0.5 * vel * ((1.0 + phi) * a + (1.0 - phi) * c)


class _Step:
    """The MOLOCH step of one domain; arrays are (k, i, j), the species first."""

    def __init__(self, base, start, tend, dev):
        p, st = base.params, base.static
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).to(dev)
        self.p, self.kz, self.nqx = p, base.dims.kz, base.dims.nqx
        self.x = {n: v.clone().to(dev) for n, v in start.items()}
        self.x["t"] = put(base.state["t"])
        self.x["w"][0] = 0.0
        self.tend = {n: v.to(dev) for n, v in (tend or {}).items()}
        self.b = {n: put(v[0]) for n, v in base.bdy.items()}  # b0 = b1
        self.m = {n: put(st[n]) for n in ("fmz", "fmzf", "rfmzu", "rfmzv", "zeta", "hx", "hy", "msfu", "msfv", "msfx")}
        col = lambda a: torch.as_tensor(np.asarray(a), device=dev).view(-1, 1, 1)
        kz, dzita = self.kz, float(st["zita"][self.kz - 1])
        k = np.arange(1, kz + 1)
        gz = lambda z: (lambda r: -p.mo_a0 * r - (3.0 - 2.0 * p.mo_a0) * r ** 2 + (2.0 - p.mo_a0) * r ** 3 + 1.0)(
            z / p.mo_ztop)
        self.gz, self.gzh, self.ff = col(gz(st["zita"])), col(gz(st["zitah"])), col(st["ffilt"])
        self.damp = col(0.125 * 0.85 * (1.0 / (k + 1.0) - 1.0 / (kz + 2.0)))
        self.filt = col(0.125 * (0.55 + 0.45 * (kz - k) / (kz - 1.0)))
        self.nudge = col(st["tnudge"]) * (p.dtsec / 7200.0)
        self.dta = p.dtsec / p.mo_nadv
        self.dts = self.dta / p.mo_nsound
        self.dtz = self.dts / dzita
        self.dtza = 0.5 * self.dta / dzita
        # relaxation weights of each grid's points (0 outside the zone)
        hefc = torch.cat([torch.zeros(kz, 1, dtype=torch.float64, device=dev), put(st["hefc"])], 1)
        zone = {n: put(st["ibnd_" + n]).long().clamp(min=0) for n in ("cr", "ud", "vd")}
        self.relax = {n: hefc[:, z] for n, z in zone.items()}
        fcx = torch.cat([torch.zeros(1, dtype=torch.float64, device=dev), put(st["fcx"])])
        self.relax_tr = fcx[zone["cr"]][1:-2, 1:-2]
        self.cor = {"u": 2 * 7.2921159e-5 * torch.sin(put(st["ulat"]) * DEG),
                    "v": 2 * 7.2921159e-5 * torch.sin(put(st["vlat"]) * DEG)}
        rlat = torch.from_numpy(st["rlat"].copy()).to(dev)
        mu, mv = self.m["msfu"], self.m["msfv"]
        if p.lrotllr:
            t = torch.sin(DEG * 0.5 * (rlat[1:-2] + rlat[2:-1]))[:, None] * self.m["msfx"][1:-2, 1:-2] / RADIUS
            self.curv = (t, t)
        else:
            self.curv = ((mu[1:-2, :-3] - mu[1:-2, 1:-2]) / p.dx, (mv[:-3, 1:-2] - mv[1:-2, 1:-2]) / p.dx)

    def advance(self, steps):
        for _ in range(steps):
            for _ in range(self.p.mo_nadv):
                s = self.sound()
                self.advect(s)
            self.end()
        return {n: self.x[n] for n in STATE if n in self.x}

    def sound(self):
        p, x, m, K = self.p, self.x, self.m, self.kz
        u, v, w, th, pi = x["u"], x["v"], x["w"], x["tetav"], x["pai"]
        dts, dtx, dtz, rd = self.dts, self.dts / p.dx, self.dtz, RGAS / CVD
        rot = p.lrotllr
        one = torch.ones_like
        mu, mv, mx = m["msfu"][:-1], m["msfv"][:, :-1], m["msfx"][:-1, :-1]
        rmu = one(mu) if rot else 1.0 / mu
        mf = mx if rot else mx * mx
        s = torch.zeros_like(w)
        I = (slice(None), slice(1, -1), slice(1, -1))
        tf = torch.zeros_like(w[I])
        tf[1:K] = 0.5 * (th[I][:-1] + th[I][1:])
        fz, fzf, thi = m["fmz"][I], m["fmzf"][I], th[I]
        hx, hy = m["hx"], m["hy"]

        def slope(a, b):  # terrain-following wind of the interior columns
            return (a[:, 1:-1, 1:-2] * hx[1:-1, 1:-2] + a[:, 1:-1, 2:-1] * hx[1:-1, 2:-1]
                    + b[:, 1:-2, 1:-1] * hy[1:-2, 1:-1] + b[:, 2:-1, 1:-1] * hy[2:-1, 1:-1])

        for n in range(p.mo_nsound):
            fu, fv = dtx * u * m["rfmzu"] * rmu, dtx * v * m["rfmzv"] / mv
            div = m["fmz"] * mf * ((fu[..., 1:] - fu[..., :-1]) + (fv[:, 1:] - fv[:, :-1]))
            s[1:K, 1:-1, 1:-1] = -0.25 * slope(u[1:] + u[:-1], v[1:] + v[:-1]) * self.gz[1:K]
            s[K:, 1:-1, 1:-1] = -0.5 * slope(u[K - 1:], v[K - 1:])
            w[K:, 1:-1, 1:-1] = -s[K:, 1:-1, 1:-1]
            zf = div[I].clone()
            if p.mo_divfilter:
                zf += self.filt * (div[:, 1:-1, :-2] + div[:, 1:-1, 2:] + div[:, :-2, 1:-1] + div[:, 2:, 1:-1]
                                   - 4.0 * div[I])
            zf += (1.0 - self.relax["cr"][:, 1:-2, 1:-2]) * dtz * fz * (s[I][:-1] - s[I][1:])
            wi, pii = w[I], pi[I]
            mult = torch.zeros_like(wi)
            for k in range(K - 1, 0, -1):
                tf[k] -= wi[k] * fzf[k] * dtz * (thi[k - 1] - thi[k])
                z = CPD * tf[k] * fzf[k]
                we = wi[k] - z * dtz * (pii[k - 1] - pii[k]) - GRAV * dts
                we = we + rd * z * dtz * (pii[k - 1] * zf[k - 1] - pii[k] * zf[k])
                zu = dtz * dtz * rd * fz[k - 1] * z * pii[k - 1] + self.ff[k]
                zd = dtz * dtz * rd * fz[k] * z * pii[k] + self.ff[k]
                piv = 1.0 / (1.0 + zd + zu - zd * mult[k + 1])
                wi[k] = piv * (we + zd * wi[k + 1])
                mult[k] = piv * zu
            for k in range(1, K):
                wi[k] += mult[k] * wi[k - 1]
            pii *= 1.0 - rd * (zf + dtz * fz * (wi[:-1] - wi[1:]))
            un, vn = u.clone(), v.clone()
            ui, vi = un[:, 1:-1, 1:-1], vn[:, 1:-1, 1:-1]
            if p.mo_divdamp:
                d = p.dx / dts * self.damp
                ui += d * mu[1:-1, 1:-1] * (div[:, 1:-1, 1:] - div[:, 1:-1, :-1])
                vi += d * (1.0 if rot else mv[1:-1, 1:-1]) * (div[:, 1:, 1:-1] - div[:, :-1, 1:-1])
            gh = GRAV * dts * self.gzh
            ui += (1.0 - self.relax["ud"][:, 1:-2, 1:-1]) * (
                self.cor["u"][1:-1, 1:-1] * dts * v[:, 1:-2, 1:] - gh * hx[1:-1, 1:-1]
                - dtx * mu[1:-1, 1:-1] * 0.5 * CPD * (th[:, 1:-1, :-1] + th[:, 1:-1, 1:])
                * (pi[:, 1:-1, 1:] - pi[:, 1:-1, :-1]))
            vi += (1.0 - self.relax["vd"][:, 1:-1, 1:-2]) * (
                -self.cor["v"][1:-1, 1:-1] * dts * u[:, 1:, 1:-2] - gh * hy[1:-1, 1:-1]
                - dtx * (1.0 if rot else mv[1:-1, 1:-1]) * 0.5 * CPD * (th[:, :-1, 1:-1] + th[:, 1:, 1:-1])
                * (pi[:, 1:, 1:-1] - pi[:, :-1, 1:-1]))
            u, v = un, vn
        s[1:K] = (w[1:K] + s[1:K]) * m["fmzf"][1:K]
        s[1:K, 0], s[1:K, -1], s[1:K, :, 0], s[1:K, :, -1] = 0.0, 0.0, 0.0, 0.0
        s[0], s[K] = 0.0, 0.0
        x["u"], x["v"] = u, v
        return s

    def advect(self, s):
        x, p = self.x, self.p
        ux, vx, wx = _to_cross(x["u"], 2), _to_cross(x["v"], 1), _to_cross(x["w"], 0)
        tx = _to_cross(x["tke"], 0) if p.ibltyp == 2 else None
        coef = self.coefficients(s)
        go = lambda f: self.waf3(f, coef)
        th, pi = go(x["tetav"]), go(x["pai"])
        nq = self.nqx if p.ipptls > 0 else 1
        q = x["qx"].clone()
        for n in range(nq):
            q[n] = go(x["qx"][n])
        ux, vx, wx = go(ux), go(vx), go(wx)
        if tx is not None:
            tx = go(tx)
        if "trac" in x:
            x["trac"] = torch.stack([go(f) for f in x["trac"]])
        a, b = ux[:, 1:-1, 1:-1], vx[:, 1:-1, 1:-1]
        a += a * b * self.curv[0] * self.dta
        b -= a * a * self.curv[1] * self.dta
        x["tetav"], x["pai"], x["qx"] = th, pi, q
        x["u"][:, 1:-1, 1:-1] = _to_stag(ux, 2)[:, 1:-1]
        x["v"][:, 1:-1, 1:-1] = _to_stag(vx, 1)[..., 1:-1]
        x["w"][1:-1] = _to_stag(wx, 0)
        if tx is not None:
            x["tke"][1:-1] = _to_stag(tx, 0)

    def coefficients(self, s):
        m, p, x = self.m, self.p, self.x
        u, v, rot = x["u"], x["v"], p.lrotllr
        zu, zd = self.dtza * m["fmz"] / m["fmzf"][:-1], self.dtza * m["fmz"] / m["fmzf"][1:]
        c = {"s": s[1:-1], "zu": zu, "zd": zd, "dvz": s[:-1] * zu - s[1:] * zd}
        dt = self.dta / p.dx
        mu, mv, mx = m["msfu"][:-1], m["msfv"][:, :-1], m["msfx"][:-1, :-1]
        c["vf"], c["uf"] = v[:, 1:-1], u[:, 1:-1, 1:-1]
        c["cy"] = c["vf"] * dt * (1.0 if rot else mv[1:-1])
        c["cx"] = c["uf"] * dt * mu[1:-1, 1:-1]
        fz = m["fmz"][:, 1:-1]
        fi, fn = (m["rfmzv"][:, 1:-2], m["rfmzv"][:, 2:-1]) if rot else (m["rfmzu"][:, 1:-1, :-1], m["rfmzu"][:, 2:, :-1])
        ri, rn = 1.0 / mv[1:-2], 1.0 / mv[2:-1]
        mr = mx[1:-1]
        vi, vn = v[:, 1:-2], v[:, 2:-1]
        ui, ue = u[:, 1:-1, 1:-2], u[:, 1:-1, 2:-1]
        fw, fe = m["rfmzu"][:, 1:-1, 1:-2], m["rfmzu"][:, 1:-1, 2:-1]
        if rot:
            c["zs"], c["zn"] = dt * ri * mr * fz * fi, dt * rn * mr * fz * fn
            c["dvy"] = vn * c["zn"] - vi * c["zs"]
            c["my"] = c["mx"] = 1.0
            c["zw"], c["ze"] = dt * mr[:, 1:-1] * fz[..., 1:-1] * fw, dt * mr[:, 1:-1] * fz[..., 1:-1] * fe
            c["dvx"] = ue * c["ze"] - ui * c["zw"]
        else:
            c["zs"], c["zn"] = dt * fz * fi, dt * fz * fn
            c["dvy"] = vn * rn * c["zn"] - vi * ri * c["zs"]
            c["my"], c["mx"] = mr * mr, (mr * mr)[:, 1:-1]
            c["zw"], c["ze"] = dt * fz[..., 1:-1] * fw, dt * fz[..., 1:-1] * fe
            c["dvx"] = ue / mu[1:-1, 2:-1] * c["ze"] - ui / mu[1:-1, 1:-2] * c["zw"]
        return c

    def waf3(self, f, c):
        """Two vertical passes, the meridional pass, the zonal pass."""
        q = f
        zero = torch.zeros_like(f[:1])
        for _ in range(2):
            d = q[:-1] - q[1:]
            zamu = c["s"] * self.dtza
            up = zamu >= 0
            num = torch.where(up, torch.cat([d[1:], zero]), torch.cat([zero, d[:-1]]))
            fl = torch.cat([zero, _waf(c["s"], zamu, up, q[1:], q[:-1], num), zero])
            q = q - fl[:-1] * c["zu"] + fl[1:] * c["zd"] + c["dvz"] * q
        d = q[:, 1:] - q[:, :-1]
        up = c["cy"] > 0
        num = torch.where(up, torch.cat([torch.zeros_like(d[:, :1]), d[:, :-1]], 1), torch.cat([d[:, 1:], d[:, -1:]], 1))
        fy = _waf(c["vf"], c["cy"], up, q[:, :-1], q[:, 1:], num)
        r = q[:, 1:-1] + c["my"] * (fy[:, :-1] * c["zs"] - fy[:, 1:] * c["zn"] + c["dvy"] * f[:, 1:-1])
        d = r[..., 1:] - r[..., :-1]
        up = c["cx"] > 0
        num = torch.where(up, torch.cat([torch.zeros_like(d[..., :1]), d[..., :-1]], 2),
                          torch.cat([d[..., 1:], d[..., -1:]], 2))
        fx = _waf(c["uf"], c["cx"], up, r[..., :-1], r[..., 1:], num)
        out = f.clone()
        out[:, 1:-1, 1:-1] = r[..., 1:-1] + c["mx"] * (fx[..., :-1] * c["zw"] - fx[..., 1:] * c["ze"]
                                                       + c["dvx"] * f[:, 1:-1, 1:-1])
        return out

    def qfactor(self, q):
        n = 5 if self.p.ipptls > 1 else 2 if self.p.ipptls == 1 else 1
        return 1.0 + EP1 * q[0] - q[1:n].sum(0)

    def floors(self):
        for n in range(self.nqx):
            q = self.x["qx"][n][:, 1:-1, 1:-1]
            q[q < QCHECK.get(n, 1.0e-16)] = QCHECK.get(n, 0.0)
        if "trac" in self.x:
            q = self.x["trac"][..., 1:-1, 1:-1]
            q[q < 1.0e-50] = 0.0

    def end(self):
        self.ring()
        x, p, b = self.x, self.p, self.b
        I = (Ellipsis, slice(1, -1), slice(1, -1))
        x["t"][I] = (x["tetav"] * x["pai"] / self.qfactor(x["qx"]))[I]
        if p.mo_top_nudge:
            x["w"][1][I] *= 1.0 - p.dtsec / 900.0

        def pull(f, fext, wgt):
            f[I] += wgt * (fext[I] - f[I])

        hcr = self.relax["cr"][:, 1:-2, 1:-2]
        for n, ext, wgt in (("u", "dub", self.relax["ud"][:, 1:-2, 1:-1]), ("v", "dvb", self.relax["vd"][:, 1:-1, 1:-2]),
                            ("t", "xtb", hcr)):
            if p.mo_top_nudge:
                pull(x[n], b[ext], self.nudge)
            pull(x[n], b[ext], wgt)
        pull(x["pai"], b["xpaib"], hcr)
        pull(x["qx"][0], b["xqb"], hcr)
        if p.present_qc and p.ipptls > 0:
            pull(x["qx"][1], b["xlb"], hcr)
        if p.present_qi and p.ipptls > 1:
            pull(x["qx"][2], b["xib"], hcr)
        x["w"][:-1][I] *= 1.0 - hcr
        if "trac" in x:
            pull(x["trac"], b["chib"], self.relax_tr)
        ux, vx = _to_cross(x["u"], 2), _to_cross(x["v"], 1)
        z1, z2 = self.m["zeta"][-2], self.m["zeta"][-1]
        tv = x["t"] * self.qfactor(x["qx"])
        lr = (tv[-2] - tv[-1]) / (z1 - z2)
        lr = torch.where(lr < -GRAV / CPD, torch.full_like(lr, -GRAV / CPD),
                         torch.where(lr > -0.005, 0.65 * lr - 0.35 * 0.00649, lr))
        ps = P00 * x["pai"][-1] ** 3.5 * torch.exp(GRAV / RGAS * z2 / (tv[-1] - lr * 0.5 * z2))
        x["ps"][I] = ps[I]
        self.floors()
        if self.tend:
            dt = p.dtsec
            x["t"][I] += dt * self.tend["tten"]
            ux[I] += dt * self.tend["uten"]
            vx[I] += dt * self.tend["vten"]
            x["qx"][I] += dt * self.tend["qxten"]
            if "trac" in x:
                x["trac"][I] += dt * self.tend["chiten"]
            self.floors()
        x["tetav"] = x["t"] * self.qfactor(x["qx"]) / x["pai"]
        if p.ibltyp == 2:
            x["tke"][I] = x["tke"][I].clamp(min=1.0e-3)
        x["u"][I] = _to_stag(ux, 2)[:, 1:-1]
        x["v"][I] = _to_stag(vx, 1)[..., 1:-1]

    def ring(self):
        """Boundary values on the outermost points; species without boundary
        data, w and TKE take their floor on inflow and the interior value on
        outflow (west and east first, then the rows with the corners)."""
        x, b, p, K = self.x, self.b, self.p, self.kz
        sides = [(2, 0), (2, -1), (1, 0), (1, -1)]
        for n, ext in (("u", "dub"), ("v", "dvb"), ("t", "xtb"), ("pai", "xpaib"), ("ps", "xpsb"), ("trac", "chib")):
            if n in x and ext in b:
                for edge in ((Ellipsis, 0), (Ellipsis, -1), (Ellipsis, 0, slice(None)), (Ellipsis, -1, slice(None))):
                    x[n][edge] = b[ext][edge]
        given = {0: "xqb"}
        if p.present_qc:
            given[1] = "xlb"
        if p.present_qi and p.ipptls > 1:
            given[2] = "xib"
        for dim, end in sides:
            wind = (b["dub"] if dim == 2 else b["dvb"]).select(dim, end)
            inside = slice(1, -1) if dim == 2 else slice(None)
            inflow = (wind > 0 if end == 0 else wind < 0)[:, inside]
            edge = lambda f: f.select(dim, end)[:, inside]
            near = lambda f: f.select(dim, 1 if end == 0 else -2)[:, inside]
            for n in range(self.nqx):
                f = x["qx"][n]
                edge(f).copy_(edge(b[given[n]]) if n in given
                              else torch.where(inflow, QCHECK.get(n, 0.0), near(f)))
            w = x["w"][:K]
            edge(w).copy_(torch.where(inflow, 0.0, near(w)))
            if p.ibltyp == 2:
                both = wind[1:] + wind[:-1]
                inflow = (both > 0 if end == 0 else both < 0)[:, inside]
                f = x["tke"]
                edge(f[:1]).fill_(1.0e-3)
                edge(f[2:]).copy_(torch.where(inflow, 1.0e-3, near(f[2:])))
