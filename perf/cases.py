"""The work this framework is timed on, through its public entry points.

Whole time steps of the lid-driven cavity (FlowSolver.step) in both multigrid
precisions from the smallest benchmark size to the largest, an ensemble of
mixed sizes stepped together, the pressure Poisson solve alone (Multigrid.solve,
one V-cycle of the harness form, and the C entry for hosts that cannot
allocate), and the device passes of one Runge-Kutta stage called one by one,
as a sub-domain of a decomposed case and a C host call them.

Every case steps or solves a lid-driven cavity of Reynolds number 100..1000 and
lid velocity 0.5..1.5 (the benchmark ensemble's ranges).  A step starts from a
weak vortex with 1 % noise and a smooth pressure.  ``exact`` restates the
reference's arithmetic in torch FP64, pass by pass, without this package.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "warpflow-les_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from warpflow import FlowSolver, Multigrid, _abi, build_topology  # noqa: E402
from warpflow.ensemble import Ensemble, cavity_case  # noqa: E402
from warpflow.fields import DeviceField  # noqa: E402

NPL = 3
DEV = "cuda:0"
ENSEMBLE_SIZES = "32,32,32,48,48,48,64,64,80,80,96,96"


def listed():
    return [
        # the smallest benchmark cavity: fixed dt, every launch a few thousand cells
        {"name": "step32_fp64", "kind": "step", "n": 32, "levels": 3,
         "precision": "fp64", "variable_dt": False},
        # a size that is not a power of two times five: coarsest level 18^3
        {"name": "step72_fp64", "kind": "step", "n": 72, "levels": 3,
         "precision": "fp64", "variable_dt": True},
        # the headline cavity, in both multigrid precisions
        {"name": "step80_fp64", "kind": "step", "n": 80, "levels": 3,
         "precision": "fp64", "variable_dt": True},
        {"name": "step80_mixed", "kind": "step", "n": 80, "levels": 3,
         "precision": "mixed", "variable_dt": True},
        # the largest served request, at the depth the server gives it
        {"name": "step128_mixed", "kind": "step", "n": 128, "levels": 4,
         "precision": "mixed", "variable_dt": True},
        # the large cavity, in both multigrid precisions
        {"name": "step256_fp64", "kind": "step", "n": 256, "levels": 5,
         "precision": "fp64", "variable_dt": True},
        {"name": "step256_mixed", "kind": "step", "n": 256, "levels": 5,
         "precision": "mixed", "variable_dt": True},
        # a parameter study: cases of the benchmark ensemble's sizes, one batch step
        {"name": "ensemble12_mixed", "kind": "ensemble", "sizes": ENSEMBLE_SIZES,
         "precision": "mixed"},
        # the pressure solver alone: the standalone 256^3 problem, and one V-cycle
        # on the harness arrays at the headline size
        {"name": "poisson256_fp64", "kind": "poisson", "n": 256, "levels": 5,
         "precision": "fp64"},
        {"name": "vcycle80_fp64", "kind": "vcycle", "n": 80, "levels": 3,
         "precision": "fp64"},
        # a C host without device allocation solves its pressure equation
        {"name": "noalloc96_fp64", "kind": "noalloc", "n": 96, "levels": 3,
         "precision": "fp64"},
        # one Runge-Kutta stage pass by pass (a sub-domain's or a C host's order)
        {"name": "stage100_fp64", "kind": "stage", "n": 100, "levels": 3,
         "precision": "fp64"},
    ]


def draw(rng):
    """A case of the same ranges: steps of 24..256 cells per axis in either
    precision, small ensembles, solves, V-cycles and stages."""
    kind = rng.choice(["step", "step", "step", "ensemble", "poisson", "vcycle", "noalloc",
                       "stage"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "ensemble":
        sizes = sorted(8 * rng.randint(3, 12) for _ in range(rng.randint(2, 12)))
        return {"kind": kind, "sizes": ",".join(map(str, sizes)), "precision": prec}
    if kind == "stage":
        return {"kind": kind, "n": 4 * round(math.exp(rng.uniform(math.log(6), math.log(60)))),
                "levels": 3, "precision": "fp64"}
    if kind == "noalloc":
        return {"kind": kind, "n": 8 * rng.randint(3, 14), "levels": 3, "precision": "fp64"}
    n = math.exp(rng.uniform(math.log(24), math.log(250)))
    if n < 100:
        n, levels = 8 * round(n / 8), 3
    elif n < 176:
        n = 16 * round(n / 16)
        levels = rng.choice([3, 4]) if n <= 128 else 4
    else:
        n, levels = 32 * round(n / 32), 5
    case = {"kind": kind, "n": n, "levels": levels, "precision": prec}
    if kind == "step":
        case["variable_dt"] = rng.random() < 0.7
    return case


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _physics(seed):
    """Reynolds number and lid velocity of a seed (benchmark ensemble ranges)."""
    r = random.Random(seed)
    return r.uniform(100.0, 1000.0), r.uniform(0.5, 1.5)


def _flow(n, seed, lid):
    """Real-cell u, v, w, p of a cavity in motion: a vortex a fifth of the lid
    velocity strong, varying along y, with 1 % noise, and a smooth pressure."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    ph = torch.rand(3, generator=g, device=DEV, dtype=torch.float64)
    c = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n
    f = (torch.arange(n, device=DEV, dtype=torch.float64) + 1.0) / n
    y = 1.0 + 0.2 * torch.cos(2 * math.pi * (c + ph[0]))[None, :, None]
    a = 0.2 * lid
    u = -a * (torch.sin(math.pi * f) ** 2)[:, None, None] * y * \
        torch.sin(2 * math.pi * c)[None, None, :]
    w = a * torch.sin(2 * math.pi * c)[:, None, None] * y * \
        (torch.sin(math.pi * f) ** 2)[None, None, :]
    v = torch.zeros_like(u)
    noise = [0.01 * (2.0 * torch.rand((n, n, n), generator=g, device=DEV,
                                      dtype=torch.float64) - 1.0) for _ in range(3)]
    p = 0.05 * lid * lid * torch.cos(math.pi * (c + ph[1]))[:, None, None] * y * \
        torch.cos(math.pi * (c + ph[2]))[None, None, :]
    return u + noise[0], v + noise[1], w + noise[2], p


def _core(t):
    return t[NPL:-NPL, NPL:-NPL, NPL:-NPL]


def _solver_inputs(sol, seed, lid):
    for name, x in zip(("u", "v", "w", "p"), _flow(sol.n, seed, lid)):
        _core(sol.f[name].t).copy_(x)
    for name in ("u", "v", "w"):
        sol.fill_bc(name)
    sol.bcs.apply_pbound(sol.f["p"], sol.n)


def _cfg(n, levels, precision, seed, variable_dt=True):
    re, lid = _physics(seed)
    return cavity_case(n, re, lid, levels=levels, precision=precision,
                       variable_dt=variable_dt, noise=0.0), lid


def _rhs(n, seed):
    """N(0, 1) on the real cells, mean removed."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = torch.randn((n, n, n), generator=g, device=DEV, dtype=torch.float64)
    return r - r.mean()


def _padded(n, core, npl):
    t = torch.zeros((n + 2 * npl,) * 3, dtype=torch.float64, device=DEV)
    t[npl:-npl, npl:-npl, npl:-npl] = core
    return t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        cfgs, lids = [], []
        for q, n in enumerate(int(x) for x in case["sizes"].split(",")):
            cfg, lid = _cfg(n, 3, case["precision"], seed * 64 + q)
            cfgs.append(cfg)
            lids.append(lid)
        ens = Ensemble(cfgs, DEV)
        for q, sol in enumerate(ens.solvers):
            _solver_inputs(sol, seed * 64 + q, lids[q])
        return {"kind": kind, "ens": ens}
    n, levels = case["n"], case["levels"]
    if kind in ("step", "stage"):
        cfg, lid = _cfg(n, levels, case["precision"], seed, case.get("variable_dt", True))
        sol = FlowSolver(cfg, build_topology(cfg), DEV)
        _solver_inputs(sol, seed, lid)
        if kind == "stage":
            _abi.call("wf_copy_oo", ctypes.byref(sol.case), sol._stream())
        return {"kind": kind, "sol": sol}
    h = 1.0 / n
    if kind == "noalloc":
        return {"kind": kind, "n": n, "levels": levels, "h": h,
                "su": _padded(n, _rhs(n, seed), NPL), "pp": _padded(n, 0.0, NPL)}
    cfg, _ = _cfg(n, levels, case["precision"], seed)
    mg = Multigrid(cfg, build_topology(cfg), DEV, h, h, h)
    if kind == "poisson":
        return {"kind": kind, "mg": mg, "su": DeviceField(_padded(n, _rhs(n, seed), NPL)),
                "pp": DeviceField(_padded(n, 0.0, NPL))}
    mg.levels[0].rhs.t.copy_(_padded(n, _rhs(n, seed), 1))
    mg.levels[0].phi.zero_()
    return {"kind": "vcycle", "mg": mg}


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _stage(sol):
    """The device passes of one Runge-Kutta stage (alpha = 1/2) and the
    divergence, in a sub-domain's order."""
    c, s = ctypes.byref(sol.case), sol._stream()
    dt = ctypes.c_void_p(sol._sc.data_ptr() + _abi.WfScalars.dt.offset)
    _abi.call("wf_wale_vis", c, s)
    for op in ("wf_conv", "wf_diff"):
        for comp, name in enumerate("uvw"):
            sol.fill_bc(name)
            _abi.call(op, c, comp, 0.5, dt, s)
    _abi.call("wf_calvel", c, 0.5, dt, s)
    _abi.call("wf_calmas", c, s)
    return {k: sol.f[k].t for k in ("ustar", "vstar", "wstar", "u", "v", "w", "vis", "su")}


def run(state):
    kind = state["kind"]
    if kind == "step":
        sol = state["sol"]
        info = sol.step()
        # rmax is left out: it is the rounding-level rest of a cancellation
        return {**{k: sol.f[k].t for k in ("u", "v", "w", "p", "vis")},
                "dt": info["dt"], "ctime": info["ctime"], "iters": info["iters"]}
    if kind == "ensemble":
        ens = state["ens"]
        infos = ens.step()
        for x in infos:
            if isinstance(x, Exception):
                raise x
        return {"cases": [[sol.f[k].t for k in ("u", "v", "w", "p", "vis")]
                          for sol in ens.solvers],
                "dt": np.array([x["dt"] for x in infos]),
                "iters": np.array([x["iters"] for x in infos])}
    if kind == "poisson":
        state["mg"].solve(state["su"], state["pp"], NPL)
        return state["pp"].t
    if kind == "vcycle":
        state["mg"]._vcycle()
        return state["mg"].levels[0].phi.t
    if kind == "noalloc":
        h = state["h"]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _abi.call("wf_mg_solve_noalloc", state["su"].data_ptr(), state["pp"].data_ptr(),
                  state["n"], state["levels"], h, h, h, stream)
        return state["pp"]
    return _stage(state["sol"])


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _vcycle_flops(n, levels):
    """6 + 6 sweeps per level and 300 on the coarsest at 13 operations a cell,
    residual and restriction 16, prolongation 16."""
    fl = 0.0
    for l in range(levels - 1):
        fl += (12 * 13 + 32) * float(n >> l) ** 3
    return fl + 300 * 13 * float(n >> (levels - 1)) ** 3


# additions, multiplications and divisions a cell of convection and diffusion
# (three components), WALE, velocity correction, divergence and dt control
_STAGE_FLOPS = 3 * (100 + 35)
_POINT_FLOPS = {"wale": 150, "calvel": 12, "calmas": 22, "dt": 16}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        parts = [work({"kind": "step", "n": int(x), "levels": 3}) for x in
                 case["sizes"].split(",")]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, levels = case["n"], case["levels"]
    cells = float(n) ** 3
    p = _POINT_FLOPS
    if kind == "step":
        # u, v, w, p, vis in and out; one multigrid solve and two divergences
        fl = 2 * _STAGE_FLOPS + p["wale"] + 3 * p["calvel"] + 2 * p["calmas"] + p["dt"]
        return {"bytes": 10 * 8 * cells, "flops": fl * cells + 4 * _vcycle_flops(n, levels)}
    if kind == "stage":
        fl = _STAGE_FLOPS + p["wale"] + p["calvel"] + p["calmas"]
        return {"bytes": 15 * 8 * cells, "flops": fl * cells}
    if kind == "vcycle":
        return {"bytes": 3 * 8 * cells, "flops": _vcycle_flops(n, levels)}
    return {"bytes": 2 * 8 * cells, "flops": 4 * _vcycle_flops(n, levels)}


# --------------------------------------------------------------------------
# the same arithmetic in torch FP64
# --------------------------------------------------------------------------
def _set_face(f, axis, layers, value, src=None, sign=1.0, a=None, b=None):
    """Ghost layers `layers` of `axis` over the box a x b of the other axes:
    a constant, or sign times the layers `src`, one after the other."""
    other = [d for d in range(3) if d != axis]
    idx = [None, None, None]
    idx[other[0]], idx[other[1]] = slice(*a), slice(*b)
    for m, g in enumerate(layers):
        idx[axis] = g
        if src is None:
            f[tuple(idx)] = value
        else:
            to = tuple(idx)
            idx[axis] = src[m]
            f[to] = sign * f[tuple(idx)]


def _fill(f, kind, n, value=0.0):
    """The reference's ordered ghost fills of u, v, w, vis and p."""
    lo, hi, last = NPL - 1, NPL + n, NPL + n - 1
    full, cut = (lo, lo + n + 2), (lo, lo + n + 1)
    low3, low_src = [lo, lo - 1, lo - 2], [NPL, NPL + 1, NPL + 2]
    up3, up_src = [hi, hi + 1, hi + 2], [last, last - 1, last - 2]
    wall3 = [last, hi, hi + 1]
    if kind == "u":
        box = dict(a=cut, b=full)
        _set_face(f, 0, low3, 0.0, a=full, b=full)
        _set_face(f, 0, wall3, 0.0, a=full, b=full)
        _set_face(f, 1, low3, None, low_src, **box)
        _set_face(f, 1, up3, None, up_src, **box)
        _set_face(f, 2, low3, None, low_src, -1.0, **box)
        _set_face(f, 2, up3, value, **box)
    elif kind == "v":
        box = dict(a=cut, b=full)
        _set_face(f, 0, low3, None, low_src, -1.0, **box)
        _set_face(f, 0, up3, None, up_src, -1.0, **box)
        _set_face(f, 1, low3, 0.0, a=full, b=full)
        _set_face(f, 1, wall3, 0.0, a=full, b=full)
        box = dict(a=full, b=cut)
        _set_face(f, 2, low3, None, low_src, -1.0, **box)
        _set_face(f, 2, up3, None, up_src, **box)
    elif kind == "w":
        box = dict(a=full, b=cut)
        _set_face(f, 0, low3, None, low_src, -1.0, **box)
        _set_face(f, 0, up3, None, up_src, -1.0, **box)
        _set_face(f, 1, low3, None, low_src, **box)
        _set_face(f, 1, up3, None, up_src, **box)
        _set_face(f, 2, low3, 0.0, a=full, b=full)
        _set_face(f, 2, wall3, 0.0, a=full, b=full)
    elif kind == "vis":
        box = dict(a=full, b=full)
        _set_face(f, 0, [NPL], value, **box)
        _set_face(f, 0, [lo], None, [NPL], **box)
        _set_face(f, 0, [last], value, **box)
        _set_face(f, 0, [hi], None, [last], **box)
        _set_face(f, 1, [lo], None, [NPL], **box)
        _set_face(f, 1, [hi], None, [last], **box)
        _set_face(f, 2, [NPL], value, **box)
        _set_face(f, 2, [lo], None, [NPL], **box)
        _set_face(f, 2, [hi], None, [last], **box)
    else:
        box = dict(a=(lo, lo + n + 3), b=(lo, lo + n + 3))
        for axis in range(3):
            _set_face(f, axis, [lo], None, [NPL], **box)
            _set_face(f, axis, [hi], None, [last], **box)


def _at(f, dims, off):
    return f[tuple(slice(NPL + o, NPL + o + d) for o, d in zip(off, dims))]


def _shift(off, axis, m):
    o = list(off)
    o[axis] += m
    return o


def _interp(f, dims, off, axis):
    g = [_at(f, dims, _shift(off, axis, m)) for m in (1, 0, -1, -2)]
    return (-g[0] + 9.0 * g[1] + 9.0 * g[2] - g[3]) / 16.0


def _advance(f, n, h, dt, alpha, comp):
    """star = old - dt alpha convection of one component."""
    vel = [f["u"], f["v"], f["w"]]
    dims = [n, n, n]
    dims[comp] = n - 1
    one = [0, 0, 0]
    one[comp] = 1
    total = 0.0
    for axis in range(3):
        flux = []
        for m in (2, 1, 0, -1):
            if axis == comp:
                flux.append(_interp(vel[comp], dims, _shift((0, 0, 0), axis, m), axis) ** 2)
            else:
                flux.append(_interp(vel[comp], dims, _shift((0, 0, 0), axis, m), axis)
                            * _interp(vel[axis], dims, _shift(one, axis, m - 1), comp))
        total = total + (-flux[0] + 27.0 * flux[1] - 27.0 * flux[2] + flux[3]) / (24.0 * h)
    name = "uvw"[comp]
    _at(f[name + "star"], dims, (0, 0, 0)).copy_(
        _at(f[name + "oo"], dims, (0, 0, 0)) - dt * alpha * total)


def _diffuse(f, n, h, dt, alpha, comp):
    name = "uvw"[comp]
    dims = [n, n, n]
    dims[comp] = n - 1
    c = f[name]
    lap = 0.0
    for axis in range(3):
        g = [_at(c, dims, _shift((0, 0, 0), axis, m)) for m in (2, 1, 0, -1, -2)]
        lap = lap + (-g[0] + 16.0 * g[1] - 30.0 * g[2] + 16.0 * g[3] - g[4]) / (12.0 * h * h)
    off = [0, 0, 0]
    if comp:
        off[comp] = 1
    star = _at(f[name + "star"], dims, (0, 0, 0))
    star.copy_(star + dt * alpha * (_at(f["vis"], dims, off) * lap))


def _correct(f, n, h, dt, alpha):
    for comp in range(3):
        name = "uvw"[comp]
        dims = [n, n, n]
        dims[comp] = n - 1
        grad = _at(f["p"], dims, _shift((0, 0, 0), comp, 1)) - _at(f["p"], dims, (0, 0, 0))
        _at(f[name], dims, (0, 0, 0)).copy_(
            _at(f[name + "star"], dims, (0, 0, 0)) - dt * alpha * grad / h)


def _divergence(f, n, h, dt):
    div = 0.0
    dims = [n, n, n]
    for comp in range(3):
        g = [_at(f["uvw"[comp]], dims, _shift((0, 0, 0), comp, m)) for m in (1, 0, -1, -2)]
        div = div + (-g[0] + 27.0 * g[1] - 27.0 * g[2] + g[3]) / (24.0 * h)
    _core(f["su"]).copy_(div / dt)
    return float((div * h * h * h).abs().max())


def _eddy_viscosity(f, n, h, rrey):
    dims = [n, n, n]
    vel = [f["u"], f["v"], f["w"]]
    g = [[None] * 3 for _ in range(3)]
    for a in range(3):
        for b in range(3):
            q = vel[a]
            if a == b:
                g[a][b] = (_at(q, dims, (0, 0, 0)) - _at(q, dims, _shift((0, 0, 0), a, -1))) / h
            else:
                up, dn = _shift((0, 0, 0), b, 1), _shift((0, 0, 0), b, -1)
                g[a][b] = 0.25 * (_at(q, dims, up) + _at(q, dims, _shift(up, a, -1))
                                  - _at(q, dims, dn) - _at(q, dims, _shift(dn, a, -1))) / h
    g2 = [[sum(g[a][c] * g[c][b] for c in range(3)) for b in range(3)] for a in range(3)]
    # the reference's last terms of zx and zy are dw/dz du/dz and dw/dz du/dy
    g2[2][0] = g[2][0] * g[0][0] + g[2][1] * g[1][0] + g[2][2] * g[0][2]
    g2[2][1] = g[2][0] * g[0][1] + g[2][1] * g[1][1] + g[2][2] * g[0][1]
    tr = (g2[0][0] + g2[1][1] + g2[2][2]) / 3.0
    sdsd = ss = 0.0
    for a in range(3):
        sdsd = sdsd + (g2[a][a] - tr) ** 2
        ss = ss + g[a][a] ** 2
        for b in range(a):
            sdsd = sdsd + 2.0 * (0.5 * (g2[a][b] + g2[b][a])) ** 2
            ss = ss + 2.0 * (0.5 * (g[a][b] + g[b][a])) ** 2
    ls = 0.46 * (h * h * h) ** (1.0 / 3.0)
    den = ss.abs() ** 2.5 + sdsd ** 1.25
    nut = torch.where(sdsd > 1.0e-8, ls * ls * sdsd ** 1.5 / den, torch.zeros_like(sdsd))
    _core(f["vis"]).copy_(rrey + nut)
    _fill(f["vis"], "vis", n, rrey)


class _Level:
    """One level of the 7-point Neumann problem: phi and rhs with one ring."""

    def __init__(self, n, h):
        self.n = n
        self.phi = torch.zeros((n + 2,) * 3, dtype=torch.float64, device=DEV)
        self.rhs = torch.zeros_like(self.phi)
        lo = torch.full((n,), 1.0 / (h * h), dtype=torch.float64, device=DEV)
        hi = lo.clone()
        lo[0] = 0.0
        hi[-1] = 0.0
        self.c = [(x.view([n if d == a else 1 for d in range(3)])) for a in range(3)
                  for x in (lo, hi)]
        self.ap = -(self.c[0] + self.c[1] + self.c[2] + self.c[3] + self.c[4] + self.c[5])
        k = torch.arange(n, device=DEV)
        odd = (k[:, None, None] + k[None, :, None] + k[None, None, :]) % 2 == 1
        self.mask = [odd, ~odd]

    def around(self):
        p, s = self.phi, slice(1, -1)
        c = self.c
        return (c[0] * p[:-2, s, s] + c[1] * p[2:, s, s] + c[2] * p[s, :-2, s]
                + c[3] * p[s, 2:, s] + c[4] * p[s, s, :-2] + c[5] * p[s, s, 2:])

    def core(self, t):
        return t[1:-1, 1:-1, 1:-1]

    def mirror(self):
        p, s = self.phi, slice(1, -1)
        p[0, s, s], p[-1, s, s] = p[1, s, s], p[-2, s, s]
        p[s, 0, s], p[s, -1, s] = p[s, 1, s], p[s, -2, s]
        p[s, s, 0], p[s, s, -1] = p[s, s, 1], p[s, s, -2]

    def relax(self, sweeps):
        core, rhs = self.core(self.phi), self.core(self.rhs)
        for _ in range(sweeps):
            for m in self.mask:
                core.copy_(torch.where(m, (rhs - self.around()) / self.ap, core))
        self.mirror()


def _prolong(c, f):
    n = f.n
    i = torch.arange(n, device=DEV)
    even = i % 2 == 0
    first = torch.where(even, i // 2 - 1, i // 2) + 1
    w = torch.where(even, 0.25, 0.75).to(torch.float64)
    x = c.phi
    for axis in range(3):
        shape = [-1 if d == axis else 1 for d in range(3)]
        x = w.view(shape) * x.index_select(axis, first) + \
            (1.0 - w).view(shape) * x.index_select(axis, first + 1)
    f.core(f.phi).add_(x)
    f.mirror()


def _vcycle(lv):
    for l, lev in enumerate(lv):
        if l:
            up = lv[l - 1]
            r = up.core(up.rhs) - (up.around() + up.ap * up.core(up.phi))
            n = lev.n
            lev.core(lev.rhs).copy_(r.view(n, 2, n, 2, n, 2).sum(dim=(1, 3, 5)) * 0.125)
            lev.phi.zero_()
        lev.relax(6 if l < len(lv) - 1 else 300)
    for l in range(len(lv) - 2, -1, -1):
        _prolong(lv[l + 1], lv[l])
        lv[l].relax(6)


def _hierarchy(n, levels, h):
    return [_Level(n >> l, h * 2.0 ** l) for l in range(levels)]


def _solve(lv, rhs):
    lv[0].core(lv[0].rhs).copy_(rhs)
    lv[0].phi.zero_()
    for _ in range(4):
        _vcycle(lv)
    return lv[0].phi


def _exact_fields(n, seed, re, lid):
    """The fields a prepared solver holds: filled from rest, then from the flow."""
    f = {k: torch.zeros((n + 2 * NPL,) * 3, dtype=torch.float64, device=DEV)
         for k in ("u", "v", "w", "p", "vis", "su", "ustar", "vstar", "wstar")}
    f["vis"].fill_(1.0 / re)
    for flow in (None, _flow(n, seed, lid)):
        for q, name in enumerate("uvw"):
            if flow is not None:
                _core(f[name]).copy_(flow[q])
            _fill(f[name], name, n, lid)
    _core(f["p"]).copy_(flow[3])
    _fill(f["p"], "p", n)
    return f


def _exact_step(n, levels, seed, variable_dt):
    re, lid = _physics(seed)
    h, rrey = 1.0 / n, 1.0 / re
    f = _exact_fields(n, seed, re, lid)
    dims = [n, n, n]
    rate, dt_cfl = 0.0, 1.0e10
    for comp in range(3):
        q = f["uvw"[comp]]
        a, b = _at(q, dims, (0, 0, 0)), _at(q, dims, _shift((0, 0, 0), comp, -1))
        rate = rate + (0.5 * (a + b)).abs() / h
        top = float(a.abs().max())
        if top > 0.0:
            dt_cfl = min(dt_cfl, h / top)
    rate = rate + 2.0 * _core(f["vis"]) * (3.0 / (h * h)) + 1.0e-30
    dt = 3.0e-4
    if variable_dt:
        dt = min(1.1 * dt, 0.8 * min(float((1.0 / rate).min()), dt_cfl))
    for name in "uvw":
        f[name + "oo"] = f[name].clone()
    _eddy_viscosity(f, n, h, rrey)
    for alpha in (0.5, 1.0):
        for comp, name in enumerate("uvw"):
            _fill(f[name], name, n, lid)
            _advance(f, n, h, dt, alpha, comp)
        for comp, name in enumerate("uvw"):
            _fill(f[name], name, n, lid)
            _diffuse(f, n, h, dt, alpha, comp)
        if alpha == 0.5:
            _correct(f, n, h, dt, alpha)
    _correct(f, n, h, dt, 1.0)
    lv = _hierarchy(n, levels, h)
    ring = tuple(slice(NPL - 1, NPL + n + 1) for _ in range(3))
    for it in range(1, 31):
        if _divergence(f, n, h, dt) < 1.0e-6 and it > 1:
            break
        f["p"][ring] += _solve(lv, _core(f["su"]))
        _fill(f["p"], "p", n)
        _correct(f, n, h, dt, 1.0)
    for name in "uvw":
        _fill(f[name], name, n, lid)
    return f, dt


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out, dts = [], []
        for q, n in enumerate(int(x) for x in case["sizes"].split(",")):
            f, dt = _exact_step(n, 3, seed * 64 + q, True)
            out.append([f[k] for k in ("u", "v", "w", "p", "vis")])
            dts.append(dt)
        return {"cases": out, "dt": np.array(dts), "iters": None}
    n, levels = case["n"], case["levels"]
    h = 1.0 / n
    if kind == "step":
        f, dt = _exact_step(n, levels, seed, case["variable_dt"])
        return {**{k: f[k] for k in ("u", "v", "w", "p", "vis")}, "dt": dt, "ctime": dt,
                "iters": None}
    if kind == "stage":
        re, lid = _physics(seed)
        f = _exact_fields(n, seed, re, lid)
        for name in "uvw":
            f[name + "oo"] = f[name].clone()
        _eddy_viscosity(f, n, h, 1.0 / re)
        for op in (_advance, _diffuse):
            for comp, name in enumerate("uvw"):
                _fill(f[name], name, n, lid)
                op(f, n, h, 3.0e-4, 0.5, comp)
        _correct(f, n, h, 3.0e-4, 0.5)
        _divergence(f, n, h, 3.0e-4)
        return {k: f[k] for k in ("ustar", "vstar", "wstar", "u", "v", "w", "vis", "su")}
    lv = _hierarchy(n, levels, h)
    if kind == "vcycle":
        lv[0].core(lv[0].rhs).copy_(_rhs(n, seed))
        _vcycle(lv)
        return lv[0].phi
    pp = torch.zeros((n + 2 * NPL,) * 3, dtype=torch.float64, device=DEV)
    pp[NPL - 1:NPL + n + 1, NPL - 1:NPL + n + 1, NPL - 1:NPL + n + 1] = \
        _solve(lv, _rhs(n, seed))
    return pp
