"""The calls whose speed this repository is judged by, over the ranges that its users run.

A case names one public call (`op`), its precision and its grid:
  levelset    Context.levelset_rk3: level-set TVD-RK3 and 3 x 25 reinitialisation sweeps
  velocity    Context.velocity_advection, apply_gravity, sourcing (viscous), velocity_boundary
  projection  Context.projection_host: host arrays in, pressure and velocity out
  frame       Context.advance_frame: curvature, CFL step, one whole order-3 time step
  batch       Batch.run_graph: many instances of uneven sizes in one graph launch
  backward    the vector-Jacobian products: of one level-set advection (`what` = "levelset"), or of one
              projection with its level-set gradient (`what` = "projection")
Grids span [0,1] in x with square cells, except the Rayleigh-Taylor cases (dy = 2 dx).
"""
import importlib
import math
import random

import numpy as np
import torch

gb = importlib.import_module("2d_engine_gb300")

F64, MIX = "fp64", "mixed"
BATCH_SIZES = (64, 96, 128, 200, 256, 384, 512)


def listed():
    return [
        # a tool's or a test's small grid, where latency and launches count; the mixed solver's lower end
        {"name": "projection_mixed_64", "op": "projection", "precision": MIX, "ni": 64, "nj": 64, "tol": 1e-8},
        # the benchmark's standalone projection: eight circles, density 1:1000, 1024^2, relative residual 1e-8
        {"name": "projection_mixed_1024", "op": "projection", "precision": MIX, "ni": 1024, "nj": 1024, "tol": 1e-8},
        # the default precision on an odd, oblong grid, to the tighter tolerance of the parity runs
        {"name": "projection_fp64_511x385", "op": "projection", "precision": F64, "ni": 511, "nj": 385, "tol": 1e-10},
        # the default precision's level-set step: a small ragged grid and an ordinary one
        {"name": "levelset_fp64_97x65", "op": "levelset", "precision": F64, "ni": 97, "nj": 65},
        {"name": "levelset_fp64_512", "op": "levelset", "precision": F64, "ni": 512, "nj": 512},
        # the mixed level-set step at the benchmark's size
        {"name": "levelset_mixed_1024", "op": "levelset", "precision": MIX, "ni": 1024, "nj": 1024},
        # the velocity stage around a projection, default precision, ragged
        {"name": "velocity_fp64_1000x750", "op": "velocity", "precision": F64, "ni": 1000, "nj": 750},
        # one frame of the plain rising bubble (128^2, relative residual 1e-10)
        {"name": "frame_fp64_128", "op": "frame", "precision": F64, "ni": 128, "nj": 128, "tol": 1e-10, "flow": "bubble"},
        # one frame of the large Rayleigh-Taylor run: mixed precision, the largest grid in use
        {"name": "frame_mixed_rt_2048", "op": "frame", "precision": MIX, "ni": 2048, "nj": 2048, "tol": 1e-8, "flow": "rt"},
        # independent rising bubbles of uneven sizes advanced together
        {"name": "batch_mixed_16", "op": "batch", "precision": MIX, "instances": 16, "ni": 512, "tol": 1e-8},
        # the two halves of a differentiated window's backward pass
        {"name": "backward_levelset_256", "op": "backward", "what": "levelset", "precision": F64, "ni": 256, "nj": 256},
        {"name": "backward_projection_256", "op": "backward", "what": "projection", "precision": F64, "ni": 256, "nj": 256,
         "tol": 1e-10},
    ]


def draw(rng: random.Random):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["levelset", "levelset", "velocity", "projection", "projection", "frame", "batch", "backward"])
    prec = rng.choice([F64, MIX])
    if op == "batch":
        return {"op": op, "precision": MIX, "instances": rng.randint(4, 16), "ni": size(96, 400), "tol": 1e-8}
    top = {"levelset": {F64: 500, MIX: 1600}, "velocity": {F64: 1600, MIX: 1600}, "projection": {F64: 900, MIX: 1500},
           "frame": {F64: 300, MIX: 1200}, "backward": {F64: 400, MIX: 400}}[op][prec]
    ni = size(40, top)
    nj = max(32, int(ni * rng.uniform(0.5, 1.0)))
    c = {"op": op, "precision": prec, "ni": ni, "nj": nj}
    if op in ("projection", "frame", "backward"):
        c["tol"] = 1e-10 if prec == F64 else 1e-8
    if op == "frame":
        c["flow"] = rng.choice(["bubble", "rt"])
    if op == "backward":
        c["precision"], c["tol"], c["what"] = F64, 1e-10, rng.choice(["levelset", "projection"])
    return c


# ---- inputs -----------------------------------------------------------------------------------------------------


def _extent(case):
    """(x_max, y_max): square cells, and dy = 2 dx for the Rayleigh-Taylor flow."""
    y = (case["nj"] - 1) / (case["ni"] - 1)
    return 1.0, 2.0 * y if case.get("flow") == "rt" else y


def _nodes(ni, nj, x_max, y_max):
    x = (np.arange(ni + 4) - 2) * (x_max / (ni - 1))
    y = (np.arange(nj + 4) - 2) * (y_max / (nj - 1))
    return x[None, :], y[:, None]


def _circles(rng, ni, nj, x_max, y_max, n=8):
    """Signed distance to the union of n circles, phi < 0 (the light phase) inside."""
    x, y = _nodes(ni, nj, x_max, y_max)
    phi = np.full((nj + 4, ni + 4), np.inf)
    for _ in range(n):
        cx, cy, r = rng.uniform(0.1, 0.9) * x_max, rng.uniform(0.1, 0.9) * y_max, rng.uniform(0.03, 0.12)
        phi = np.minimum(phi, np.sqrt((x - cx) ** 2 + (y - cy) ** 2) - r)
    return phi


def _faces(rng, nj, ni, walls):
    """Random face values U[-1,1] with zero wall faces, smoothed by 4 Jacobi passes (ghost 2)."""
    a = rng.uniform(-1.0, 1.0, (nj, ni))
    for k in range(5):
        if k:
            b = a.copy()
            b[1:-1, 1:-1] = (a[1:-1, 1:-1] + a[:-2, 1:-1] + a[2:, 1:-1] + a[1:-1, :-2] + a[1:-1, 2:]) / 5.0
            a = b
        if walls == "x":
            a[:, 0] = a[:, -1] = 0.0
        else:
            a[0] = a[-1] = 0.0
    return np.pad(a, 2)


def _ghost_copies(a, g=3):
    """The interior of a ghost-2 array with g ghost layers that copy its second interior line, corners zero."""
    f = a[2:-2, 2:-2]
    nj, ni = f.shape
    out = np.zeros((nj + 2 * g, ni + 2 * g))
    out[g:g + nj, g:g + ni] = f
    out[g:g + nj, :g], out[g:g + nj, g + ni:] = f[:, 1:2], f[:, ni - 2:ni - 1]
    out[:g, g:g + ni], out[g + nj:, g:g + ni] = f[1:2], f[nj - 2:nj - 1]
    return out


def _fields(case, seed):
    """The host arrays of a case (phi, u, v, ua, va, p), from the seed alone."""
    rng = np.random.default_rng(seed)
    ni, nj = case["ni"], case["nj"]
    xm, ym = _extent(case)
    flow = case.get("flow")
    x, y = _nodes(ni, nj, xm, ym)
    if flow == "bubble":
        cx, cy, r = rng.uniform(0.45, 0.55), rng.uniform(0.3, 0.45) * ym, rng.uniform(0.1, 0.2) * min(1.0, ym)
        phi, amp = np.sqrt((x - cx) ** 2 + (y - cy) ** 2) - r, 0.1
    elif flow == "rt":
        phi, amp = y - 0.5 * ym - rng.uniform(0.03, 0.06) * np.cos(2 * np.pi * (x - rng.uniform(0.0, 0.1))), 0.05
    else:
        phi, amp = _circles(rng, ni, nj, xm, ym), 1.0
    u, v = amp * _faces(rng, nj, ni + 1, "x"), amp * _faces(rng, nj + 1, ni, "y")
    return dict(phi=np.ascontiguousarray(phi), u=u, v=v, ua=_ghost_copies(u), va=_ghost_copies(v), p=np.zeros((nj + 2, ni + 2)))


def _physics(case):
    if case.get("flow") == "rt":
        return dict(water_density=3.0, air_density=1.0, surface_tension=0.0)
    return dict(water_density=1000.0, air_density=1.0, surface_tension=0.0728)


def _viscosities(case):
    if case.get("flow") == "rt":
        return dict(water_viscosity=1e-3, air_viscosity=1e-3)
    return dict(water_viscosity=1.0, air_viscosity=0.01)


def _context(case, f):
    c = gb.Context(case["ni"], case["nj"], 0.0, 0.0, *_extent(case),
                   advection_precision=gb.PRECISION_MIXED if case["precision"] == MIX else gb.PRECISION_FP64, **_physics(case))
    c.set_flow_params(viscosity=True, cfl_number=0.5, **_viscosities(case))
    for name, fid in (("phi", gb.FIELD_PHI), ("u", gb.FIELD_U), ("v", gb.FIELD_V), ("ua", gb.FIELD_UA), ("va", gb.FIELD_VA),
                      ("p", gb.FIELD_P)):
        c.set(fid, f[name])
    return c


def _opts(case):
    return gb.solve_opts(precision=gb.PRECISION_MIXED if case["precision"] == MIX else gb.PRECISION_FP64, tolerance=case["tol"],
                         max_iterations=2000)


class _Device:
    """A field on the GPU as it lies in a context, without a copy; keeps the context (and a batch that owns it) open."""

    def __init__(self, ctx, field):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": ctx.shape(field), "typestr": "<f8", "data": (ctx.device_ptr(field), False),
                                         "version": 3, "strides": None, "stream": None}


def _view(ctx, field):
    return torch.as_tensor(_Device(ctx, field), device="cuda")


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _dt(case):
    """Half a cell per unit velocity; under the explicit viscous limit where the viscosity acts."""
    dx = 1.0 / (case["ni"] - 1)
    return min(0.5 * dx, 0.2 * dx * dx / 0.01) if case["op"] == "velocity" else 0.5 * dx


def prepare(case, seed):
    if case["op"] == "batch":
        return _prepare_batch(case, seed)
    f = _fields(case, seed)
    s = {"case": case, "dt": _dt(case), "ctx": _context(case, f)}
    c = s["ctx"]
    if "tol" in case:
        s["opts"] = _opts(case)
    if case["op"] == "projection":
        s["in"] = {k: _pinned(f[k].shape) for k in ("phi", "u", "v", "p")}
        for k, a in s["in"].items():
            a[...] = f[k]
        s["out"] = {k + "_out": _pinned(f[k].shape) for k in ("p", "u", "v")}
    elif case["op"] == "frame":
        s["prev"] = 0.0
        for _ in range(2):  # a run under way: its pressure is the next projection's start
            s["prev"], _ = c.advance_frame(cfl=1.0, prev_dt=s["prev"], opts=s["opts"], allow_max_iters=True)
    elif case["op"] == "backward":
        rng = np.random.default_rng(seed + 7919)
        if case["what"] == "levelset":
            s["lam"] = rng.standard_normal(f["phi"].shape)
        else:
            c.projection(s["dt"], s["opts"], allow_max_iters=True)
            s["lam"] = _faces(rng, case["nj"], case["ni"] + 1, "x"), _faces(rng, case["nj"] + 1, case["ni"], "y")
    if case["op"] in ("levelset", "velocity", "frame"):
        c.checkpoint_save()
    c.synchronize()
    return s


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    sizes = [n for n in BATCH_SIZES if n <= max(96, case["ni"])]
    grids, phis, params, flows = [], [], [], []
    for k in range(case["instances"]):
        n = sizes[k % len(sizes)]
        x, y = _nodes(n, n, 1.0, 1.0)
        grids.append((n, n, 1.0, 1.0))
        phis.append(np.sqrt((x - 0.5) ** 2 + (y - rng.uniform(0.2, 0.4)) ** 2) - rng.uniform(0.1, 0.2))
        params.append(dict(water_density=float(np.exp(rng.uniform(np.log(10), np.log(1000)))), air_density=1.0))
        flows.append(dict(water_viscosity=0.01 * float(np.exp(rng.uniform(0.0, np.log(100)))), air_viscosity=0.01, viscosity=True))
    b = gb.Batch(grids, params=params, flows=flows)
    opts = gb.solve_opts(precision=gb.PRECISION_MIXED, tolerance=case["tol"], max_iterations=2000)
    views = [b.context(k) for k in range(b.n)]
    for c, p in zip(views, phis):
        c.owner = b
        c.set(gb.FIELD_PHI, np.ascontiguousarray(p))
    dts, _ = b.run_graph(1, opts=opts, allow_max_iters=True)  # the run is under way, its graph captured
    for c in views:
        c.checkpoint_save()
        c.synchronize()
    return {"case": case, "batch": b, "views": views, "opts": opts, "prev": dts}


# ---- one pass ---------------------------------------------------------------------------------------------------


def run(state):
    s, case = state, state["case"]
    op = case["op"]
    if op == "batch":
        for c in s["views"]:
            c.checkpoint_restore()
        dts, _ = s["batch"].run_graph(1, dts=s["prev"].copy(), opts=s["opts"], allow_max_iters=True)
        return {"dt": dts, "fields": [[_view(c, f) for f in (gb.FIELD_PHI, gb.FIELD_U, gb.FIELD_V)] for c in s["views"]]}
    c = s["ctx"]
    if op == "projection":
        c.projection_host(s["dt"], s["opts"], **s["in"], **s["out"], allow_max_iters=True)
        return s["out"]
    if op == "backward":
        if case["what"] == "levelset":
            return dict(zip(("phi", "ua", "va"), c.weno5_adjoint(s["dt"], s["lam"])))
        u, v, _ = c.projection_adjoint(s["dt"], *s["lam"], opts=s["opts"], allow_max_iters=True)
        return {"u": u, "v": v, "phi": c.projection_phi_gradient(s["dt"])}
    c.checkpoint_restore()
    if op == "levelset":
        c.levelset_rk3(s["dt"])
        return {"phi": _view(c, gb.FIELD_PHI)}
    if op == "velocity":
        c.velocity_advection(s["dt"])
        c.apply_gravity(s["dt"])
        c.sourcing(s["dt"])
        c.velocity_boundary()
        return {k: _view(c, f) for k, f in (("u", gb.FIELD_U), ("v", gb.FIELD_V), ("ua", gb.FIELD_UA), ("va", gb.FIELD_VA))}
    dt, _ = c.advance_frame(cfl=1.0, prev_dt=s["prev"], opts=s["opts"], allow_max_iters=True)
    return {"dt": dt, **{k: _view(c, f) for k, f in (("phi", gb.FIELD_PHI), ("u", gb.FIELD_U), ("v", gb.FIELD_V), ("p", gb.FIELD_P))}}


# Floating-point operations per node: one WENO5 advection or reinitialisation sweep (four one-sided derivatives of 80),
# the ENO3 advection of both components, the viscous stage, an assembly with its velocity update, and one iteration of
# multigrid-preconditioned CG (two red-black sweeps a side; 4/3 for the coarser levels).
_SWEEP, _ENO, _VISC, _ASSEMBLE, _CG = 336.0, 230.0, 160.0, 120.0, 4.0 / 3.0 * 60.0 + 25.0


def work(case):
    """Every input read and every output written once; iteration counts of a typical solve (cold 16, under way 8)."""
    if case["op"] == "batch":
        sizes = [n for n in BATCH_SIZES if n <= max(96, case["ni"])]
        nodes = sum(float(sizes[k % len(sizes)]) ** 2 for k in range(case["instances"]))
    else:
        nodes = float(case["ni"] * case["nj"])
    levelset = 78 * _SWEEP
    per = {"levelset": (4, levelset), "velocity": (7, _ENO + _VISC), "projection": (7, _ASSEMBLE + 16 * _CG),
           "frame": (10, levelset + 3 * (_ENO + _VISC + _ASSEMBLE + 8 * _CG)),
           "batch": (10, levelset + 3 * (_ENO + _VISC + _ASSEMBLE + 8 * _CG)),
           "backward": (7, 900.0 if case.get("what") == "levelset" else _ASSEMBLE + 16 * _CG)}[case["op"]]
    return {"bytes": 8.0 * per[0] * nodes, "flops": per[1] * nodes}


# ---- the same results in 64 bits, by torch ----------------------------------------------------------------------


def _weno_side(a1, a2, a3, a4, a5, eps=1e-6):
    c13, q = 13.0 / 12.0, 0.25
    s1 = c13 * (a1 - 2 * a2 + a3) ** 2 + q * (a1 - 4 * a2 + 3 * a3) ** 2
    s2 = c13 * (a2 - 2 * a3 + a4) ** 2 + q * (a2 - a4) ** 2
    s3 = c13 * (a3 - 2 * a4 + a5) ** 2 + q * (3 * a3 - 4 * a4 + a5) ** 2
    w1, w2, w3 = 0.1 / (eps + s1) ** 2, 0.6 / (eps + s2) ** 2, 0.3 / (eps + s3) ** 2
    s = w1 + w2 + w3
    return (w1 * (a1 / 3 - 7 * a2 / 6 + 11 * a3 / 6) + w2 * (-a2 / 6 + 5 * a3 / 6 + a4 / 3) + w3 * (a3 / 3 + 5 * a4 / 6 - a5 / 6)) / s


def _lines(f, dim, o):
    """The six first differences of every node along dim; values off the grid are the second interior line."""
    n = f.shape[dim]
    at = torch.arange(-3, n + 3, device=f.device)
    at = torch.where(at < 0, torch.ones_like(at), torch.where(at >= n, torch.full_like(at, n - 2), at))
    g = f.index_select(dim, at)
    d = o * (g.narrow(dim, 1, n + 5) - g.narrow(dim, 0, n + 5))
    return [d.narrow(dim, k, n) for k in range(6)]


def _sides(f, dim, o):
    d = _lines(f, dim, o)
    return _weno_side(*d[:5]), _weno_side(*d[5:0:-1])


def _advect(phi, ua, va, dt, odx, ody):
    """One level-set advection of a ghost-2 phi, with the extrapolation of its ghosts (corners keep theirs)."""
    f = phi[2:-2, 2:-2]
    nj, ni = f.shape
    u = (ua[3:-3, 4:4 + ni] + ua[3:-3, 3:3 + ni]) * 0.5
    v = (va[4:4 + nj, 3:-3] + va[3:3 + nj, 3:-3]) * 0.5
    (mx, px), (my, py) = _sides(f, 1, odx), _sides(f, 0, ody)
    g = f - dt * (u * torch.where(u > 0, mx, px) + v * torch.where(v > 0, my, py))
    left, low = phi[2:-2, 1:2], phi[1:2, 2:-2]  # the outer layer reads the inner one's old value
    r1, t1 = 2 * g[:, -1:] - g[:, -2:-1], 2 * g[-1:] - g[-2:-1]
    rows = torch.cat([2 * left - g[:, :1], 2 * g[:, :1] - g[:, 1:2], g, r1, 2 * r1 - g[:, -1:]], 1)
    below = torch.cat([phi[:2, :2], torch.cat([2 * low - g[:1], 2 * g[:1] - g[1:2]], 0), phi[:2, -2:]], 1)
    above = torch.cat([phi[-2:, :2], torch.cat([t1, 2 * t1 - g[-1:]], 0), phi[-2:, -2:]], 1)
    return torch.cat([below, rows, above], 0)


def _reinit(f, dx, odx, ody, sweeps=25, scaling=5):
    s = f / torch.sqrt(f * f + dx * dx)
    for _ in range(sweeps):
        g2 = 0.0
        keep = torch.zeros_like(f, dtype=torch.bool)
        for dim, o in ((1, odx), (0, ody)):
            m, p = _sides(f, dim, o)
            sm, sp = s * m, s * p
            shock = (sp < 0) & (sm > 0)
            sss = s * (p.abs() - m.abs()) / (p - m)
            g = torch.where((sp >= 0) & (sm >= 0), m, torch.where((sp <= 0) & (sm <= 0), p, torch.zeros_like(p)))
            g = torch.where(shock, torch.where(sss > 0, m, p), g)
            if dim == 1:
                keep = shock & (sss == 0)
            g2 = g2 + g * g
        f = torch.where(keep, f, f - dx / scaling * s * (torch.sqrt(g2) - 1))
    return f


def _levelset(phi, ua, va, dt, dx, odx, ody):
    def mix(a, x, c0):
        y = x.clone()
        y[2:-2, 2:-2] = c0 * a[2:-2, 2:-2] + (1 - c0) * x[2:-2, 2:-2]
        return y

    b = _advect(_advect(phi, ua, va, dt, odx, ody), ua, va, dt, odx, ody)
    b = mix(phi, _advect(mix(phi, b, 0.75), ua, va, dt, odx, ody), 1 / 3.0)
    f0 = b[2:-2, 2:-2]
    f = _reinit(_reinit(f0, dx, odx, ody), dx, odx, ody)
    f = _reinit(0.75 * f0 + 0.25 * f, dx, odx, ody)
    b[2:-2, 2:-2] = f0 / 3.0 + f * (2 / 3.0)
    return b


def _curvature(phi, dx, dy):
    c, l, r, b, t = phi[2:-2, 2:-2], phi[2:-2, 1:-3], phi[2:-2, 3:-1], phi[1:-3, 2:-2], phi[3:-1, 2:-2]
    px, py = (r - l) / (2 * dx), (t - b) / (2 * dy)
    pxx, pyy = (r - 2 * c + l) / dx ** 2, (t - 2 * c + b) / dy ** 2
    pxy = (phi[3:-1, 3:-1] - phi[1:-3, 3:-1] - phi[3:-1, 1:-3] + phi[1:-3, 1:-3]) / (4 * dx * dy)
    k = -(px * px * pyy - 2 * px * py * pxy + py * py * pxx) / (px * px + py * py) ** 1.5
    top = 1.0 / min(dx, dy)
    return k.clamp(-top, top)


def _project(phi, u, v, dt, dx, dy, water, air, sigma):
    """PROJECTION_2D::Solve from a zero pressure: (p, u, v), the system solved by Jacobi-preconditioned CG until it stands."""
    f = phi[2:-2, 2:-2]
    nj, ni = f.shape
    left, low = phi[2:-2, 1:2].clone(), phi[1:2, 2:-2].clone()
    phi = phi.clone()
    phi[2:-2, 0:1], phi[2:-2, 1:2] = 2 * left - f[:, :1], 2 * f[:, :1] - f[:, 1:2]
    phi[2:-2, -2:-1] = 2 * f[:, -1:] - f[:, -2:-1]
    phi[0:1, 2:-2], phi[1:2, 2:-2] = 2 * low - f[:1], 2 * f[:1] - f[1:2]
    phi[-2:-1, 2:-2] = 2 * f[-1:] - f[-2:-1]
    jc = torch.nn.functional.pad(sigma * _curvature(phi, dx, dy), (1, 1, 1, 1))
    rho = torch.where(f <= 0, torch.full_like(f, 1 / air), torch.full_like(f, 1 / water))
    w = torch.nn.functional.pad(rho, (1, 1, 1, 1))
    w[:, 0], w[:, -1], w[0], w[-1] = w[:, 2], w[:, -3], w[2], w[-3]
    q = phi[1:-1, 1:-1]

    def faces(dim, h):
        n = q.shape[dim]
        cut = (lambda a: a[1:-1]) if dim == 1 else (lambda a: a[:, 1:-1])
        one, two = (lambda a: cut(a.narrow(dim, 0, n - 1))), (lambda a: cut(a.narrow(dim, 1, n - 1)))
        vc, vn, pc, pn = two(w), one(w), two(q), one(q)
        ac, an = pc.abs(), pn.abs()
        beta = vc * vn * (an + ac) / (vc * an + vn * ac)
        crosses = (pc <= 0) != (pn <= 0)
        jump = torch.where(crosses, (two(jc) * an + one(jc) * ac) / (ac + an), torch.zeros_like(ac))
        flux = torch.where(pc <= 0, jump, -jump) * beta / h ** 2  # the cell on the + side; the other cell's is its negative
        return beta, flux, jump, pc, pn

    bx, fx, jx, pcx, pnx = faces(1, dx)
    by, fy, jy, pcy, pny = faces(0, dy)
    iu, iv = u[2:-2, 2:-2], v[2:-2, 2:-2]
    div = ((iu[:, 1:] - iu[:, :-1]) / dx + (iv[1:] - iv[:-1]) / dy) / dt
    rhs = -div - (fx[:, :-1] - fx[:, 1:]) - (fy[:-1] - fy[1:])
    ix, iy = bx.clone(), by.clone()
    ix[:, 0] = ix[:, -1] = 0
    iy[0] = iy[-1] = 0
    diag = ix[:, 1:] + ix[:, :-1] + iy[1:] + iy[:-1]
    diag[0, 0] += bx[0, 0] + by[0, 0]
    diag = diag / dx ** 2
    cx, cy = ix[:, 1:-1] / dx ** 2, iy[1:-1] / dy ** 2

    def apply(x):
        y = diag * x
        y[:, 1:] -= cx * x[:, :-1]
        y[:, :-1] -= cx * x[:, 1:]
        y[1:] -= cy * x[:-1]
        y[:-1] -= cy * x[1:]
        return y

    x, bb = torch.zeros_like(rhs), float((rhs * rhs).sum())
    for _ in range(2):
        r = rhs - apply(x)
        z = r / diag
        d, rz = z.clone(), (r * z).sum()
        for it in range(40000):
            ad = apply(d)
            a = rz / (d * ad).sum()
            x += a * d
            r -= a * ad
            z = r / diag
            new = (r * z).sum()
            d.mul_(new / rz).add_(z)
            rz = new
            if it % 200 == 199 and not float((r * r).sum()) > 1e-28 * bb:
                break
    p = torch.nn.functional.pad(x, (1, 1, 1, 1))

    def update(old, dim, h, jump, pc, pn):
        n = p.shape[dim]
        cut = (lambda a: a[1:-1]) if dim == 1 else (lambda a: a[:, 1:-1])
        dp = cut(p.narrow(dim, 1, n - 1)) - cut(p.narrow(dim, 0, n - 1))
        e, m = 1.5 * h, 0.5 * (pc + pn)
        hs = 0.5 + m / e * 0.5 + 0.5 / 3.141592 * torch.sin(3.141592 * m / e)
        hs = torch.where(m < -e, torch.zeros_like(m), torch.where(m > e, torch.ones_like(m), hs))
        same = pc * pn >= 0
        o = torch.where(same, torch.where(pc <= 0, torch.full_like(m, 1.0 / air), torch.full_like(m, 1.0 / water)),
                        1.0 / (air + (water - air) * hs))
        g = torch.where(same, dp, torch.where(pc < 0, dp + jump, dp - jump))
        out = old.clone()
        inner = out[2:-2, 2:-2].narrow(dim, 0, n - 2)  # faces on the + side wall are left alone
        inner -= (dt * g * o / h).narrow(dim, 0, n - 2)
        return out

    return p, update(u, 1, dx, jx, pcx, pnx), update(v, 0, dy, jy, pcy, pny)


def exact(case, seed):
    if case["op"] not in ("levelset", "projection", "backward") or case.get("what") == "projection":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = {k: torch.from_numpy(a).to(dev) for k, a in _fields(case, seed).items()}
    xm, ym = _extent(case)
    dx, dy, dt = xm / (case["ni"] - 1), ym / (case["nj"] - 1), _dt(case)
    if case["op"] == "projection":
        ph = _physics(case)
        out = _project(f["phi"], f["u"], f["v"], dt, dx, dy, ph["water_density"], ph["air_density"], ph["surface_tension"])
        return dict(zip(("p_out", "u_out", "v_out"), out))
    if case["op"] == "levelset":
        return {"phi": _levelset(f["phi"], f["ua"], f["va"], dt, dx, 1 / dx, 1 / dy)}
    lam = torch.from_numpy(np.random.default_rng(seed + 7919).standard_normal(f["phi"].shape)).to(dev)
    ins = [f[k].requires_grad_(True) for k in ("phi", "ua", "va")]
    return dict(zip(("phi", "ua", "va"), torch.autograd.grad(_advect(*ins, dt, 1 / dx, 1 / dy), ins, lam)))
