"""The work that users of forestclaw_b200 have it do, as cases that can be timed.

listed()             the cases, draw(rng) one more of the same ranges
prepare(case, seed)  what a program holds before the call: a solver (or server)
                     on the GPU and its initial state
run(state)           one pass through the public entry points, and its outputs
work(case)           the bytes and operations one pass cannot do without
exact(case, seed)    what a pass on meshes of one level returns, in plain torch

Kinds of cases:
  uniform  a mesh of one level, `steps` macro steps from the state the last
           pass left, then the frame (get_q into a pinned host buffer)
  level    the same mesh driven level by level, as a host code with a schedule
           of its own does: update_single_step, ghost_update
  amr      subcycled macro steps on a refined mesh between two regrids
  run      a whole solve: initialize, run with its regrids, the final frame
  serve    an ensemble of solves through the server, from submit to results
"""
from __future__ import annotations

import math

import numpy as np
import torch

import forestclaw_b200 as fcb
from forestclaw_b200 import serve as fcb_serve
from forestclaw_b200 import workloads

MEQN = {"advection": 1, "swe": 3, "euler": 4, "geoclaw": 3, "filament": 1}
# Operations (add, multiply, divide, square root, compare/select) of one cell
# update, ghost-region work of the reference's patch step included, for the
# patch sizes the repository's operation count was taken at (bench.py); the
# filament's capacity form adds its divisions to the advection count.
OPS = {"advection": 193.25, "swe": 1090.2, "euler": 2005.2, "geoclaw": 1326.4, "filament": 220.0}
KROOT = 1 << 28
# rho, u, v, p of the quadrant problem the repository's tests use
QUADRANTS = ((1.5, 0.0, 0.0, 1.5), (0.532258064516129, 1.206045378311055, 0.0, 0.3),
             (0.137992831541219, 1.206045378311055, 1.206045378311055, 0.029032258064516),
             (0.532258064516129, 0.0, 1.206045378311055, 0.3))


def _case(name, kind, equation, mx, minlevel, maxlevel, steps, precision="fp64", version=4, limiter=4, walls=False,
          cfl_each_step=False, requests=0):
    c = dict(kind=kind, equation=equation, mx=mx, minlevel=minlevel, maxlevel=maxlevel, steps=steps,
             precision=precision, version=version, limiter=limiter, walls=walls, cfl_each_step=cfl_each_step,
             requests=requests)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the plain-method advection problem: 256 patches, 200 steps, the CFL
        # number read after every one (latency and launches)
        _case("swirl_256_patches", "uniform", "advection", 16, 4, 4, 200, cfl_each_step=True),
        # the headline mesh: 65,536 patches of 16 x 16, a frame every 50 steps
        _case("swirl_65536_patches", "uniform", "advection", 16, 8, 8, 50),
        # the same in the mixed FP32/FP64 form
        _case("swirl_65536_mixed", "uniform", "advection", 16, 8, 8, 50, precision="mixed"),
        # a basin with solid walls: Roe shallow water, 1,024 patches of 32 x 32
        _case("swe_basin", "uniform", "swe", 32, 5, 5, 20, walls=True),
        # clawpack 5 update driven by a host code's own schedule, 256 patches
        _case("swe_v5_level_calls", "level", "swe", 32, 4, 4, 20, version=5, limiter=3, cfl_each_step=True),
        # four quadrant states, mixed precision, 4,096 patches of 16 x 16
        _case("euler_mixed", "uniform", "euler", 16, 6, 6, 15, precision="mixed"),
        # dam break on a refined mesh (levels 3-6): macro steps between two regrids
        _case("swe_amr_steps", "amr", "swe", 32, 3, 6, 3),
        # the same problem as a user's run: initialize, regrid after every step
        _case("swe_amr_run", "run", "swe", 32, 3, 6, 4),
        # Euler quadrants on a deeper refined mesh of small patches
        _case("euler_amr_steps", "amr", "euler", 16, 2, 6, 2),
        # waves over bathymetry (GeoClaw f-waves, stored aux), levels 4-6
        _case("bathymetry_amr_steps", "amr", "geoclaw", 32, 4, 6, 2),
        # the filament run: mapped brick with capacity, manifold advection
        _case("filament_run", "run", "filament", 32, 3, 5, 4),
        # twelve dam breaks of two patch sizes served together
        _case("serve_12_dam_breaks", "serve", "swe", 0, 2, 5, 0, requests=12),
    ]


def draw(rng):
    """One more case of the listed ones' ranges, no larger than the largest."""
    kind = rng.choices(("uniform", "level", "amr", "run"), (5, 2, 4, 1))[0]
    if kind in ("uniform", "level"):
        eq = rng.choices(("advection", "swe", "euler"), (4, 3, 2))[0]
        precision = rng.choice(("fp64", "fp64", "mixed"))
        version = rng.choice((4, 4, 5))
        sizes = (8, 16, 32) if precision == "mixed" or version == 5 else (8, 16, 32, 64)
        mx = rng.choice(sizes)
        most = 1 << (24 if eq == "advection" else 20)
        cells = math.exp(rng.uniform(math.log(1 << 12), math.log(most)))
        level = max(0, min(8, round(math.log2(math.sqrt(cells) / mx))))
        n = mx << level
        room = 1.5e11 / (n * n * OPS[eq])
        steps = max(3, min(int(math.exp(rng.uniform(math.log(7), math.log(200)))), int(room)))
        # the quadrants' inflow tears away from a wall, and superbee sharpens the
        # systems' waves into noise over thousands of steps
        walls = eq == "swe" and rng.random() < 0.5
        limiter = rng.choice((1, 2, 3, 4, 4) if eq == "advection" else (1, 3, 4, 4))
        return _case(None, kind, eq, mx, level, level, steps, precision, version, limiter, walls,
                     kind == "level" or rng.random() < 0.3)
    eq = rng.choice(("swe", "swe", "euler", "geoclaw", "filament"))
    if kind == "run":
        eq = rng.choice(("swe", "filament"))
    mx = rng.choice((8, 16, 32))
    top = {8: 6, 16: 6, 32: 5}[mx] - (1 if eq in ("filament", "geoclaw") else 0)
    maxlevel = rng.randint(4, top)
    minlevel = rng.randint(2, maxlevel - 1)
    if eq == "geoclaw":
        minlevel = max(minlevel, 3)
    version = 5 if eq == "swe" and rng.random() < 0.3 else 4
    return _case(None, kind, eq, mx, minlevel, maxlevel, rng.randint(1, 3), "fp64", version,
                 rng.choice((3, 4)) if eq != "filament" else 3, False)


# ---------------------------------------------------------------------------
# What a program holds before the call
# ---------------------------------------------------------------------------
def _n(case):
    return case["mx"] << case["maxlevel"]


def _dt(case):
    """A fixed step of CFL 0.3 to 0.9 on the coarsest level of the mesh, with room for
    what the state may become after many passes."""
    n = case["mx"] << case["minlevel"]
    return {"advection": 0.9, "swe": 0.3, "euler": 0.2, "geoclaw": 0.5, "filament": 0.08}[case["equation"]] / n


def _options(case, seed):
    eq, mx, lo, hi = case["equation"], case["mx"], case["minlevel"], case["maxlevel"]
    m = MEQN[eq]
    u = np.random.default_rng(seed).uniform(-1.0, 1.0, size=4) if case["kind"] == "run" else np.zeros(4)
    if eq == "advection":
        o = workloads.uniform_swirl(hi, mx)
    elif eq == "swe":
        o = workloads.amr_shallow_water(seed=0, minlevel=lo, maxlevel=hi, mx=mx)
        o.problem_params = (0.5, 0.5, 0.25 + 0.05 * float(u[0]), 2.0 + 0.1 * float(u[1]), 1.0)
        o.initial_dt = 0.5 / (mx << lo)
        o.tfinal = case["steps"] * 0.45 / (mx << lo)
    elif eq == "euler":
        o = workloads.amr_euler(seed=0, minlevel=lo, maxlevel=hi, mx=mx)
        o.problem_params = tuple(s[k] for k in range(4) for s in QUADRANTS) + (0.5, 0.5)
    elif eq == "geoclaw":
        o = workloads.bathymetry(seed=0, minlevel=lo, maxlevel=hi, mx=mx)
    else:
        o = workloads.filament(minlevel=lo, maxlevel=hi, mx=mx, claw_version=case["version"])
        o.problem_params = (0.0, 0.0, 0.5 + 0.02 * float(u[0]), 1.0 + 0.02 * float(u[1]), 0.25)
        o.tfinal = case["steps"] * 0.1 / (mx << lo)
    o.claw_version = case["version"]
    o.mthlim = (case["limiter"],) * m
    o.precision = fcb.PRECISION_MIXED if case["precision"] == "mixed" else fcb.PRECISION_FP64
    if case["walls"]:
        o.mthbc = (3, 3, 3, 3)
    if case["kind"] != "run":
        o.regrid_interval = 0
        o.use_fixed_dt = 1
    return o


def _pad(q, walls):
    """Ghost cells of the domain (two deep): left and right, then bottom and top."""
    def mirrored(a, dim, comp, low):
        n = a.shape[dim]
        if walls:
            g = a.narrow(dim, 0 if low else n - 2, 2).flip(dim).clone()
            g[comp] = -g[comp]
            return g
        return a.narrow(dim, 0 if low else n - 1, 1).expand(*[2 if d == dim else -1 for d in range(a.dim())])
    q = torch.cat([mirrored(q, 2, 1, True), q, mirrored(q, 2, 1, False)], 2)
    return torch.cat([mirrored(q, 1, 2, True), q, mirrored(q, 1, 2, False)], 1)


def _patches(padded, case):
    """The leaves' arrays in Morton order, ghost cells included, from the padded mesh."""
    mx, p = case["mx"], 1 << case["maxlevel"]
    u = padded.unfold(1, mx + 4, mx).unfold(2, mx + 4, mx)  # (m, py, px, ny, nx)
    k = torch.arange(p * p, device=padded.device)
    x, y = torch.zeros_like(k), torch.zeros_like(k)
    for b in range(case["maxlevel"]):
        x |= ((k >> (2 * b)) & 1) << b
        y |= ((k >> (2 * b + 1)) & 1) << b
    q = u[:, y, x].transpose(0, 1)  # (patches, m, ny, nx)
    return (q.permute(0, 2, 3, 1) if case["version"] == 5 else q).contiguous()


def _initial(case, seed):
    """The initial state of a mesh of one level: the equation's standard problem
    (step, dam break, quadrants) with smooth seeded waves on it."""
    n, dev = _n(case), torch.device("cuda")
    g = np.random.default_rng(seed)
    x = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n
    X, Y = x[None, :], x[:, None]
    wave = torch.zeros(n, n, dtype=torch.float64, device=dev)
    for _ in range(4):
        kx, ky, px, py = (float(v) for v in (*g.integers(1, 6, 2), *g.uniform(0, 2 * math.pi, 2)))
        wave += 0.25 * torch.cos(2 * math.pi * kx * X + px) * torch.cos(2 * math.pi * ky * Y + py)
    if case["equation"] == "advection":
        q = ((X < 0.5).double() + 0.1 * wave)[None]
    elif case["equation"] == "swe":
        r0 = 0.25 + 0.05 * float(g.uniform(-1, 1))
        h = torch.where((X - 0.5) ** 2 + (Y - 0.5) ** 2 < r0 * r0, 2.0, 1.0) + 0.05 * wave
        q = torch.stack([h, torch.zeros_like(h), torch.zeros_like(h)])
    else:
        right, up = (X >= 0.5).expand(n, n), (Y >= 0.5).expand(n, n)
        which = torch.where(right, torch.where(up, 0, 3), torch.where(up, 1, 2))
        s = torch.tensor(QUADRANTS, dtype=torch.float64, device=dev)[which]  # (n, n, 4)
        rho, u, v, p = (s[..., k] for k in range(4))
        rho, p = rho * (1 + 0.05 * wave), p * (1 - 0.05 * wave)
        q = torch.stack([rho, rho * u, rho * v, p / (1.4 - 1.0) + 0.5 * rho * (u * u + v * v)])
    return q


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.float64, pin_memory=True).numpy()


def _perturb(q, solver, seed):
    """Smooth seeded waves on the mass (or, for a scalar, the value) of a refined mesh's state."""
    o, g = solver.options, np.random.default_rng(seed)
    lv = np.array(solver.leaves(), dtype=np.float64)
    h = 1.0 / (o.mx * np.exp2(lv[:, 0]))
    c = np.arange(-2, o.mx + 2) + 0.5
    X, Y = lv[:, 1, None] / KROOT + h[:, None] * c, lv[:, 2, None] / KROOT + h[:, None] * c
    wave = np.zeros((len(lv), o.ny, o.nx))
    for _ in range(3):
        kx, ky, px, py = (*g.integers(1, 6, 2), *g.uniform(0, 2 * math.pi, 2))
        wave += np.cos(2 * math.pi * ky * Y + py)[:, :, None] * np.cos(2 * math.pi * kx * X + px)[:, None, :] / 3
    amp = 1e-4 if o.solver_kind == fcb.SOLVER_GEOCLAW_FWAVE else 0.01
    f = 1.0 + amp * wave
    if o.claw_version == 5:
        q[..., :] *= f[..., None]
    else:
        q *= f[:, None]
    return q


def prepare(case, seed):
    if case["kind"] == "serve":
        reqs = []
        base = workloads.dam_break_requests(case["requests"], 1, maxlevels=(3, 4, 5), tfinal=(0.04, 0.08))
        g = np.random.default_rng(seed)
        for o in base:  # the mix of sizes is the case's, the dams are the seed's
            o.problem_params = (0.5, 0.5, float(g.uniform(0.1, 0.3)), float(g.uniform(1.5, 3.0)), 1.0)
            o.initial_dt = 0.9 / (o.mx * 4) / (o.problem_params[3] ** 0.5 + 1)
            reqs.append(o)
        server = fcb_serve.Server(64 << 30)
        outs = [np.zeros(1100 * o.meqn * o.ny * o.nx) for o in reqs]
        return {"case": case, "server": server, "requests": reqs, "outs": outs}
    solver = fcb.Solver(_options(case, seed))
    solver.initialize()
    state = {"case": case, "solver": solver, "t": 0.0, "dt": _dt(case)}
    if case["kind"] in ("uniform", "level"):
        q = _patches(_pad(_initial(case, seed), case["walls"]), case)
        state["out"] = _pinned(q.shape)
        torch.from_numpy(state["out"]).copy_(q)
        solver.set_q(state["out"])
    elif case["kind"] == "amr":
        solver.set_q(_perturb(solver.get_q(), solver, seed))
        state["out"] = _pinned(solver.get_q().shape)
    else:
        # room for the mesh at any time of the run: a refined ring of up to 24
        # patches' width around every level's front
        o = solver.options
        room = sum(min(4 ** l, 24 * 2 ** l) for l in range(o.minlevel, o.maxlevel + 1)) * o.brick ** 2
        state["out"] = _pinned(room * o.meqn * o.ny * o.nx)
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "serve":
        server = state["server"]
        ids = [server.submit(o) for o in state["requests"]]
        server.run_until_idle()
        sizes = []
        for rid, out in zip(ids, state["outs"]):
            q = server.get_q(rid)
            out[:q.size] = q.reshape(-1)
            sizes.append(q.shape[0])
            server.release(rid)
        return {"q": state["outs"], "patches": sizes}
    s, t, dt = state["solver"], state["t"], state["dt"]
    if case["kind"] == "run":
        s.initialize()
        s.run()
        s.get_q(state["out"])
        return {"q": state["out"], "patches": s.num_patches, "t": s.curr_time}
    cfl = 0.0
    if case["kind"] == "level":
        lv = case["maxlevel"]
        for _ in range(case["steps"]):
            cfl = max(cfl, s.update_single_step(lv, t, dt))
            t += dt
            s.ghost_update(lv, lv, t, 0)
    elif case["cfl_each_step"]:
        for _ in range(case["steps"]):
            cfl = max(cfl, s.advance_all_levels(t, dt))
            t += dt
    else:
        for _ in range(case["steps"]):
            s.advance_all_levels_async(t, dt)
            t += dt
        cfl = s.read_max_cfl()
    state["t"] = t
    return {"q": s.get_q(state["out"]), "cfl": cfl}


def _cells(case):
    """(cell updates of a pass, cells of the state) for the listed meshes: exact on
    meshes of one level, about the refined part's size elsewhere."""
    mx, lo, hi, steps = case["mx"], case["minlevel"], case["maxlevel"], case["steps"]
    if case["kind"] in ("uniform", "level"):
        n = _n(case) ** 2
        return n * steps, n
    if case["kind"] == "serve":
        # ~64 patches of each 16/32 request refined along a circle, 10 macro steps
        return case["requests"] * 64 * 576 * 40, case["requests"] * 64 * 576
    # a front of length ~1.6 refined to level hi, graded to the coarser levels around it
    blocks = 4 if case["equation"] == "filament" else 1
    patches = {l: min(4 ** l, 11 * 2 ** l) * blocks for l in range(lo, hi + 1)}
    cells = sum(patches.values()) * mx * mx
    updates = sum(p * 2 ** (l - lo) for l, p in patches.items()) * mx * mx * steps
    return updates, cells


def work(case):
    updates, cells = _cells(case)
    m = MEQN[case["equation"]]
    # the state read once and written once, and the frame that comes back
    return {"bytes": 24.0 * m * cells, "flops": OPS[case["equation"]] * updates}


# ---------------------------------------------------------------------------
# The same passes in plain torch, 64 bits: the wave-propagation step on the whole
# mesh (patches with exact ghost cells are a partition of it)
# ---------------------------------------------------------------------------
def _left(a):
    return torch.roll(a, 1, -1)


def _right(a):
    return torch.roll(a, -1, -1)


def _phi(limiter, r):
    if limiter == 1:
        return torch.clamp(r, 0.0, 1.0)
    if limiter == 2:
        return torch.maximum(torch.clamp(2 * r, 0.0, 1.0), torch.clamp(r, max=2.0))
    if limiter == 3:
        return (r + r.abs()) / (1 + r.abs())
    return torch.clamp(torch.minimum(torch.clamp((1 + r) / 2, max=2.0), 2 * r), min=0.0)


def _rp_advection(q, mu, mv, speed):
    d = q - _left(q)
    s = speed[None]
    return d[None], s, s.clamp(max=0.0) * d, s.clamp(min=0.0) * d, None


def _sfract(s_out, s_in, s):
    """Entropy fix of one acoustic wave: s_out and s_in its speeds on its two sides."""
    f = torch.where(s < 0, s, torch.zeros_like(s))
    return torch.where((s_out < 0) & (s_in > 0), s_out * (s_in - s) / (s_in - s_out), f)


def _rp_swe(q, mu, mv, speed):
    ql = _left(q)
    hl, hr = ql[0], q[0]
    sl, sr = hl.sqrt(), hr.sqrt()
    u, v = ((ql[k] / sl + q[k] / sr) / (sl + sr) for k in (mu, mv))
    a = ((hl + hr) / 2).sqrt()
    d = q - ql
    a1, a2, a3 = ((u + a) * d[0] - d[mu]) / (2 * a), d[mv] - v * d[0], (-(u - a) * d[0] + d[mu]) / (2 * a)
    w = torch.zeros((3,) + q.shape, dtype=q.dtype, device=q.device)
    w[0, 0], w[0, mu], w[0, mv] = a1, a1 * (u - a), a1 * v
    w[1, mv] = a2
    w[2, 0], w[2, mu], w[2, mv] = a3, a3 * (u + a), a3 * v
    s = torch.stack([u - a, u, u + a])
    s0 = ql[mu] / hl - hl.sqrt()
    h1 = hl + w[0, 0]
    s1 = (ql[mu] + w[0, mu]) / h1 - h1.sqrt()
    am = _sfract(s0, s1, s[0]) * w[0]
    s3r = q[mu] / hr + hr.sqrt()
    h3 = hr - w[2, 0]
    s3 = (q[mu] - w[2, mu]) / h3 + h3.sqrt()
    am = am + (s[1] <= 0) * (s[1] * w[1] + _sfract(s3, s3r, s[2]) * w[2])
    am = torch.where((s0 > 0) & (s[0] > 0), torch.zeros_like(am), am)
    return w, s, am, (s[:, None] * w).sum(0) - am, (u, v, a)


def _rpt_swe(asdq, mu, mv, roe):
    u, v, a = roe
    a1, a3 = ((v + a) * asdq[0] - asdq[mv]) / (2 * a), (-(v - a) * asdq[0] + asdq[mv]) / (2 * a)
    a2 = asdq[mu] - u * asdq[0]
    w = torch.zeros((3,) + asdq.shape, dtype=asdq.dtype, device=asdq.device)
    w[0, 0], w[0, mu], w[0, mv] = a1, a1 * u, a1 * (v - a)
    w[1, mu] = a2
    w[2, 0], w[2, mu], w[2, mv] = a3, a3 * u, a3 * (v + a)
    s = torch.stack([v - a, v, v + a])[:, None]
    return (s.clamp(max=0) * w).sum(0), (s.clamp(min=0) * w).sum(0)


def _rp_euler(q, mu, mv, speed):
    g1, gam = 1.4 - 1.0, 1.4
    ql = _left(q)

    def pressure(s):
        return g1 * (s[3] - 0.5 * (s[mu] ** 2 + s[mv] ** 2) / s[0])
    sl, sr = ql[0].sqrt(), q[0].sqrt()
    u, v = ((ql[k] / sl + q[k] / sr) / (sl + sr) for k in (mu, mv))
    h = ((ql[3] + pressure(ql)) / sl + (q[3] + pressure(q)) / sr) / (sl + sr)
    u2 = u * u + v * v
    a2 = g1 * (h - 0.5 * u2)
    a = a2.sqrt()
    d = q - ql
    a3 = g1 / a2 * ((h - u2) * d[0] + u * d[mu] + v * d[mv] - d[3])
    as_ = d[mv] - v * d[0]
    a4 = (d[mu] + (a - u) * d[0] - a * a3) / (2 * a)
    a1 = d[0] - a3 - a4
    w = torch.zeros((4,) + q.shape, dtype=q.dtype, device=q.device)
    w[0, 0], w[0, mu], w[0, mv], w[0, 3] = a1, a1 * (u - a), a1 * v, a1 * (h - u * a)
    w[1, mv], w[1, 3] = as_, as_ * v
    w[2, 0], w[2, mu], w[2, mv], w[2, 3] = a3, a3 * u, a3 * v, a3 * 0.5 * u2
    w[3, 0], w[3, mu], w[3, mv], w[3, 3] = a4, a4 * (u + a), a4 * v, a4 * (h + u * a)
    s = torch.stack([u - a, u, u, u + a])

    def sound(x):
        return (gam * pressure(x) / x[0]).sqrt()
    s0 = ql[mu] / ql[0] - sound(ql)
    x = ql + w[0]
    am = _sfract(s0, x[mu] / x[0] - sound(x), s[0]) * w[0]
    y = q - w[3]
    fix = _sfract(y[mu] / y[0] + sound(y), q[mu] / q[0] + sound(q), s[3])
    am = am + (s[1] < 0) * (s[1] * w[1] + s[2] * w[2] + fix * w[3])
    am = torch.where((s0 >= 0) & (s[0] > 0), torch.zeros_like(am), am)
    return w, s, am, (s[:, None] * w).sum(0) - am, (u, v, a, h, u2, g1 / a2)


def _rpt_euler(asdq, mu, mv, roe):
    u, v, a, h, u2, g1a2 = roe
    a3 = g1a2 * ((h - u2) * asdq[0] + u * asdq[mu] + v * asdq[mv] - asdq[3])
    a2 = asdq[mu] - u * asdq[0]
    a4 = (asdq[mv] + (a - v) * asdq[0] - a * a3) / (2 * a)
    a1 = asdq[0] - a3 - a4
    w = torch.zeros((3,) + asdq.shape, dtype=asdq.dtype, device=asdq.device)
    w[0, 0], w[0, mu], w[0, mv], w[0, 3] = a1, a1 * u, a1 * (v - a), a1 * (h - v * a)
    w[1, 0], w[1, mu], w[1, mv], w[1, 3] = a3, a3 * u + a2, a3 * v, a3 * 0.5 * u2 + a2 * u
    w[2, 0], w[2, mu], w[2, mv], w[2, 3] = a4, a4 * u, a4 * (v + a), a4 * (h + v * a)
    s = torch.stack([v - a, v, v + a])[:, None]
    return (s.clamp(max=0) * w).sum(0), (s.clamp(min=0) * w).sum(0)


def _sweep(case, q, dtd, mu, mv, normal, across):
    """One direction (the last axis) over all rows: the flux corrections at every
    interface, the transverse parts into the rows below and above, the speeds."""
    eq = case["equation"]
    rp = {"advection": _rp_advection, "swe": _rp_swe, "euler": _rp_euler}[eq]
    w, s, am, ap, roe = rp(q, mu, mv, normal)
    n2 = (w * w).sum(1)
    r = torch.where(s > 0, (_left(w) * w).sum(1), (w * _right(w)).sum(1)) / torch.where(n2 == 0, torch.ones_like(n2), n2)
    wl = torch.where((n2 == 0)[:, None], w, _phi(case["limiter"], r)[:, None] * w)
    cq = ((s.abs() * (1 - s.abs() * dtd))[:, None] * wl).sum(0)
    parts = []
    for asdq, at_left in ((am + cq, True), (ap - cq, False)):
        if eq == "advection":
            lo = across
            hi = torch.roll(across, -1, -2)
            if at_left:
                lo, hi = _left(lo), _left(hi)
            b = lo.clamp(max=0) * asdq, hi.clamp(min=0) * asdq
        else:
            b = (_rpt_swe if eq == "swe" else _rpt_euler)(asdq, mu, mv, roe)
        parts.append([-0.5 * dtd * x for x in b])
    down, up = (_right(parts[0][k]) + parts[1][k] for k in (0, 1))
    return am + 0.5 * cq, -ap + 0.5 * cq, down, up, s


def _turn(a):
    return a.transpose(-1, -2)


def _step(case, q, t, dt):
    """One step of the padded mesh: its new interior and the CFL number."""
    n = _n(case)
    dtd = dt * n
    u = v = None
    if case["equation"] == "advection":  # swirl velocities from the stream function's differences
        x = (torch.arange(n + 5, dtype=torch.float64, device=q.device) - 2) / n
        f = torch.sin(math.pi * x) ** 2
        psi = f[:, None] * f[None, :] / math.pi
        vt = math.cos(2 * math.pi * (t + dt / 2) / 2.0) * n
        u, v = vt * (psi[1:, :-1] - psi[:-1, :-1]), -vt * (psi[:-1, 1:] - psi[:-1, :-1])
    xm, xp, xd, xu, sx = _sweep(case, q, dtd, 1, 2, u, v)
    got = _sweep(case, _turn(q).contiguous(), dtd, 2, 1, None if v is None else _turn(v), None if u is None else _turn(u))
    ym, yp, yd, yu, sy = (_turn(a) for a in got)
    below, above = lambda a: torch.roll(a, 1, -2), lambda a: torch.roll(a, -1, -2)  # noqa: E731
    df = _right(xm) + yu + _right(yd) - (xp + _left(yu) + yd)
    dg = xu + above(xd) + above(ym) - (below(xu) + xd + yp)
    new = (q - dtd * df - dtd * dg)[:, 2:-2, 2:-2].contiguous()
    cfl = max(sx[:, 1:-1, 2:-1].abs().max().item(), sy[:, 2:-1, 1:-1].abs().max().item()) * dtd
    return new, cfl


def exact(case, seed):
    """A first pass on a mesh of one level.  Refined meshes and served solves go
    through hundreds of dependent regrid and ghost-exchange steps of leaves of
    several levels: far over the time a plain evaluation may take."""
    if case["kind"] not in ("uniform", "level"):
        return None
    q, t, dt, cfl = _initial(case, seed), 0.0, _dt(case), 0.0
    for _ in range(case["steps"]):
        q, c = _step(case, _pad(q, case["walls"]), t, dt)
        cfl = max(cfl, c)
        t += dt
    return {"q": _patches(_pad(q, case["walls"]), case).cpu().numpy(), "cfl": cfl}
