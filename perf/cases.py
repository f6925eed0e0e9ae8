"""Timed cases: what a program that uses this package has it do, through forestclaw_b200.Solver.

A pass is the stretch between two output frames of a run: a number of coarse steps of one
forest (or one batch of forests) and the read of q back to page-locked host memory.  Every
pass starts from the same saved step (restore_step), so passes can be repeated.  Four kinds:

  uniform  a forest of one level; the solution is known in 64 bits from a plain torch
           restatement of the wave-propagation method on the undivided grid (exact)
  amr      an adaptive, subcycled forest after some steps with regrids, as in mid-run
  batch    many independent adaptive forests in one solver (tsunami instances)
  run      a whole run from t = 0 with its CFL control and a regrid after every step

The frames of FP32-wave runs are kept in single precision, the type of their waves and of
the package's VTK frames; FP64 runs keep theirs in FP64.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import forestclaw_b200 as fb
from forestclaw_b200 import problems

PRESETS = {"swirl": problems.SWIRL, "dam": problems.DAM, "tsunami": problems.TSUNAMI,
           "bubble": problems.SHOCKBUBBLE, "sphere": problems.SPHERE}

# floating operations of one cell update, about (two Riemann solves with limiter, second-order
# and transverse corrections): counted from the formulas
FLOPS = {"swirl": 60, "sphere": 70, "dam": 500, "tsunami": 600, "bubble": 1100}


def listed():
    return [
        # scalar advection, uniform level 4 of 32x32 patches: the configuration of 200 fixed steps
        dict(name="swirl_u4_32_f64", kind="uniform", problem="swirl", f32=False, mx=32, level=4, mi=1, mj=1,
             limiter=4, order2=2, wall=False, steps=16),
        # the smallest call: four patches, one step, all latency and launches
        dict(name="swirl_u1_16_f64", kind="uniform", problem="swirl", f32=False, mx=16, level=1, mi=1, mj=1,
             limiter=4, order2=2, wall=False, steps=1),
        # radial dam on an adaptive forest, levels 3 to 7: the headline workload, in both forms
        dict(name="dam_amr37_16_f32", kind="amr", problem="dam", f32=True, mx=16, minlevel=3, maxlevel=7,
             time_sync=True, tuned=True, spinup=12, steps=16),
        dict(name="dam_amr37_16_f64", kind="amr", problem="dam", f32=False, mx=16, minlevel=3, maxlevel=7,
             time_sync=True, tuned=True, spinup=12, steps=8),
        # the same solver on a large uniform forest: throughput of the level update
        dict(name="dam_u6_16_f32", kind="uniform", problem="dam", f32=True, mx=16, level=6, mi=1, mj=1,
             limiter=4, order2=2, wall=False, steps=32),
        # small patches of a 3x2 brick between reflecting walls, van Leer limiter
        dict(name="dam_u4_8_f64_wall", kind="uniform", problem="dam", f32=False, mx=8, level=4, mi=3, mj=2,
             limiter=3, order2=2, wall=True, steps=16),
        # ensemble of tsunami forests of uneven depth, f-waves over bathymetry
        dict(name="tsunami_batch_8_f32", kind="batch", problem="tsunami", f32=True, mx=8, instances=32, minlevel=2,
             maxlevel=6, time_sync=True, tuned=True, spinup=4, steps=4),
        # one tsunami domain, uniform, FP64
        dict(name="tsunami_u5_16_f64", kind="uniform", problem="tsunami", f32=False, mx=16, level=5, mi=1, mj=1,
             limiter=4, order2=2, wall=False, steps=16),
        # shock hitting a bubble, exact Euler solver, adaptive levels 4 to 7
        dict(name="bubble_amr47_16_f32", kind="amr", problem="bubble", f32=True, mx=16, minlevel=4, maxlevel=7,
             time_sync=True, tuned=True, spinup=8, steps=4),
        dict(name="bubble_u4_16_f64", kind="uniform", problem="bubble", f32=False, mx=16, level=4, mi=2, mj=1,
             limiter=4, order2=2, wall=True, steps=16),
        # advection on the cubed sphere (six blocks, capacity and edge lengths from the mapping)
        dict(name="sphere_amr36_32_f32", kind="amr", problem="sphere", f32=True, mx=32, minlevel=3, maxlevel=6,
             time_sync=False, tuned=True, spinup=4, steps=8),
        # the radial dam's regression run from start to end: 5 steps, 5 regrids, time sync
        dict(name="dam_run15_16_f64", kind="run", problem="dam", f32=False, mx=16, minlevel=1, maxlevel=5, steps=5),
    ]


def draw(rng: random.Random):
    kind = rng.choice(("uniform", "uniform", "uniform", "amr", "amr", "batch", "run"))
    if kind == "uniform":
        problem = rng.choice(("swirl", "dam", "dam", "tsunami", "bubble"))
        f32 = rng.random() < 0.5
        mx = rng.choice((16, 32) if problem == "swirl" else (8, 16))
        mi, mj = (2, 1) if problem == "bubble" else (rng.randint(1, 5), rng.randint(1, 5))
        # patches, spread over their logarithm: 1 to about 1000 of 32x32, 4000 of 16x16, 8000 of 8x8
        most = {32: 1000, 16: 4000, 8: 8000}[mx]
        level = round(0.5 * math.log2(max(1.0, math.exp(rng.uniform(0.0, math.log(most))) / (mi * mj))))
        while level > 0 and mi * mj * 4 ** level > most:
            level -= 1
        return dict(kind=kind, problem=problem, f32=f32, mx=mx, level=level, mi=mi, mj=mj,
                    limiter=rng.choice((1, 2, 3, 4, 4, 4)), order2=rng.choice((1, 2, 2, 2)),
                    wall=problem == "bubble" or (problem == "dam" and rng.random() < 0.5), steps=rng.randint(4, 16))
    if kind == "amr":
        problem = rng.choice(("dam", "dam", "tsunami", "bubble", "sphere"))
        lo = {"dam": (1, 3), "tsunami": (1, 3), "bubble": (2, 4), "sphere": (2, 3)}[problem]
        minlevel = rng.randint(*lo)
        depth = rng.randint(1, 2 if problem == "sphere" else 3)
        return dict(kind=kind, problem=problem, f32=rng.random() < 0.5,
                    mx=rng.choice((16, 32) if problem == "sphere" else (8, 16)), minlevel=minlevel,
                    maxlevel=minlevel + depth, time_sync=problem != "sphere" and rng.random() < 0.75,
                    tuned=rng.random() < 0.5, spinup=4, steps=rng.randint(2, 8))
    if kind == "batch":
        minlevel = rng.randint(1, 2)
        return dict(kind=kind, problem="tsunami", f32=rng.random() < 0.5, mx=rng.choice((8, 16)),
                    instances=rng.randint(3, 24), minlevel=minlevel, maxlevel=minlevel + rng.randint(1, 3),
                    time_sync=rng.random() < 0.75, tuned=rng.random() < 0.5, spinup=2, steps=rng.randint(2, 6))
    return dict(kind="run", problem="dam", f32=False, mx=rng.choice((8, 16)), minlevel=rng.randint(1, 2),
                maxlevel=rng.randint(3, 5), steps=5)


def _sides(problem):
    return (0.0, 2.0, 0.0, 1.0) if problem == "bubble" else (0.0, 1.0, 0.0, 1.0) if problem == "swirl" else \
        (-1.0, 1.0, -1.0, 1.0)


def _cells(case) -> float:
    """Interior cells updated in one pass, about (adaptive forests follow their fronts)."""
    mx2 = case["mx"] ** 2
    if case["kind"] == "uniform":
        return case["steps"] * mx2 * case["mi"] * case["mj"] * 4.0 ** case["level"]
    lo, hi = case["minlevel"], case["maxlevel"]
    # patches along the fronts double per level (the dam's rings more than that); a subcycled
    # step takes 2^(l - lo) substeps of level l; a batch's instances end at up to two levels less
    base = {"dam": 1.4 * hi, "tsunami": 3.5, "bubble": 5.5, "sphere": 4.5}[case["problem"]]
    blocks = {"bubble": 2, "sphere": 6}.get(case["problem"], 1)
    per_step = sum(min(blocks * 4.0 ** l, base * 2.0 ** l) * 2.0 ** (l - lo) for l in range(lo, hi + 1)) * mx2
    return case["steps"] * per_step * 0.4 * case["instances"] if case["kind"] == "batch" else case["steps"] * per_step


def work(case):
    p = PRESETS[case["problem"]]
    cells = _cells(case)
    # q read and written and aux read once per cell update
    return {"bytes": cells * 8.0 * (2 * p["meqn"] + p["maux"]), "flops": cells * FLOPS[case["problem"]]}


# ---------------------------------------------------------------------------------------
# solvers
# ---------------------------------------------------------------------------------------
def _parameters(problem, rng):
    """The physical parameters a user varies from run to run.  Adaptive forests take the
    preset's, so that their leaves are the same for every seed."""
    if problem == "dam":
        return dict(x0=rng.uniform(-0.03, 0.03), y0=rng.uniform(-0.03, 0.03), r0=rng.uniform(0.28, 0.32),
                    hin=rng.uniform(1.9, 2.1))
    if problem == "bubble":
        return dict(x0=rng.uniform(0.48, 0.52), y0=rng.uniform(0.48, 0.52), r0=rng.uniform(0.19, 0.21),
                    rhob=rng.uniform(0.13, 0.15))
    if problem == "tsunami":
        return dict(pdata=_tsunami(rng))
    return {}


def _tsunami(rng):
    """Bathymetry centre and two Gaussian humps of the surface."""
    pd = [rng.uniform(-0.5, 0.5), rng.uniform(-0.5, 0.5), 2.0]
    for _ in range(2):
        pd += [rng.uniform(0.1, 0.2), rng.uniform(0.1, 0.15), rng.uniform(-0.6, 0.6), rng.uniform(-0.6, 0.6)]
    return tuple(pd)


def _solver(case, **kw):
    o = problems.options(PRESETS[case["problem"]], mx=case["mx"], my=case["mx"],
                         precision=fb.PREC_FP32WAVE if case["f32"] else fb.PREC_FP64, **kw)
    return fb.Solver(o)


def _frame(s, f32):
    """Page-locked memory for one frame of q, and the single-precision copy of FP32-wave runs."""
    shape = (s.num_patches, s.opts.meqn, s.ny, s.nx)
    return torch.empty(shape, dtype=torch.float64, pin_memory=True), torch.zeros(shape if f32 else 0, dtype=torch.float32)


def _install(s, case, rng):
    """The state the pass starts from: the current q with smooth waves of the seed on it."""
    frame, single = _frame(s, case["f32"])
    s.get_q_ptr(frame.data_ptr())
    q = frame.cuda()
    lev, _, gx, gy = (torch.from_numpy(a.copy()).cuda() for a in s.patch_info().T)
    at = torch.arange(-2, case["mx"] + 2, device="cuda") + 0.5
    x, y = ((g[:, None] + at / case["mx"]) / 2.0 ** lev[:, None] for g in (gx, gy))
    waves = torch.zeros_like(x[:, None, :] + y[:, :, None])
    for _ in range(3):
        kx, ky, ph = rng.randint(1, 6), rng.randint(1, 6), rng.uniform(0, 6.28)
        waves += torch.sin(math.pi * (kx * x[:, None, :] + ky * y[:, :, None]) + ph)
    q *= 1.0 + {"tsunami": 5e-4}.get(case["problem"], 5e-3) * waves[:, None]
    frame.copy_(q)
    s.set_q_ptr(frame.data_ptr())
    if case["kind"] == "amr":
        s.ghost_update(case["minlevel"], case["maxlevel"], 0.0)
    s.save_step()
    return frame, single


def prepare(case, seed):
    rng = random.Random(seed)
    return {"uniform": _prepare_uniform, "amr": _prepare_amr, "batch": _prepare_batch, "run": _prepare_run}[
        case["kind"]](case, rng)


def _prepare_uniform(case, rng):
    L = case["level"]
    par, q = _initial(case, rng)
    kw = dict(_uniform_options(case), **par)
    s = _solver(case, minlevel=L, maxlevel=L, mi=case["mi"], mj=case["mj"], **kw)
    s.initialize()                               # forest and aux
    frame, single = _frame(s, case["f32"])
    frame.copy_(_patches(case, q))
    s.set_q_ptr(frame.data_ptr())
    s.ghost_update(L, L, 0.0)
    s.save_step()
    return dict(kind="uniform", solver=s, frame=frame, single=single, t=0.0, dt=_uniform_dt(case), steps=case["steps"])


def _prepare_amr(case, rng):
    problem, lo = case["problem"], case["minlevel"]
    s = _solver(case, minlevel=lo, maxlevel=case["maxlevel"], subcycle=1, time_sync=int(case["time_sync"]))
    s.initialize()
    n = case["mx"] << lo
    if problem == "sphere":
        dt = 0.45 * (0.5 * math.pi / n) / (2.0 * math.pi) / 2.0
    else:
        a, b, c, d = _sides(problem)
        dt = 0.8 * (d - c) / n / {"dam": 2.1, "tsunami": 1.5, "bubble": 3.4}[problem]
    t = 0.0
    for k in range(case["spinup"]):
        cfl = s.advance(t, dt)
        t += dt
        dt *= 0.85 / cfl
        if k % 4 == 3 or k + 1 == case["spinup"]:
            s.regrid()
    if case["tuned"]:
        s.autotune(3)
    frame, single = _install(s, case, rng)
    return dict(kind="amr", solver=s, frame=frame, single=single, t=t, dt=dt, steps=case["steps"])


def _prepare_batch(case, rng):
    lo, hi, mx = case["minlevel"], case["maxlevel"], case["mx"]
    insts, own = [], random.Random(case["instances"])
    for k in range(case["instances"]):           # uneven depths; the leaves are the same for every seed
        a = lo + k % 2
        insts.append(dict(minlevel=a, maxlevel=max(a, hi - k % 3), pdata=_tsunami(own)))
    s = _solver(case, minlevel=0, maxlevel=0, subcycle=1, time_sync=int(case["time_sync"]))
    s.set_instances(insts)
    s.initialize()
    dt = np.array([0.8 * (2.0 / (mx << x["minlevel"])) / 1.5 for x in insts])
    for k in range(case["spinup"]):
        dt = dt * 0.85 / s.advance_instances(dt)
    s.regrid()
    if case["tuned"]:
        s.autotune(3)
    frame, single = _install(s, case, rng)
    return dict(kind="batch", solver=s, frame=frame, single=single, dt=dt, steps=case["steps"])


def _prepare_run(case, rng):
    # the options of the radial dam's regression run, cell averages of the disc included
    s = _solver(case, minlevel=case["minlevel"], maxlevel=case["maxlevel"], subcycle=1, time_sync=1,
                ax=-2.5, bx=2.5, ay=-2.5, by=2.5, r0=0.5, hin=2.0 + rng.uniform(-1e-4, 1e-4),
                smooth_refine=1, smooth_level=case["maxlevel"] - 1, refinement_criteria=fb.TAG_GRADIENT,
                refine_threshold=0.5, coarsen_threshold=0.25, qinit_cellave=1, regrid_interval=1, nout=1,
                tfinal=0.4, initial_dt=0.0625, max_cfl=1.0, desired_cfl=0.9)
    return dict(kind="run", solver=s)


def run(state):
    s = state["solver"]
    if state["kind"] == "run":
        s.initialize()
        counters = s.run()
        return {"q": s.get_q(), "mass": s.mass(), "advances": counters["count_amr_advance"],
                "patches": counters["global_num_patches"]}
    s.restore_step()
    cfl = []
    if state["kind"] == "batch":
        for _ in range(state["steps"]):
            cfl.append(s.advance_instances(state["dt"]))
    else:
        t, dt = state["t"], state["dt"]
        for _ in range(state["steps"]):
            cfl.append(s.advance(t, dt))
            t += dt
    frame, single, cfl = state["frame"], state["single"], np.array(cfl)
    s.get_q_ptr(frame.data_ptr())
    return {"q": single.copy_(frame), "cfl": cfl.astype(np.float32)} if single.numel() else {"q": frame, "cfl": cfl}


# ---------------------------------------------------------------------------------------
# uniform forests: inputs, and the same steps in plain torch (64 bits) on the undivided grid
# ---------------------------------------------------------------------------------------
def _uniform_options(case):
    p, problem = PRESETS[case["problem"]], case["problem"]
    kw = dict(order=(2, case["order2"]), mthlim=(case["limiter"],) * p["mwaves"])
    if case["wall"] and problem != "bubble":
        kw["mthbc"] = (3, 3, 3, 3)
    return kw


def _grid(case):
    ax, bx, ay, by = _sides(case["problem"])
    nx, ny = case["mi"] * case["mx"] << case["level"], case["mj"] * case["mx"] << case["level"]
    return nx, ny, ax, ay, (bx - ax) / nx, (by - ay) / ny


def _uniform_dt(case):
    _, _, _, _, dx, dy = _grid(case)
    return 0.8 * min(dx, dy) / {"swirl": 1.0, "dam": 2.2, "tsunami": 1.5, "bubble": 3.6}[case["problem"]]


def _coordinates(case, centred=True):
    """Padded cell coordinates (centres, or lower left corners), 2 ghost cells around."""
    nx, ny, ax, ay, dx, dy = _grid(case)
    off = 0.5 if centred else 0.0
    x = ax + (torch.arange(-2, nx + 2, dtype=torch.float64, device="cuda") + off) * dx
    y = ay + (torch.arange(-2, ny + 2, dtype=torch.float64, device="cuda") + off) * dy
    return x[None, :], y[:, None]


def _initial(case, rng):
    """Solver parameters and the padded global field q[meqn, ny + 4, nx + 4]: the problem's own
    initial state with smooth waves on it."""
    problem = case["problem"]
    par = _parameters(problem, rng)
    x, y = _coordinates(case)
    waves = torch.zeros_like(x + y)
    for _ in range(4):
        kx, ky, ph, amp = rng.randint(1, 6), rng.randint(1, 6), rng.uniform(0, 6.28), rng.uniform(0.3, 1.0)
        waves += amp * torch.sin(math.pi * (kx * x + ky * y) + ph)
    if problem == "swirl":
        q = (torch.where(x < 0.5, 1.0, 0.0) + 0.05 * waves)[None]
    elif problem == "dam":
        r2 = (x - par["x0"]) ** 2 + (y - par["y0"]) ** 2
        h = torch.where(r2 < par["r0"] ** 2, par["hin"], 1.0) + 0.01 * waves
        q = torch.stack([h, 0.02 * waves.flip(0), 0.02 * waves.flip(1)])
    elif problem == "tsunami":
        pd = par["pdata"]
        eta = 0.005 * waves
        for k in range(int(pd[2])):
            a, w, cx, cy = pd[3 + 4 * k:7 + 4 * k]
            eta = eta + a * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / w ** 2)
        q = torch.stack([eta - _bathymetry(case, par), torch.zeros_like(eta), torch.zeros_like(eta)])
    else:
        rho = torch.where((x - par["x0"]) ** 2 + (y - par["y0"]) ** 2 < par["r0"] ** 2, par["rhob"], 1.0)
        rho, p = rho * (1 + 0.01 * waves), 1 + 0.01 * waves.flip(1)
        u, v = 0.02 * waves.flip(0) + 0 * y, 0.02 * waves
        q = torch.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])
        q = torch.where((x < 0.2)[None], _inflow(par)[:, None, None], q)
    _boundary(case, par, q)
    return par, q.contiguous()


def _bathymetry(case, par):
    x, y = _coordinates(case)
    return -1.0 + 0.5 * torch.exp(-50.0 * ((x - par["pdata"][0]) ** 2 + (y - par["pdata"][1]) ** 2))


def _inflow(par):
    """The state behind a Mach 1.22 shock into (rho, p) = (1, 1) at rest."""
    g, m = 1.4, 1.22
    p = 1 + 2 * g * (m * m - 1) / (g + 1)
    r = ((g - 1) + (g + 1) * p) / ((g + 1) + (g - 1) * p)
    u = (p - 1) / math.sqrt(g) / math.sqrt(0.5 * (g + 1) / g * p + 0.5 * (g - 1) / g)
    return torch.tensor([r, r * u, 0.0, 0.5 * r * u * u + p / (g - 1)], dtype=torch.float64, device="cuda")


def _boundary(case, par, q):
    """Two ghost cells on each side, x sides first: extrapolation, reflecting walls or inflow."""
    wall = case["wall"]
    for axis, mom in ((2, 1), (1, 2)):
        a = q.transpose(1, 2) if axis == 1 else q
        for side in (0, 1):
            for g in (0, 1):
                ghost = 1 - g if side == 0 else a.shape[2] - 2 + g
                first = 2 if side == 0 else a.shape[2] - 3
                mirror = 2 + g if side == 0 else a.shape[2] - 3 - g
                bubble_x = case["problem"] == "bubble" and axis == 2
                if bubble_x and side == 0:
                    a[:, :, ghost] = _inflow(par)[:, None]
                elif wall and not bubble_x:
                    a[:, :, ghost] = a[:, :, mirror]
                    a[mom, :, ghost] = -a[mom, :, mirror]
                else:
                    a[:, :, ghost] = a[:, :, first]


def _patches(case, q):
    """The padded global field as patches [n, meqn, my + 4, mx + 4], Morton order."""
    mx = case["mx"]
    p = q.unfold(1, mx + 4, mx).unfold(2, mx + 4, mx)          # [m, py, px, my + 4, mx + 4]
    _, py, px = p.shape[:3]
    key = lambda i, j: sum(((i >> b) & 1) << 2 * b | ((j >> b) & 1) << 2 * b + 1 for b in range(16))  # noqa: E731
    order = sorted(((key(i, j), j * px + i) for j in range(py) for i in range(px)))
    at = torch.tensor([k for _, k in order], device=q.device)
    return p.permute(1, 2, 0, 3, 4).reshape(py * px, *p.shape[:1], mx + 4, mx + 4)[at].contiguous()


def _limiter(kind, r):
    zero = torch.zeros_like(r)
    if kind == 1:
        return torch.maximum(zero, r.clamp(max=1.0))
    if kind == 2:
        return torch.maximum(torch.maximum(zero, (2 * r).clamp(max=1.0)), r.clamp(max=2.0))
    if kind == 3:
        return (r + r.abs()) / (1 + r.abs())
    return torch.maximum(zero, torch.minimum(((1 + r) / 2).clamp(max=2.0), 2 * r))


def _dot(a, b):
    return (a * b).sum(1)


class _Advection:
    """aux[0], aux[1]: velocities at the left and lower edge of each cell."""
    fwave = False

    def normal(self, ql, qr, al, ar):
        w, s = (qr - ql)[None], ar[0][None]
        return w, s, s.clamp(max=0) * w[0], s.clamp(min=0) * w[0], None

    def transverse(self, ex, ql, qr, below, here, above, a):
        return here[1].clamp(max=0) * a, above[1].clamp(min=0) * a


class _Roe:
    """Shallow water, Roe averages with the Harten-Hyman entropy fix, g = 1."""
    fwave = False

    def normal(self, ql, qr, al, ar):
        hl, hr = ql[0], qr[0]
        rl, rr = hl.sqrt(), hr.sqrt()
        u, v = ((ql[m] / rl + qr[m] / rr) / (rl + rr) for m in (1, 2))
        a = (0.5 * (hl + hr)).sqrt()
        d = qr - ql
        a1, a2, a3 = ((u + a) * d[0] - d[1]) / (2 * a), d[2] - v * d[0], ((a - u) * d[0] + d[1]) / (2 * a)
        z = torch.zeros_like(u)
        w = torch.stack([torch.stack([a1, a1 * (u - a), a1 * v]), torch.stack([z, z, a2]),
                         torch.stack([a3, a3 * (u + a), a3 * v])])
        s = torch.stack([u - a, u, u + a])
        c = lambda q: (q[1] / q[0], q[0].sqrt())  # noqa: E731
        (ul, cl), (ur, cr) = c(ql), c(qr)
        (u1, c1), (u3, c3) = c(ql + w[0]), c(qr - w[2])
        s0, s1, s3, s03 = ul - cl, u1 - c1, u3 + c3, ur + cr
        frac1 = torch.where((s0 < 0) & (s1 > 0), s0 * (s1 - s[0]) / (s1 - s0), s[0].clamp(max=0))
        trans3 = (s3 < 0) & (s03 > 0)
        frac3 = torch.where(trans3, s3 * (s03 - s[2]) / (s03 - s3), s[2].clamp(max=0))
        super_l = (s0 > 0) & (s[0] > 0)
        am = frac1 * w[0] + torch.where(s[1] > 0, z, s[1]) * w[1] + torch.where(s[1] > 0, z, frac3) * w[2]
        am = torch.where(super_l, torch.zeros_like(am), am)
        return w, s, am, (s[:, None] * w).sum(0) - am, (u, v, a)

    def transverse(self, ex, ql, qr, below, here, above, q):
        u, v, a = ex
        a1, a2, a3 = ((v + a) * q[0] - q[2]) / (2 * a), q[1] - u * q[0], ((a - v) * q[0] + q[2]) / (2 * a)
        z = torch.zeros_like(u)
        w = [torch.stack([a1, a1 * u, a1 * (v - a)]), torch.stack([z, a2, z]), torch.stack([a3, a3 * u, a3 * (v + a)])]
        s = (v - a, v, v + a)
        return sum(x.clamp(max=0) * y for x, y in zip(s, w)), sum(x.clamp(min=0) * y for x, y in zip(s, w))


class _FWave:
    """Shallow water over bathymetry aux[0] as f-waves, g = 1; the water is deep everywhere."""
    fwave = True

    def normal(self, ql, qr, al, ar):
        hl, hr = ql[0], qr[0]
        ul, vl, ur, vr = ql[1] / hl, ql[2] / hl, qr[1] / hr, qr[2] / hr
        cl, cr = hl.sqrt(), hr.sqrt()
        u, c = (cl * ul + cr * ur) / (cl + cr), (0.5 * (hl + hr)).sqrt()
        f1 = qr[1] - ql[1]
        f2 = 0.5 * hr ** 2 + hr * ur ** 2 - 0.5 * hl ** 2 - hl * ul ** 2 + 0.5 * (hl + hr) * (ar[0] - al[0])
        f3 = hr * ur * vr - hl * ul * vl
        s1, s3 = torch.minimum(ul - cl, u - c), torch.maximum(ur + cr, u + c)
        b1, b3 = (s3 * f1 - f2) / (s3 - s1), (f2 - s1 * f1) / (s3 - s1)
        z = torch.zeros_like(u)
        w = torch.stack([torch.stack([b1, b1 * s1, b1 * vl]), torch.stack([z, z, f3 - b1 * vl - b3 * vr]),
                         torch.stack([b3, b3 * s3, b3 * vr])])
        s = torch.stack([s1, 0.5 * (s1 + s3), s3])
        right = torch.where(s.signbit(), 0.0, 1.0)[:, None]
        return w, s, ((1 - right) * w).sum(0), (right * w).sum(0), None

    def transverse(self, ex, ql, qr, below, here, above, a):
        hl, hr = ql[0], qr[0]
        ul, vl, ur, vr = ql[1] / hl, ql[2] / hl, qr[1] / hr, qr[2] / hr
        cl, cr = hl.sqrt(), hr.sqrt()
        u, v, c = (ul * cl + ur * cr) / (cl + cr), (vl * cl + vr * cr) / (cl + cr), (0.5 * (hl + hr)).sqrt()
        s1, s3 = torch.minimum(v - c, vl - cl), torch.maximum(v + c, vr + cr)
        b1, b2, b3 = (s3 * a[0] - a[2]) / (s3 - s1), a[1] - u * a[0], (a[2] - s1 * a[0]) / (s3 - s1)
        one, z = torch.ones_like(u), torch.zeros_like(u)
        w = [b1 * torch.stack([one, u, s1]), b2 * torch.stack([z, one, z]), b3 * torch.stack([one, u, s3])]
        s = (s1, u, s3)
        return sum(x.clamp(max=0) * y for x, y in zip(s, w)), sum(x.clamp(min=0) * y for x, y in zip(s, w))


class _Euler:
    """2D Euler, gamma = 1.4, exact Riemann solver (Newton on the star pressure), Roe-type
    transverse split."""
    fwave = False
    g = 1.4

    def _side(self, p, r, ps, c):
        g = self.g
        shock = p > ps
        q = ((2 / (g + 1) / r) / ((g - 1) / (g + 1) * ps + p)).sqrt()
        z = (p / ps) ** ((g - 1) / (2 * g))
        f = torch.where(shock, (p - ps) * q, 2 * c / (g - 1) * (z - 1))
        d = torch.where(shock, (1 - 0.5 * (p - ps) / ((g - 1) / (g + 1) * ps + p)) * q, z * ps / p / (r * c))
        return f, d

    def normal(self, ql, qr, al, ar):
        g = self.g
        prim = lambda q: (q[0], q[1] / q[0], q[2] / q[0],  # noqa: E731
                          (g - 1) * (q[3] - 0.5 * (q[1] ** 2 + q[2] ** 2) / q[0]))
        (rl, ul, vl, pl), (rr, ur, vr, pr) = prim(ql), prim(qr)
        cl, cr = (g * pl / rl).sqrt(), (g * pr / rr).sqrt()
        p = (0.5 * (pl + pr) - 0.125 * (ur - ul) * (rl + rr) * (cl + cr)).clamp(min=1e-6)
        for _ in range(8):
            (fl, dl), (fr, dr) = self._side(p, rl, pl, cl), self._side(p, rr, pr, cr)
            p = (p - (fl + fr + ur - ul) / (dl + dr)).clamp(min=1e-6)
        (fl, _), (fr, _) = self._side(p, rl, pl, cl), self._side(p, rr, pr, cr)
        us = 0.5 * (ul + ur + fr - fl)
        still = (pl == pr) & (ul == ur)
        p, us = torch.where(still, pl, p), torch.where(still, ul, us)
        k = (g - 1) / (g + 1)
        star = lambda r, ps: torch.where(p > ps, r * (p / ps + k) / (k * p / ps + 1), r * (p / ps) ** (1 / g))  # noqa: E731
        sl, sr = star(rl, pl), star(rr, pr)
        bl, br = (g * p / sl).sqrt(), (g * p / sr).sqrt()
        speed = lambda ps: ((g + 1) / (2 * g) * p / ps + (g - 1) / (2 * g)).sqrt()  # noqa: E731
        s1 = torch.where(p > pl, ul - cl * speed(pl), ul - cl)
        s3 = torch.where(p > pr, ur + cr * speed(pr), ur + cr)
        state = lambda r, u, v, p: torch.stack([r, r * u, r * v, p / (g - 1) + 0.5 * r * (u * u + v * v)])  # noqa: E731
        qsl, qsr = state(sl, us, vl, p), state(sr, us, vr, p)
        w = torch.stack([qsl - ql, qsr - qsl, qr - qsr])
        # the state on the interface
        left = us >= 0
        fan = lambda sgn, r, u, c, ps: (  # noqa: E731
            r * (2 / (g + 1) + sgn * k / c * u) ** (2 / (g - 1)), 2 / (g + 1) * (sgn * c + (g - 1) / 2 * u),
            ps * (2 / (g + 1) + sgn * k / c * u) ** (2 * g / (g - 1)))
        fl0, fr0 = fan(1, rl, ul, cl, pl), fan(-1, rr, ur, cr, pr)
        keep_l = s1 >= 0
        star_l = torch.where(p > pl, ~keep_l, ~keep_l & (us - bl < 0))
        keep_r = s3 <= 0
        star_r = torch.where(p > pr, ~keep_r, ~keep_r & (us + br > 0))
        pick = lambda a, sa, fa, b, sb, fb_: torch.where(  # noqa: E731
            left, torch.where(keep_l, a, torch.where(star_l, sa, fa)), torch.where(keep_r, b, torch.where(star_r, sb, fb_)))
        r0 = pick(rl, sl, fl0[0], rr, sr, fr0[0])
        u0 = pick(ul, us, fl0[1], ur, us, fr0[1])
        p0 = pick(pl, p, fl0[2], pr, p, fr0[2])
        q0 = state(r0, u0, torch.where(left, vl, vr), p0)
        flux = lambda q, u, p: torch.stack([q[1], q[1] * u + p, q[2] * u, u * (q[3] + p)])  # noqa: E731
        f0 = flux(q0, u0, p0)
        hl, hr = rl.sqrt(), rr.sqrt()
        avg = lambda a, b: (a * hl + b * hr) / (hl + hr)  # noqa: E731
        u, v, h = avg(ul, ur), avg(vl, vr), avg((ql[3] + pl) / rl, (qr[3] + pr) / rr)
        return w, torch.stack([s1, us, s3]), f0 - flux(ql, ul, pl), flux(qr, ur, pr) - f0, (u, v, h)

    def transverse(self, ex, ql, qr, below, here, above, q):
        u, v, h = ex
        a2 = (self.g - 1) * (h - 0.5 * (u * u + v * v))
        a = a2.sqrt()
        b3 = (self.g - 1) / a2 * ((h - u * u - v * v) * q[0] + u * q[1] + v * q[2] - q[3])
        b2 = q[1] - u * q[0]
        b4 = (q[2] + (a - v) * q[0] - a * b3) / (2 * a)
        b1 = q[0] - b3 - b4
        w = [torch.stack([b1, b1 * u, b1 * (v - a), b1 * (h - v * a)]),
             torch.stack([b3, b3 * u + b2, b3 * v, b3 * 0.5 * (u * u + v * v) + b2 * u]),
             torch.stack([b4, b4 * u, b4 * (v + a), b4 * (h + v * a)])]
        s = (v - a, v, v + a)
        return sum(x.clamp(max=0) * y for x, y in zip(s, w)), sum(x.clamp(min=0) * y for x, y in zip(s, w))


SOLVERS = {"swirl": _Advection, "dam": _Roe, "tsunami": _FWave, "bubble": _Euler}


def _sweep(rp, q, aux, lam, limiter, order2):
    """One x sweep over the padded field: the fluctuation fluxes (fm, fp) of every interface
    i (between cells i and i + 1), the transverse fluxes into the lower and the upper face of
    every cell, and the largest CFL number.  aux: padded like q, or None."""
    ql, qr = q[..., :-1], q[..., 1:]
    al, ar = (aux[..., :-1], aux[..., 1:]) if aux is not None else (None, None)
    w, s, am, ap, ex = rp.normal(ql, qr, al, ar)
    cfl = (s[:, 1:-1, 1:-1].abs() * lam).max()       # as a patch: not on its outermost rows and interfaces
    wl, wr, wi, si = w[..., :-2], w[..., 2:], w[..., 1:-1], s[..., 1:-1]
    norm = _dot(wi, wi)
    r = torch.where(si > 0, _dot(wl, wi), _dot(wi, wr)) / torch.where(norm == 0, 1.0, norm)
    w = w.clone()
    w[..., 1:-1] = torch.where(norm == 0, 1.0, _limiter(limiter, r))[:, None] * wi
    strength = torch.where(s.signbit(), -1.0, 1.0) if rp.fwave else s.abs()
    cq = ((strength * (1 - s.abs() * lam))[:, None] * w).sum(0)
    fm, fp = am + 0.5 * cq, 0.5 * cq - ap
    if order2 == 2:
        am, ap = am + cq, ap - cq
    lower, upper = torch.zeros_like(q), torch.zeros_like(q)
    row = lambda a, k: None if a is None else torch.roll(a, -k, 1)  # noqa: E731
    for part, cells, a in ((am, slice(0, -1), al), (ap, slice(1, None), ar)):
        bm, bp = rp.transverse(ex, ql, qr, row(a, -1), a, row(a, 1), part)
        lower[..., cells] -= 0.5 * lam * bm
        upper[..., cells] -= 0.5 * lam * bp
    return fm, fp, lower, upper, cfl


def _turn(problem, a, field):
    """Rows and columns exchanged; normal and tangential components with them."""
    if a is None:
        return None
    a = a.transpose(1, 2)
    if problem == "swirl":
        return a[[1, 0]] if not field else a
    return a[[0, 2, 1, 3][:a.shape[0]]] if field else a


def exact(case, seed):
    """q and the CFL numbers of a pass over a uniform forest; adaptive forests have no undivided grid."""
    if case["kind"] != "uniform":
        return None
    problem = case["problem"]
    par, q = _initial(case, random.Random(seed))
    nx, ny, ax, ay, dx, dy = _grid(case)
    dt, rp, t, cfls = _uniform_dt(case), SOLVERS[problem](), 0.0, []
    aux = _bathymetry(case, par)[None] if problem == "tsunami" else None
    for _ in range(case["steps"]):
        if problem == "swirl":
            vt = math.cos(2.0 * math.pi * (t + dt / 2.0) / PRESETS["swirl"]["tperiod"])
            x, y = _coordinates(case, centred=False)
            psi = lambda x, y: (torch.sin(math.pi * x) ** 2 * torch.sin(math.pi * y) ** 2) / math.pi  # noqa: E731
            aux = torch.stack([vt / dy * (psi(x, y + dy) - psi(x, y)), -vt / dx * (psi(x + dx, y) - psi(x, y))])
        fm, fp, gl, gu, cx = _sweep(rp, q, aux, dt / dx, case["limiter"], case["order2"])
        hm, hp, fl, fu, cy = _sweep(rp, _turn(problem, q, True), _turn(problem, aux, False), dt / dy, case["limiter"],
                                    case["order2"])
        back = lambda a: _turn(problem, a, True)  # noqa: E731
        hm, hp, fl, fu = back(hm), back(hp), back(fl), back(fu)
        across = gl[:, 1:, :] + gu[:, :-1, :]              # on the faces between rows j and j + 1
        along = fl[:, :, 1:] + fu[:, :, :-1]
        fm, fp, hm, hp = fm + along, fp + along, hm + across, hp + across
        q = q.clone()
        q[:, 1:-1, 1:-1] -= dt / dx * (fm[:, 1:-1, 1:] - fp[:, 1:-1, :-1]) + dt / dy * (hm[:, 1:, 1:-1] - hp[:, :-1, 1:-1])
        _boundary(case, par, q)
        cfls.append(max(float(cx), float(cy)))
        t += dt
    return {"q": _patches(case, q), "cfl": np.array(cfls)}
