"""Timed cases of the DFSPH solver through its public Python interface (DFSPHCUDA).

A frame is what a simulation program does between two pictures: it hands the solver the particles'
state, advances it one time step (after moving the walls or a body), and reads positions and velocities
back. A search is the neighbour search alone (neighbors_search and its counts), which
programs call that bring their own solver. The fluid is a disordered block near rest density in a tank
of single-layer walls, moving like the flow in a sloshing tank; sizes, radii, tolerances and modes are
those of the benchmark configurations, the tests and the wave tank.

Run-time inputs live in pinned host memory, as the solver's interface takes them from the host.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from splishsplash_for_cuda_b200.dfsph import DFSPHCUDA
from splishsplash_for_cuda_b200.scene import Configuration, Scene, box_wall

RHO0 = 1000.0
FLUID_SPACING = 0.8 ** (1.0 / 3.0)  # lattice spacing over 2r at rest density, particle mass 0.8 rho0 (2r)^3;
# a case's "spacing" scales it: 1 is compressed everywhere by its disorder (tens of iterations), 1.006 and
# above a fluid that was solved in the step before (the solvers' least iterations)
WALL_GAP = 1.14                     # first lattice plane to the wall, in lattice spacings


def _case(name=None, nx=30, ny=30, nz=30, radius=0.025, kind="frame", precision=32, cfl=True, dt=0.0006,
          max_error=0.01, divergence=True, viscosity=0.01, walls="static", learned=False, spacing=1.006):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, radius=radius, precision=precision, cfl=cfl, dt=dt,
             max_error=max_error, divergence=divergence, viscosity=viscosity, walls=walls, learned=learned, spacing=spacing)
    return c if name is None else dict(name=name, **c)


def listed():
    return [
        # the smallest scene of the tests and of the smoke run: an interactive program's step
        _case("pool_1k", 10, 10, 10, 0.025, dt=0.0015, cfl=False),
        # the small dam break
        _case("dam_27k", 30, 30, 30, 0.025, dt=0.0015),
        # a rigid body driven through the fluid, with the fluid's force and torque on it after each step
        _case("body_63k", 45, 36, 39, 0.02, dt=0.0012, walls="body", cfl=False, spacing=1.015),
        # ragged tank of a viscous fluid without the divergence solver
        _case("ragged_150k", 37, 91, 45, 0.0125, dt=0.00075, divergence=False, viscosity=0.05),
        # the 250 k dam break
        _case("dam_250k", 63, 63, 63, 0.0125, dt=0.00075),
        # the same in the FP64 build
        _case("dam_250k_fp64", 63, 63, 63, 0.0125, dt=0.00075, precision=64),
        # a tall column at a tight tolerance: many solver iterations per step
        _case("column_262k", 32, 256, 32, 0.01, cfl=False, max_error=0.005, spacing=1.0015),
        # a column with the learned warm start
        _case("learned_262k", 64, 64, 64, 0.01, cfl=False, learned=True),
        # the headline workload: a million particles, moving walls, CFL time step
        _case("slosh_1m", 100, 100, 100, 0.01, walls="moving"),
        # a search for a program with its own solver
        _case("search_1m", 125, 80, 100, 0.01, kind="search"),
        # the column collapse
        _case("column_2m", 100, 200, 100, 0.008, dt=0.0005, max_error=0.005),
        # the wave tank
        _case("tank_4m", 400, 100, 100, 0.01, walls="moving"),
    ]


def draw(rng):
    # 1 k to 4 M particles (evenly over the logarithm), tank shapes from a cube to 6 : 1
    kind = rng.choice(["frame"] * 6 + ["search"])
    precision = 64 if kind == "frame" and rng.random() < 0.12 else 32
    walls = rng.choice(["static", "static", "moving", "body"]) if kind == "frame" else "static"
    learned = kind == "frame" and precision == 32 and walls == "static" and rng.random() < 0.2
    top = 4.0e5 if precision == 64 or learned else 1.0e6 if walls == "body" else 3.6e6
    n = math.exp(rng.uniform(math.log(1.0e3), math.log(top)))
    a, b = math.exp(rng.uniform(-0.9, 0.9)), math.exp(rng.uniform(-0.9, 0.9))
    side = (n / (a * b)) ** (1.0 / 3.0)
    nx, ny, nz = max(8, round(side)), max(8, round(side * a)), max(8, round(side * b))
    radius = rng.choice([0.008, 0.01, 0.0125, 0.02, 0.025])
    return _case(None, nx, ny, nz, radius, kind=kind, precision=precision,
                 cfl=rng.random() < 0.6, dt=rng.choice([0.04, 0.05, 0.06]) * radius,
                 divergence=learned or rng.random() < 0.85, viscosity=rng.choice([0.01, 0.01, 0.05]), walls=walls,
                 learned=learned, spacing=1.03 if walls == "body" else rng.choice([1.004, 1.008, 1.015, 1.03]))


# ---- inputs -------------------------------------------------------------------------------------------
def _inputs(case, seed):
    """Fluid positions and velocities (float32), boundary samples, the body's range and the walls' motion."""
    rng = np.random.default_rng(seed)
    d = 2.0 * case["radius"]
    s = case["spacing"] * FLUID_SPACING * d
    cnt = (case["nx"], case["ny"], case["nz"])
    extent = [(c - 1) * s + 2.0 * WALL_GAP * s for c in cnt]
    box = [math.ceil(e / d) * d for e in extent]
    box[1] = math.ceil(1.4 * extent[1] / d) * d  # head room
    axes = [WALL_GAP * s + s * np.arange(c) + (0.5 * (box[a] - extent[a]) if a != 1 else 0.0) for a, c in enumerate(cnt)]
    x = np.stack(np.meshgrid(*axes, indexing="ij"), axis=-1).reshape(-1, 3)
    boundary = box_wall((0.0, 0.0, 0.0), box, d)
    first, count = 0, boundary.shape[0]
    if case["walls"] == "body":  # a box of half a tank's width hanging in the middle of the fluid
        half = np.array([max(1, round(0.15 * c)) * d for c in cnt])
        centre = np.array([0.5 * box[0], 0.5 * extent[1], 0.5 * box[2]])
        body = box_wall(centre - half, centre + half, d)
        first, count = boundary.shape[0], body.shape[0]
        boundary = np.concatenate([boundary, body])
        x = x[np.any(np.abs(x - centre) > half + 0.9 * s, axis=1)]
    x = x.astype(np.float32) + rng.uniform(-0.05 * s, 0.05 * s, x.shape).astype(np.float32)
    # a divergence-free flow along the tank, at rest at the end walls and the floor, and 1 % of noise
    speed = 2.0 * rng.uniform(0.7, 1.0)
    k = math.pi / box[0]
    v = np.zeros_like(x)
    v[:, 0] = speed * np.sin(k * x[:, 0])
    v[:, 1] = -speed * k * x[:, 1] * np.cos(k * x[:, 0])
    v *= min(1.0, box[0] / (math.pi * box[1]))
    v += rng.normal(0.0, 0.01 * speed, v.shape).astype(np.float32)
    drive = (1.0 if case["walls"] == "body" else 0.3) * rng.uniform(0.5, 1.0)  # speed of the moving walls or the body
    return x, v, boundary.astype(np.float32), first, count, drive


def _motion(case, drive):
    """Displacement and velocity, along x, of the moving walls or the body in a frame."""
    return (drive * case["dt"], 0.0, 0.0), (drive, 0.0, 0.0)


def _scene(case, x, boundary):
    cfg = Configuration(timeStepSize=case["dt"], particleRadius=case["radius"], density0=RHO0, viscosity=case["viscosity"],
                        cflMethod=1 if case["cfl"] else 0, cflFactor=0.4, cflMaxTimeStepSize=2.0 * case["dt"],
                        maxIterations=100, maxError=case["max_error"], maxIterationsV=100, maxErrorV=0.1,
                        enableDivergenceSolver=case["divergence"])
    return Scene(config=cfg, fluid=x, boundary=boundary)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a[:0]).dtype, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def prepare(case, seed):
    x, v, boundary, first, count, drive = _inputs(case, seed)
    d = DFSPHCUDA(_scene(case, x, boundary), precision=case["precision"])
    if case["walls"] == "body":
        d.set_param("boundary_forces", 1)
    if case["learned"]:
        d.set_learned_warm_start(True)
    if case["kind"] == "search":
        out = (_pinned(np.zeros((x.shape[0], 2), np.uint32)),)
    else:
        out = (_pinned(np.zeros_like(x)), _pinned(np.zeros_like(v)))
    return dict(case=case, solver=d, x=_pinned(x), v=_pinned(v), out=out, first=first, count=count, drive=drive,
                centre=boundary[first:first + count].astype(np.float64).mean(axis=0))


# ---- one pass -----------------------------------------------------------------------------------------
def run(state):
    case, d = state["case"], state["solver"]
    d.update_fluid(state["x"], state["v"])
    if case["kind"] == "search":
        d.neighbors_search()
        return {"counts": d.field("neighbor_counts", out=state["out"][0])}
    if case["walls"] != "static":
        position, velocity = _motion(case, state["drive"])
        d.move_boundary_rigid(state["first"], state["count"], None, position, velocity, None)
    stats = d.step()
    x, v = d.m_data.readDynamicData(*state["out"])
    got = {"x": x, "v": v, "iterations": int(stats.iterations), "iterations_v": int(stats.iterations_v)}
    if case["walls"] == "body":
        force, torque = d.body_wrench([state["first"]], [state["count"]], [state["centre"] + position])
        got["force"], got["torque"] = force.astype(np.float32), torque.astype(np.float32)
    return got


def _count(case):
    n = case["nx"] * case["ny"] * case["nz"]
    if case["walls"] == "body":
        n -= round(0.3 * case["nx"]) * round(0.3 * case["ny"]) * round(0.3 * case["nz"])
    return n


def work(case):
    """Bytes: the state handed over and read back, and for each step every particle's record and its ~32
    neighbours' indices once per pass over the neighbours (a search, four fixed passes, and the solvers'
    least iterations at two passes each). Flops: ~20 per neighbour and pass, ~8 per search candidate."""
    n, real = _count(case), 8 if case["precision"] == 64 else 4
    io, search = 48 * n, n * (4 * real + 4 * 32)
    if case["kind"] == "search":
        return {"bytes": 12 * n + search + 8 * n, "flops": 8.0 * 216 * n}
    passes = 5 + 4 + (8 if case["divergence"] else 0)
    step = search + passes * n * (12 * real + 4 * 32)
    return {"bytes": io + step, "flops": n * (8.0 * 216 + passes * 20.0 * 32)}


# ---- the same step in 64 bits -------------------------------------------------------------------------
def _pairs(x, y, H, same):
    """Index pairs (i, j) with |x_i - y_j| < H, from a cell grid of y; same: x is y, without i = j."""
    lo = torch.minimum(x.min(0).values, y.min(0).values)
    cx, cy = ((x - lo) / H).floor().long() + 1, ((y - lo) / H).floor().long() + 1
    dim = torch.maximum(cx.max(0).values, cy.max(0).values) + 2
    key = (cy[:, 2] * dim[1] + cy[:, 1]) * dim[0] + cy[:, 0]
    key, order = key.sort()
    ii, jj = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):  # the cells x - 1, x, x + 1 are one run of the sorted keys
            row = ((cx[:, 2] + dz) * dim[1] + cx[:, 1] + dy) * dim[0] + cx[:, 0]
            a, b = torch.searchsorted(key, row - 1), torch.searchsorted(key, row + 1, right=True)
            n = b - a
            i = torch.repeat_interleave(torch.arange(x.shape[0], device=x.device), n)
            j = order[torch.arange(i.numel(), device=x.device) - (n.cumsum(0) - n - a)[i]]
            near = ((x[i] - y[j]) ** 2).sum(1) < H * H
            if same:
                near &= i != j
            ii.append(i[near].int())
            jj.append(j[near].int())
    return torch.cat(ii), torch.cat(jj)


class _Kernel:
    """The cubic spline of support H."""

    def __init__(self, H):
        self.H, self.k, self.l = H, 8.0 / (math.pi * H ** 3), 48.0 / (math.pi * H ** 3)

    def W(self, r):
        q = r.norm(dim=1) / self.H
        return self.k * torch.where(q <= 0.5, 6 * q ** 3 - 6 * q ** 2 + 1, 2 * (1 - q).clamp(min=0) ** 3)

    def grad(self, r):
        rl = r.norm(dim=1)
        q = rl / self.H
        c = self.l * torch.where(q <= 0.5, q * (3 * q - 2), -((1 - q).clamp(min=0) ** 2))
        return r * torch.where(rl > 1e-6, c / (rl * self.H), torch.zeros_like(c))[:, None]


def exact(case, seed):
    """The frame in 64 bits: the DFSPH step as the solver documents it, over explicit pair lists."""
    if case["kind"] == "search" or case["learned"]:
        return None  # whole numbers; a network whose inference is in 16 bits by design
    fx, fv, boundary, first, count, drive = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, v, rest = (torch.from_numpy(a).to(dev).double() for a in (fx, fv, boundary))
    n, r = x.shape[0], case["radius"]
    H = float(np.float32(4.0 * r))
    K = _Kernel(H)
    mass = float(np.float32(0.8 * (2.0 * r) ** 3 * RHO0))
    cfg = _scene(case, fx, boundary).config

    def add(size, index, value):
        return torch.zeros((size, *value.shape[1:]), dtype=torch.float64, device=dev).index_add_(0, index, value)

    bi, bj = _pairs(rest, rest, H, True)
    psi = RHO0 / (K.k + add(rest.shape[0], bi, K.W(rest[bi] - rest[bj])))
    kap, kapv = torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
    h, ratio, it, itv = case["dt"], 1.0, 0, 0
    moved = torch.zeros(rest.shape[0], 1, dtype=torch.float64, device=dev)
    moved[first:first + count] = 1.0
    b, bv = rest, torch.zeros_like(rest)
    if case["walls"] != "static":
        p, pv = (torch.tensor(t, dtype=torch.float64, device=dev) for t in _motion(case, drive))
        b, bv = rest + moved * p, moved * pv
    (i, j), (bi, bj) = _pairs(x, x, H, True), _pairs(x, b, H, False)
    g, gb = mass * K.grad(x[i] - x[j]), psi[bj, None] * K.grad(x[bi] - b[bj])
    w = K.W(x[i] - x[j])
    nf, nb = (torch.bincount(t, minlength=n) for t in (i, bi))
    sparse = torch.where(nf < 20, nf + nb, nf) < 20
    dev_rho = mass * K.k - RHO0 + mass * add(n, i, w) + add(n, bi, psi[bj] * K.W(x[bi] - b[bj]))
    sg = add(n, i, (g * g).sum(1)) + add(n, bi, (gb * gb).sum(1)) + ((add(n, i, g) + add(n, bi, gb)) ** 2).sum(1)
    alpha = -1.0 / h / sg.clamp(min=1e-5)
    force = torch.zeros_like(rest)

    def divergence(v):
        return add(n, i, ((v[i] - v[j]) * g).sum(1)) + add(n, bi, ((v[bi] - bv[bj]) * gb).sum(1))

    def jacobi(k, force):
        ks, kb = k[i] + k[j], k[bi]
        ks, kb = (torch.where(t.abs() > 1e-5, t, torch.zeros_like(t)) for t in (ks, kb))
        force -= add(rest.shape[0], bj, mass * kb[:, None] * gb)
        return add(n, i, ks[:, None] * g) + add(n, bi, kb[:, None] * gb), force

    if case["divergence"]:
        kapv = (kapv * ratio / 2).clamp(min=-0.5)
        source = divergence(v).clamp(min=0)
        source[sparse] = 0
        act = (source > 0).double()
        ks, kb = (kapv[i] + kapv[j]) * act[i], kapv[bi] * act[bi]
        ks, kb = (torch.where(t.abs() > 1e-5, t, torch.zeros_like(t)) for t in (ks, kb))
        v = v + h * (add(n, i, ks[:, None] * g) + add(n, bi, kb[:, None] * gb))
        force -= add(rest.shape[0], bj, mass * kb[:, None] * gb)
        kapv = torch.zeros_like(kapv)
        eta = cfg.maxErrorV * 0.01 * RHO0 / h
        res = divergence(v).clamp(min=0).masked_fill(sparse, 0)
        itv = 0
        while True:
            k = res * alpha
            kapv = kapv + k
            dv, force = jacobi(k, force)
            v = v + h * dv
            res = divergence(v).clamp(min=0).masked_fill(sparse, 0)
            itv += 1
            if not ((res.mean() > eta or itv < 3) and itv < cfg.maxIterationsV):
                break
    acc = -(case["viscosity"] / h) * add(n, i, (mass / (RHO0 + dev_rho[j]) * w)[:, None] * (v[i] - v[j]))
    acc = acc + torch.tensor(cfg.gravitation, dtype=torch.float64, device=dev)
    hf = case["dt"]
    if case["cfl"]:
        top = float(((v + acc * h) ** 2).sum(1).max())
        hf = max(min(cfg.cflFactor * 0.4 * 2.0 * r / math.sqrt(top), cfg.cflMaxTimeStepSize), 1e-4)
    ratio = h / hf
    v = v + h * acc
    dv, force = jacobi((kap * ratio ** 2).clamp(min=-0.5), force)
    v = v + hf * dv
    alpha = alpha / hf
    kap = torch.zeros_like(kap)
    eta = cfg.maxError * 0.01 * RHO0
    it = 0
    while True:
        res = (dev_rho + hf * divergence(v)).clamp(min=0)
        k = res * alpha
        kap = kap + k
        if it and not ((res.mean() > eta or it < 2) and it < cfg.maxIterations):
            break
        dv, force = jacobi(k, force)
        v = v + hf * dv
        it += 1
    x = x + h * v
    h = hf
    got = {"x": x, "v": v, "iterations": None, "iterations_v": None}
    if case["walls"] == "body":
        centre = torch.from_numpy(boundary[first:first + count].astype(np.float64).mean(axis=0)).to(dev) + p
        f, arm = force[first:first + count], b[first:first + count] - centre
        got["force"], got["torque"] = f.sum(0)[None], torch.linalg.cross(arm, f).sum(0)[None]
    return got
