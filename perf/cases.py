"""Performance cases of the lattice-Boltzmann time step, through the Python front end.

A case is a dict of plain values; `listed()` names the ones that are always
measured and `draw(rng)` gives more of the same ranges.  `kind` says how a
program uses the library:

  model     a program keeps one model and advances it by LBMpropagate(ticks),
            reading the fields into its own pinned arrays and the particles
            after each block of ticks (the monitoring or output loop of a run)
  program   the whole short program: modelInit from host fields, addSquirmer,
            LBMpropagate, read the final fields (what a sweep's member costs)
  restart   distributions set from the host, a block of ticks, distributions
            and stress tensor read back (checkpointing and analysis)
  batch     a sweep of unequal 2D replicas advanced together by LBMbatch
  gradient  swimming speed of a squirmer and its derivatives (lbm_adjoint)

Grids are periodic unless `walls` is "channel" (walls on y) or "lid" (walls
on y, the upper one moving).  Coordinates are centred on the origin, as the
reference's particle mass wants it, and swimming speeds and initial flows are
small enough that no particle reaches the periodic boundary however often a
state is advanced.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lbmengine.jl_b200"))

_MODEL = dict(kind="model", lattice="D2Q9", nx=64, ny=64, nz=1, storage="f32", collision="trt", tau=0.8, force=0.0,
              walls="none", particle="none", count=0, radius=0.0, bonds=False, ticks=100)


def _case(name=None, **kw):
    c = dict(_MODEL, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: a 64 x 64 box with one squirmer, watched every ten ticks
        _case("watch_64x64", particle="squirmer", count=1, radius=6.0, ticks=10),
        # the plain 2D method: 256 x 128, BGK, FP64 storage, one squirmer of radius 10
        _case("plain2d_f64", nx=256, ny=128, storage="f64", collision="bgk", particle="squirmer", count=1, radius=10.0),
        # odd sizes, walls, a moving lid and a free bead: none of the 4-node rows of the periodic cases
        _case("lid_201x65", nx=201, ny=65, walls="lid", particle="bead", count=1, radius=7.5, tau=0.9),
        # the plain 3D method, FP32 and FP16 storage
        _case("squirmer128_f32", lattice="D3Q19", nx=128, ny=128, nz=128, tau=0.7, force=2e-8, particle="squirmer",
              count=1, radius=8.0),
        _case("squirmer128_f16", lattice="D3Q19", nx=128, ny=128, nz=128, tau=0.7, force=2e-8, particle="squirmer",
              count=1, radius=8.0, storage="f16"),
        # a suspension: 64 squirmers of radius 6 in 192^3, BF16 storage
        _case("suspension192_bf16", lattice="D3Q19", nx=192, ny=192, nz=192, tau=0.65, particle="squirmer", count=64,
              radius=6.0, storage="bf16"),
        # the largest: 256^3 of decaying flow, no particle
        _case("flow256_f32", lattice="D3Q19", nx=256, ny=256, nz=256, tau=0.6),
        # a ragged 3D channel, D3Q27, two bonded beads (a dumbbell) in a body force
        _case("channel_d3q27", lattice="D3Q27", nx=90, ny=62, nz=46, walls="channel", tau=0.8, force=1e-7,
              particle="bead", count=2, radius=5.0, bonds=True, ticks=50),
        # a parameter sweep: 128 unequal 2D replicas
        _case("sweep_128", kind="batch", count=128, ticks=100),
        # a gradient with binomial checkpointing
        _case("gradient64", kind="gradient", lattice="D3Q19", nx=64, ny=64, nz=64, tau=0.7, force=1e-6,
              particle="squirmer", count=1, radius=8.0, ticks=60),
        # a short program from start to end
        _case("program128", kind="program", lattice="D3Q19", nx=128, ny=128, nz=128, tau=0.7, force=1e-6,
              particle="squirmer", count=1, radius=8.0, ticks=20),
        # restart and analysis of a D3Q15 box
        _case("restart_d3q15", kind="restart", lattice="D3Q15", nx=96, ny=64, nz=80, tau=0.9, collision="bgk",
              force=1e-6, ticks=50),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model2d"] * 4 + ["model3d"] * 5 + ["batch", "gradient", "program", "restart"])
    tau = round(rng.uniform(0.6, 1.0), 3)
    collision = rng.choice(["trt", "trt", "bgk"])
    if kind == "model2d":
        walls = rng.choice(["none", "none", "channel", "lid"])
        c = _case(nx=_log_int(rng, 48, 1500), ny=_log_int(rng, 48, 1000), walls=walls, tau=max(tau, 0.7),
                  collision=collision, storage=rng.choice(["f32", "f32", "f64", "f16"]), ticks=rng.choice([10, 50, 100]))
        if rng.random() < 0.5:  # rows of four nodes, as most programs choose them
            c["nx"] = 4 * max(12, c["nx"] // 4)
        if walls == "lid":  # the wall function is evaluated node by node on the host
            c["nx"], c["ny"] = min(c["nx"], 300), min(c["ny"], 200)
        if walls != "none" and c["storage"] == "f16":
            c["storage"] = "f32"
        if rng.random() < 0.7:
            c.update(particle=rng.choice(["squirmer", "bead"]), count=1, radius=round(rng.uniform(5.0, 10.0), 2))
        return c
    if kind == "batch":
        return _case(kind="batch", count=_log_int(rng, 16, 128), ticks=rng.choice([50, 100, 200]))
    sizes = [_log_int(rng, 24, 200) for _ in range(3)]
    if rng.random() < 0.6:
        sizes[0] = 4 * max(6, sizes[0] // 4)
    if kind == "gradient":
        sizes = [min(64, max(28, s)) for s in sizes]
        return _case(kind="gradient", lattice="D3Q19", nx=sizes[0], ny=sizes[1], nz=sizes[2], tau=max(tau, 0.65),
                     force=1e-6, particle="squirmer", count=1, radius=round(rng.uniform(4.0, 8.0), 2),
                     ticks=rng.choice([30, 50]))
    storage = rng.choice(["f32", "f32", "f32", "f16", "bf16", "f64"])
    lattice = rng.choice(["D3Q19", "D3Q19", "D3Q19", "D3Q15", "D3Q27"])
    c = _case(lattice=lattice, nx=sizes[0], ny=sizes[1], nz=sizes[2], storage=storage, tau=max(tau, 0.65),
              collision=collision, force=rng.choice([0.0, 2e-8]), ticks=rng.choice([10, 50]))
    if kind == "restart":
        c.update(kind="restart", nx=min(sizes[0], 96), ny=min(sizes[1], 96), nz=min(sizes[2], 96))
        return c
    room = min(sizes)
    if room >= 28:
        c.update(particle=rng.choice(["squirmer", "squirmer", "bead"]), radius=round(rng.uniform(4.0, 6.0), 2))
        cells = (sizes[0] // 28) * (sizes[1] // 28) * (sizes[2] // 28)
        c["count"] = rng.randint(1, max(1, min(24, cells)))
    if kind == "program":
        c.update(kind="program", ticks=20, count=min(1, c["count"]))
    elif rng.random() < 0.25 and storage in ("f32", "f64"):
        c["walls"] = "channel"
    return c


# ---- inputs ------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _grid(case):
    dims = 2 if case["lattice"] == "D2Q9" else 3
    return dims, [case["nx"], case["ny"], case["nz"]][:dims]


def _limits(n):
    return (-float(n // 2), float(n - 1 - n // 2))


def _flow(n, seed, amplitude):
    """A smooth random flow: rho [z, y, x] and u [d, z, y, x] (2D: [y, x]), FP64."""
    rng = np.random.default_rng(seed)
    dims, dev = len(n), _device()
    grids = torch.meshgrid(*[torch.arange(k, dtype=torch.float64, device=dev) * (2 * math.pi / k) for k in n[::-1]],
                           indexing="ij")[::-1]
    fields = []
    for comp in range(dims + 1):
        f = torch.zeros(tuple(n[::-1]), dtype=torch.float64, device=dev)
        for _ in range(2):
            k = rng.integers(-2, 3, dims)
            arg = sum(int(k[a]) * grids[a] for a in range(dims)) + float(rng.uniform(0, 2 * math.pi))
            f += float(rng.uniform(0.3, 1.0)) * torch.sin(arg)
        fields.append(f)
    return 1.0 + 1e-5 * fields[0], amplitude * torch.stack(fields[1:])


def _pinned(shape):
    """A column-major float64 array in pinned host memory, as read_fields wants it."""
    t = torch.empty(int(np.prod(shape)), dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy().reshape(shape, order="F")


def _host(t):
    """Device field [.., y, x] as a column-major host array (x first)."""
    shape = tuple(t.shape[::-1])
    out = _pinned(shape)
    torch.from_numpy(out.reshape(-1, order="F")).copy_(t.reshape(-1))
    return out


def _particles(case, n, seed):
    """Keyword sets of the case's particles: well apart, inside the box and off its boundary."""
    rng = np.random.default_rng(seed + 77)
    dims, r = len(n), case["radius"]
    out, centres = [], []
    room = [min(k / 2 - r - 4.0, 1e9) for k in n]
    tries = 0
    while len(centres) < case["count"]:
        tries += 1
        if case["count"] == 1:  # near the centre
            c = rng.uniform(-0.5, 0.5, dims)
        elif case["bonds"]:  # a dumbbell along x
            c = np.array([(-1.0 if not centres else 1.0) * (r + 4.0)] + [0.0] * (dims - 1)) + rng.uniform(-0.5, 0.5, dims)
        else:
            c = np.array([rng.uniform(-room[k], room[k]) for k in range(dims)])
        apart = 2 * r + (6.0 if tries < 5000 else 3.0)
        if all(np.linalg.norm(c - q) >= apart for q in centres):
            centres.append(c)
        elif tries > 20000:
            break
    for c in centres:
        e = rng.standard_normal(dims)
        e /= np.linalg.norm(e)
        kw = dict(radius=r, position=[float(v) for v in c], massDensity=3.0, coupleForces=True, coupleTorques=True)
        if case["particle"] == "squirmer":
            kw.update(swimmingSpeed=1e-4 if dims == 3 else 5e-5, beta=float(rng.uniform(-5, 5)),
                      swimmingDirection=[float(v) for v in e])
        else:
            kw.update(velocity=[float(v) for v in 1e-4 * e])
        out.append(kw)
    return out


def _lid_speed(seed):
    return 1e-3 * (1.0 + 0.1 * (seed % 7))


def _model_keywords(case, seed):
    dims, n = _grid(case)
    kw = dict(dims=dims, velocities=case["lattice"], collisionModel=case["collision"], latticeParameter=1.0,
              relaxationTimeRatio=case["tau"], storage=case["storage"], xlims=_limits(n[0]), ylims=_limits(n[1]))
    if case["collision"] == "trt":
        kw["kineticParameter"] = 3 / 16
    if dims == 3:
        kw["zlims"] = _limits(n[2])
    if case["force"]:
        kw["forceDensity"] = [case["force"]] + [0.0] * (dims - 1)
    if case["walls"] != "none":
        kw["walledDimensions"] = [2]
        if case["walls"] == "lid":
            top, speed = _limits(n[1])[1], _lid_speed(seed)
            kw["movingWalls"] = lambda x, y: [speed, 0.0] if y >= top else [0.0, 0.0]
    return kw


def _amplitude(case):
    return 2e-4


def _build(kw, rho, u, parts, case):
    import lbmengine as lbm
    model = lbm.modelInit(massDensity=rho, fluidVelocity=u, **kw)
    for p in parts:
        (lbm.addSquirmer if case["particle"] == "squirmer" else lbm.addBead)(model, **p)
    if case["bonds"]:
        lbm.addLinearBond(model, 1, 2, equilibriumDisplacement=2 * case["radius"] + 8.0, stiffness=1e-3)
    return model


def _sweep(case, seed):
    """(side, radius, tau, position, direction, beta) of each replica of a batch."""
    rng = np.random.default_rng(seed)
    order = random.Random(12345 + case["count"])  # the grids are the case's, the rest is the seed's
    out = []
    for _ in range(case["count"]):
        side, r = order.choice([64, 96, 128, 192, 256]), float(order.randint(6, 12))
        ang = float(rng.uniform(0, 2 * math.pi))
        pos = [float(v) for v in rng.uniform(-(side / 2 - r - 8), side / 2 - r - 8, 2)]
        out.append((side, r, float(rng.uniform(0.65, 1.0)), pos, [math.cos(ang), math.sin(ang)],
                    float(rng.uniform(-5, 5))))
    return out


def _sweep_particle(rep):
    side, r, tau, pos, e, beta = rep
    return dict(radius=r, position=pos, massDensity=3.0, swimmingSpeed=5e-5, beta=beta, swimmingDirection=e,
                coupleForces=True, coupleTorques=True)


def prepare(case, seed):
    import lbmengine as lbm
    if case["kind"] == "batch":
        reps = _sweep(case, seed)
        batch = lbm.LBMbatch([(dict(dims=2, latticeParameter=1.0, relaxationTimeRatio=tau, collisionModel="trt",
                                    kineticParameter=3 / 16, xlims=_limits(side)), [("squirmer", _sweep_particle(rep))])
                              for rep in reps for side, _, tau, *_ in [rep]])
        batch.autotune()
        cells = sum(s * s for s, *_ in reps)
        rho, u = _pinned((cells,)), _pinned((2 * cells,))
        views, at = [], 0
        for side, *_ in reps:
            k = side * side
            views.append((rho[at:at + k].reshape((side, side), order="F"),
                          u[2 * at:2 * (at + k)].reshape((side, side, 2), order="F")))
            at += k
        return dict(case=case, batch=batch, rho=rho, u=u, views=views)
    dims, n = _grid(case)
    kw, parts = _model_keywords(case, seed), _particles(case, n, seed)
    if case["kind"] == "gradient":
        import lbmengine.adjoint as adj
        return dict(case=case, model=adj.build_swimmer(kw, parts[0]))
    rho0, u0 = _flow(n, seed, _amplitude(case))
    rho0, u0 = _host(rho0), _host(u0)
    if case["kind"] == "program":
        return dict(case=case, kw=kw, parts=parts, rho0=rho0, u0=u0, rho=_pinned(tuple(n)), u=_pinned(tuple(n) + (dims,)))
    if case["kind"] == "restart":
        model = lbm.modelInit(**kw)
        f0 = _equilibrium(case, *[_back(t) for t in (rho0, u0)]).cpu().numpy()
        q = f0.shape[0]
        return dict(case=case, model=model, f0=f0.reshape(-1).reshape(tuple(n) + (q,), order="F"))
    model = _build(kw, rho0, u0, parts, case)
    return dict(case=case, model=model, rho=_pinned(tuple(n)), u=_pinned(tuple(n) + (dims,)))


def _states(model):
    rows = [list(s.position) + list(s.velocity) + list(s.angular_velocity) + list(s.swimming_direction)
            for s in model.particle_states()]
    a = np.array(rows, dtype=np.float64).reshape(-1, 12)
    return dict(position=a[:, 0:3], velocity=a[:, 3:6], spin=a[:, 6:9], direction=a[:, 9:12])


def run(state):
    import lbmengine as lbm
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].step(case["ticks"])
        for m, (r, u) in zip(state["batch"].replicas, state["views"]):
            m.read_fields(r, u)
        return dict(rho=state["rho"], u=state["u"])
    if case["kind"] == "gradient":
        import lbmengine.adjoint as adj
        T = case["ticks"]
        out = adj.swimming_speed_gradient(state["model"], T, (T // 3, T), snapshots=16)
        return dict(value=out.value, grad=out.grad)
    if case["kind"] == "restart":
        model = state["model"]
        model.distributions = state["f0"]
        lbm.LBMpropagate(model, ticks=case["ticks"])
        return dict(f=model.distributions, stress=model.viscous_stress_tensor())
    if case["kind"] == "program":
        model = _build(state["kw"], state["rho0"], state["u0"], state["parts"], case)
    else:
        model = state["model"]
    lbm.LBMpropagate(model, ticks=case["ticks"])
    model.read_fields(state["rho"], state["u"])
    out = dict(rho=state["rho"], u=state["u"])
    if case["count"]:
        out["particles"] = _states(model)
    if case["kind"] == "program":
        model.close()
    return out


_BYTES = {"f32": 4, "f64": 8, "f16": 2, "bf16": 2}


def work(case):
    """Populations read and written once per tick (a tick of a grid beyond the caches moves them), plus the fields
    that cross the host link; arithmetic of the collision (about 8 operations per direction and node)."""
    if case["kind"] == "batch":
        cells = sum(s * s for s, *_ in _sweep(case, 0))
        return dict(bytes=cells * (2.0 * 9 * 4 * case["ticks"] + 24), flops=cells * 9 * 8.0 * case["ticks"])
    dims, n = _grid(case)
    cells, q, size = float(np.prod(n)), int(case["lattice"].split("Q")[1]), _BYTES[case["storage"]]
    ticks = case["ticks"]
    if case["kind"] == "gradient":  # forward once, the adjoint populations (FP64) once backwards
        return dict(bytes=cells * q * ticks * (2.0 * size + size + 16), flops=cells * q * ticks * 40.0)
    ends = {"model": 8.0 * (1 + dims), "program": 16.0 * (1 + dims), "restart": 16.0 * q + 8.0 * dims * dims}[case["kind"]]
    return dict(bytes=cells * (2.0 * q * size * ticks + ends), flops=cells * q * 8.0 * ticks)


# ---- the same in 64 bits, plain torch ------------------------------------------

def _vectors(lattice):
    axis = lambda d: [tuple(s if a == b else 0 for b in range(d)) for a in range(d) for s in (-1, 1)]  # noqa: E731
    if lattice == "D2Q9":
        c = [(0, 0)] + axis(2) + [(-1, -1), (1, -1), (-1, 1), (1, 1)]
        w = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
        return c, w
    edges = [(0, a, b) for b in (-1, 1) for a in (-1, 1)] + [(a, 0, b) for b in (-1, 1) for a in (-1, 1)] + \
        [(a, b, 0) for b in (-1, 1) for a in (-1, 1)]
    corners = [(a, b, d) for d in (-1, 1) for b in (-1, 1) for a in (-1, 1)]
    if lattice == "D3Q15":
        return [(0, 0, 0)] + axis(3) + corners, [2 / 9] + [1 / 9] * 6 + [1 / 72] * 8
    if lattice == "D3Q19":
        return [(0, 0, 0)] + axis(3) + edges, [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
    return [(0, 0, 0)] + axis(3) + edges + corners, [8 / 27] + [2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8


def _back(a):
    """A column-major host array as a device tensor with x last."""
    return torch.from_numpy(np.ascontiguousarray(a.T)).to(_device())


def _equilibrium(case, rho, u):
    c, w = _vectors(case["lattice"])
    uu = (u * u).sum(0)
    f = torch.empty((len(c),) + tuple(rho.shape), dtype=torch.float64, device=rho.device)
    for i, (ci, wi) in enumerate(zip(c, w)):
        cu = sum(ci[k] * u[k] for k in range(len(ci)))
        f[i] = wi * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu)
    return f


class _Body:
    """One particle of the FP64 reference (state as 0-d / 1-d tensors, so that gradients flow)."""

    def __init__(self, kw, dims, coords, dev, B1=None, B2=None):
        t = lambda v: torch.tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
        self.r, self.dims = kw["radius"], dims
        self.R, self.v = t(kw["position"]), t(kw.get("velocity", [0.0] * dims))
        self.w = t([0.0] * (1 if dims == 2 else 3))
        self.squirmer = "swimmingSpeed" in kw
        self.e = t(kw.get("swimmingDirection", [1.0] + [0.0] * (dims - 1)))
        self.B1 = t(1.5 * kw["swimmingSpeed"]) if self.squirmer and B1 is None else B1
        self.B2 = self.B1 * kw["beta"] if self.squirmer and B2 is None else B2
        d2 = 0.0
        for a in range(dims):  # the reference counts the nodes of a sphere about the origin
            shape = [1] * dims
            shape[dims - 1 - a] = -1
            d2 = d2 + (coords[a] ** 2).reshape(shape)
        self.m = kw["massDensity"] * float((d2 < self.r ** 2).sum())
        self.I = (0.5 if dims == 2 else 0.4) * self.m * self.r ** 2
        self.key = None
        self.snapshot()

    def snapshot(self):
        self.s = (self.R, self.v, self.w, self.e)

    def slip(self, X):
        """Node velocity at points X [n, d] from the last snapshot."""
        R, v, w, e = self.s
        xr = X - R
        if self.dims == 2:
            up = v + torch.stack([-w[0] * xr[:, 1], w[0] * xr[:, 0]], 1)
        else:
            up = v + torch.linalg.cross(w.expand_as(xr), xr)
        if self.squirmer:
            ur = xr / torch.sqrt((xr * xr).sum(1, keepdim=True))
            ed = (ur * e).sum(1, keepdim=True)
            up = up + (self.B1 + self.B2 * ed) * (ed * ur - e)
        return up

    def update(self, F, T):
        self.v = self.v + F / self.m
        self.R = self.R + self.v
        self.w = self.w + T / self.I
        if self.squirmer:
            th = torch.sqrt((self.w * self.w).sum())
            if float(th) != 0.0:
                k, ct, st = self.w / th, torch.cos(th), torch.sin(th)
                if self.dims == 2:
                    e = torch.stack([self.e[0] * ct - k[0] * self.e[1] * st, self.e[1] * ct + k[0] * self.e[0] * st])
                else:
                    e = self.e * ct + torch.linalg.cross(k, self.e) * st + k * (k @ self.e) * (1 - ct)
                self.e = e / torch.sqrt((e * e).sum())
        self.snapshot()


class _Reference:
    """The tick of the reference (collide, stream, walls, Ladd links, particles) in FP64 on whole-field tensors."""

    def __init__(self, case, n, f, parts, seed, theta=None):
        dev = f.device
        self.case, self.n, self.dims, self.f, self.dev = case, n, len(n), f, dev
        self.c, self.w = _vectors(case["lattice"])
        self.opp = [self.c.index(tuple(-v for v in ci)) for ci in self.c]
        self.coords = [torch.arange(k, dtype=torch.float64, device=dev) + _limits(k)[0] for k in n]
        th = theta or {}
        self.tau = th.get("tau", case["tau"])
        self.taum = (3 / 16) / (self.tau - 0.5) + 0.5
        self.F = th.get("F", torch.tensor([case["force"]] + [0.0] * (self.dims - 1), dtype=torch.float64, device=dev))
        self.guo = bool(case["force"])
        self.wall = None
        if case["walls"] != "none":
            self.wall = torch.zeros(tuple(n[::-1]), dtype=torch.bool, device=dev)
            y = self.wall.movedim(-2, 0)
            y[0], y[-1] = True, True
            self.lid = _lid_speed(seed) if case["walls"] == "lid" else 0.0
        self.bodies = [_Body(p, self.dims, self.coords, dev, th.get("B1"), th.get("B2")) for p in parts]

    def moments(self):
        rho = self.f.sum(0)
        j = [sum(ci[k] * self.f[i] for i, ci in enumerate(self.c) if ci[k]) for k in range(self.dims)]
        if self.guo:
            j = [jk + 0.5 * Fk for jk, Fk in zip(j, self.F)]
        if self.wall is None:
            return rho, [jk / rho for jk in j]
        safe = torch.where(self.wall, torch.ones_like(rho), rho)
        return rho, [torch.where(self.wall, torch.zeros_like(jk), jk / safe) for jk in j]

    def collide(self):
        rho, u = self.moments()
        f, trt = self.f, self.case["collision"] == "trt"
        uu = sum(uk * uk for uk in u)
        uF = sum(uk * Fk for uk, Fk in zip(u, self.F)) if self.guo else None
        out = [None] * len(self.c)
        for i, ci in enumerate(self.c):
            ib = self.opp[i]
            if ib < i:
                continue
            w = self.w[i]
            cu = sum((u[k] if ci[k] > 0 else -u[k]) for k in range(self.dims) if ci[k]) if any(ci) else 0.0 * uu
            ev, od = w * rho * (1 + 4.5 * cu * cu - 1.5 * uu), w * rho * 3 * cu
            gp = gm = 0.0
            if self.guo:
                cF = sum(ci[k] * self.F[k] for k in range(self.dims))
                gp, gm = w * (-3 * uF + 9 * cu * cF), w * 3 * cF
            if trt:
                fp, fm = 0.5 * (f[i] + f[ib]), 0.5 * (f[i] - f[ib])
                dp = -(fp - ev) / self.tau + (1 - 0.5 / self.tau) * gp
                dm = -(fm - od) / self.taum + (1 - 0.5 / self.taum) * gm
                out[i] = f[i] + dp + dm
                if ib != i:
                    out[ib] = f[ib] + dp - dm
            else:
                k = 1 - 0.5 / self.tau
                out[i] = f[i] - (f[i] - ev - od) / self.tau + k * (gp + gm)
                if ib != i:
                    out[ib] = f[ib] - (f[ib] - ev + od) / self.tau + k * (gp - gm)
        return rho, out

    def links(self, b):
        """Boundary links of a body: direction index, flat fluid cell, link rows; kept until the mask changes."""
        dims, n = self.dims, self.n
        R = [float(v) for v in b.R]
        lo = [math.floor(R[k] - b.r - _limits(n[k])[0]) - 3 for k in range(dims)]
        hi = [math.ceil(R[k] + b.r - _limits(n[k])[0]) + 3 for k in range(dims)]
        ax = [torch.arange(lo[k], hi[k] + 1, device=self.dev) for k in range(dims)]
        inside = [(a >= 0) & (a < n[k]) for k, a in enumerate(ax)]
        d2, ok = 0.0, True
        for k in range(dims):
            shape = [1] * dims
            shape[dims - 1 - k] = -1
            d2 = d2 + ((ax[k].double() + _limits(n[k])[0] - R[k]) ** 2).reshape(shape)
            ok = inside[k].reshape(shape) & ok
        S = (d2 < b.r ** 2) & ok
        if b.key is not None and b.key[0] == lo and torch.equal(b.key[1], S):
            return b.links
        dims_t = tuple(range(dims))
        L = torch.stack([torch.roll(S, tuple(ci[::-1]), dims_t) & ~S for ci in self.c])
        at = L.nonzero()
        j, pos = at[:, 0], [at[:, dims - k] for k in range(dims)]  # pos[k]: local index along axis k
        cj = torch.tensor(self.c, device=self.dev)[j]
        gl = [(ax[k][pos[k]] % n[k]) for k in range(dims)]
        sr = [((ax[k][pos[k]] - cj[:, k]) % n[k]) for k in range(dims)]
        cell, src = gl[-1], sr[-1]
        for k in range(dims - 2, -1, -1):
            cell, src = cell * n[k] + gl[k], src * n[k] + sr[k]
        X = torch.stack([self.coords[k][gl[k]] for k in range(dims)], 1)
        Y = torch.stack([self.coords[k][sr[k]] for k in range(dims)], 1)
        b.key = (lo, S)
        b.links = (j, cell, X, Y, cj.double(), torch.tensor(self.opp, device=self.dev)[j],
                   torch.tensor(self.w, dtype=torch.float64, device=self.dev)[j])
        return b.links

    def tick(self):
        rho, fs = self.collide()
        dims_t = tuple(range(self.dims))
        new = []
        for i, ci in enumerate(self.c):
            g = torch.roll(fs[i], tuple(ci[::-1]), dims_t) if any(ci) else fs[i]
            if self.wall is not None:
                from_wall = torch.roll(self.wall, tuple(ci[::-1]), dims_t)
                back = fs[self.opp[i]]
                if self.lid:  # the moving wall's term, at nodes whose source is the upper wall
                    top = torch.zeros_like(self.wall)
                    top.movedim(-2, 0)[-1] = True
                    top = torch.roll(top, tuple(ci[::-1]), dims_t)
                    back = back + torch.where(top, 6 * self.w[i] * rho * (ci[0] * self.lid), torch.zeros_like(rho))
                g = torch.where(from_wall, back, g)
                g = torch.where(self.wall, torch.zeros_like(g), g)
            new.append(g)
        f = torch.stack(new)
        del new
        shape, cells = f.shape, rho.numel()
        force = []
        if self.bodies:
            flat = f.reshape(-1)
            star = torch.stack(fs).reshape(-1)
            del fs
            rows, vals = [], []
            for b in self.bodies:
                j, cell, X, Y, cj, opp, w = self.links(b)
                out = star[opp * cells + cell]
                val = out + 6 * w * rho.reshape(-1)[cell] * (cj * b.slip(Y)).sum(1)
                s = out + val
                rows.append(j * cells + cell)
                vals.append(val)
                F = -(s[:, None] * cj).sum(0)
                arm = X - b.R
                if self.dims == 2:
                    T = -(s * (arm[:, 0] * cj[:, 1] - arm[:, 1] * cj[:, 0])).sum().reshape(1)
                else:
                    T = -(s[:, None] * torch.linalg.cross(arm, cj)).sum(0)
                force.append([F, T])
            flat = flat.index_put((torch.cat(rows),), torch.cat(vals))
            f = flat.reshape(shape)
        if self.case["bonds"]:
            a, b = self.bodies[:2]
            d = b.R - a.R
            dist = torch.sqrt((d * d).sum())
            pull = 1e-3 * (dist - (2 * self.case["radius"] + 8.0)) * d / dist
            force[0][0] = force[0][0] + pull
            force[1][0] = force[1][0] - pull
        for b, (F, T) in zip(self.bodies, force):
            b.update(F, T)
        self.f = f


def _fields_out(ref):
    rho, u = ref.moments()
    rho, u = rho.cpu().numpy(), torch.stack(u).cpu().numpy()
    return rho.transpose(), u.transpose(tuple(range(u.ndim - 1, 0, -1)) + (0,))


def _initial(case, n, seed):
    """Initial populations as modelInit makes them from the case's flow: zero on walls, the Guo half force taken off."""
    rho, u = _flow(n, seed, _amplitude(case))
    wall = None
    if case["walls"] != "none":
        wall = torch.zeros_like(rho, dtype=torch.bool)
        y = wall.movedim(-2, 0)
        y[0], y[-1] = True, True
        rho, u = torch.where(wall, 0.0, rho), torch.where(wall, 0.0, u)
    if case["force"]:
        shift = 0.5 * case["force"] / rho if wall is None else torch.where(wall, 0.0, 0.5 * case["force"] / torch.where(wall, 1.0, rho))
        u = torch.cat([(u[0] - shift)[None], u[1:]])
    return _equilibrium(case, rho, u)


def exact(case, seed):
    dev = _device()
    if case["kind"] == "batch":
        if case["ticks"] * case["count"] > 13000:  # over about 20 seconds
            return None
        rhos, us = [], []
        for side, r, tau, pos, e, beta in _sweep(case, seed):
            c = _case(nx=side, ny=side, tau=tau)
            f = _equilibrium(c, torch.ones((side, side), dtype=torch.float64, device=dev),
                             torch.zeros((2, side, side), dtype=torch.float64, device=dev))
            ref = _Reference(c, [side, side], f, [_sweep_particle((side, r, tau, pos, e, beta))], seed)
            for _ in range(case["ticks"]):
                ref.tick()
            a, b = _fields_out(ref)
            rhos.append(a.ravel(order="F"))
            us.append(b.ravel(order="F"))
        return dict(rho=np.concatenate(rhos), u=np.concatenate(us))
    dims, n = _grid(case)
    parts = _particles(case, n, seed)
    if case["kind"] == "gradient":
        leaf = lambda v: torch.tensor(v, dtype=torch.float64, device=dev, requires_grad=True)  # noqa: E731
        B1 = leaf(1.5 * parts[0]["swimmingSpeed"])
        B2 = leaf(1.5 * parts[0]["swimmingSpeed"] * parts[0]["beta"])
        tau, F = leaf(case["tau"]), leaf([case["force"]] + [0.0] * (dims - 1))
        shape = tuple(n[::-1])
        one = torch.ones(shape, dtype=torch.float64, device=dev)
        c, w = _vectors(case["lattice"])
        u0 = [-0.5 * F[k] for k in range(dims)]
        uu = sum(v * v for v in u0)
        f = torch.stack([w[i] * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu) * one for i, ci in enumerate(c)
                         for cu in [sum(ci[k] * u0[k] for k in range(dims))]])
        ref = _Reference(case, n, f, parts, seed, dict(B1=B1, B2=B2, tau=tau, F=F))
        e0, T, J = ref.bodies[0].e, case["ticks"], 0.0
        for t in range(1, T + 1):
            ref.tick()
            if t >= T // 3:
                J = J + (ref.bodies[0].v * e0).sum()
        J = J / (T - T // 3 + 1)
        g = torch.autograd.grad(J, [B1, B2, tau, F])
        return dict(value=float(J), grad=dict(B1=float(g[0]), B2=float(g[1]), tau=float(g[2]), Fx=float(g[3][0]),
                                              Fy=float(g[3][1]), Fz=float(g[3][2]) if dims == 3 else 0.0))
    if case["kind"] == "restart":
        f = _equilibrium(case, *_flow(n, seed, _amplitude(case)))
        ref = _Reference(case, n, f, [], seed)
        for _ in range(case["ticks"]):
            ref.tick()
        rho, u = ref.moments()
        neq = ref.f - _equilibrium(case, rho, torch.stack(u))
        d = [[-(1 - 0.5 / case["tau"]) * sum(ci[a] * ci[b] * neq[i] for i, ci in enumerate(ref.c) if ci[a] * ci[b])
              for b in range(dims)] for a in range(dims)]
        stress = np.stack([np.stack([d[a][b].cpu().numpy().transpose() for b in range(dims)], -1) for a in range(dims)], -2)
        fout = ref.f.cpu().numpy()
        return dict(f=fout.transpose(tuple(range(dims, 0, -1)) + (0,)), stress=stress)
    ref = _Reference(case, n, _initial(case, n, seed), parts, seed)
    for _ in range(case["ticks"]):
        ref.tick()
    rho, u = _fields_out(ref)
    out = dict(rho=rho, u=u)
    if case["count"]:
        pad = lambda t: list(t.tolist()) + [0.0] * (3 - t.numel())  # noqa: E731
        cols = [[pad(getattr(b, k)) for b in ref.bodies] for k in ("R", "v", "w", "e")]
        if case["particle"] != "squirmer":
            cols[3] = [[0.0] * 3 for _ in ref.bodies]
        spin = np.array(cols[2]) if case["storage"] in ("f32", "f64") else None
        out["particles"] = dict(position=np.array(cols[0]), velocity=np.array(cols[1]), spin=spin,
                                direction=np.array(cols[3]))
    return out
