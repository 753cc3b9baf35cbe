"""The work that programs hand to this framework, as measurable cases.

A case names a workload by its sizes. ``prepare`` builds the scenario and the
simulation handle (or network) a program keeps, ``run`` is one pass through
the public entry points, ``work`` the bytes and operations a pass cannot do
without, and ``exact`` the same pass in 64-bit arithmetic, in plain torch.

A pass of a simulation is one output interval of a run: a few steps and the
read of the particle state at its end. Passes on one handle continue the
simulation, as a program's do.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import ultraballpit_b200
from ultraballpit_b200 import domain
from ultraballpit_b200.closure import ClosureNet
from ultraballpit_b200.kernel import BOUNDARY_SDF, CELL_ORDER_MORTON, CELL_ORDER_ROWS, CudaBatch, CudaKernel

FIELDS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "density", "pressure", "mass")
WEIGHTS = os.path.join(os.path.dirname(ultraballpit_b200.__file__), "data", "closure_weights.npy")

# listed neighbours per particle inside the fluid (h = 1.3 dx, support 2h), and operations per pair of the
# XSPH sum, the density and density-diffusion sums, and the pressure and viscosity sums
NEIGHBOURS, PAIR_FLOPS = 78, 25 + 40 + 60
# particle state of one step: position, mass, velocity, acceleration, density, pressure in; the same out
STATE_BYTES = 48


def listed():
    dam = dict(bx=0.1, by=0.2, bz=0.1, lx=0.4, ly=0.2, lz=0.1, sphere=False, morton=False)
    return [
        # the smallest simulations, driven by the host: an orchestrator asks for the time step, steps and checks
        # the error metrics each step (2,000 particles)
        dict(name="dam_break_10mm_host_loop", kind="host", dx=0.01, steps=10, **dam),
        # an ordinary small simulation on the device time step (31,250 particles)
        dict(name="dam_break_4mm", kind="auto", dx=0.004, steps=20, **dam),
        # a box of odd sizes, the other storage order (about 90,000 particles)
        dict(name="odd_box_morton", kind="auto", dx=0.0029, steps=20, bx=0.1213, by=0.1471, bz=0.1227, lx=0.3117,
             ly=0.1471, lz=0.1639, sphere=False, morton=True),
        # the server's loop: optimistic time steps and a viewer frame per interval (250,000 particles)
        dict(name="dam_break_2mm_optimistic", kind="optimistic", dx=0.002, steps=10, **dam),
        # the largest single simulation, with an obstacle whose forces are read (2,000,000 particles)
        dict(name="dam_break_1mm_sphere", kind="auto", dx=0.001, steps=10, **dict(dam, sphere=True)),
        # many uneven simulations in one batch, a time step each (16 boxes of 2,000 to 200,000 particles)
        dict(name="boxes_2mm_batch", kind="batch", boxes=16, lo=2000, hi=200000, dx=0.002, boxes_seed=7, steps=10),
        # the homogenised wall mode around a sphere (about 68,000 particles)
        dict(name="tank_sdf_walls", kind="sdf", dx=0.0025, lx=0.12, ly=0.1, lz=0.12, fill=0.0925, radius=0.02,
             steps=20),
        # the learned near-wall closure evaluated in the step, in a moving tank (about 24,000 particles)
        dict(name="tank_closure", kind="closure", dx=0.004, lx=0.1, ly=0.1, lz=0.2, fill=0.16, radius=0.02, steps=20),
        # training that closure: one epoch of mini-batches over captured samples
        dict(name="closure_train", kind="train", n=50000, batch=1024),
    ]


def draw(rng):
    kind = rng.choice(("host", "auto", "auto", "auto", "optimistic", "batch", "sdf", "closure", "train"))
    if kind == "train":
        return dict(kind=kind, n=rng.randrange(5000, 80000), batch=rng.choice((256, 500, 1024, 4096)))
    if kind == "batch":
        boxes = rng.randrange(3, 25)
        return dict(kind=kind, boxes=boxes, lo=1000, hi=int(math.exp(rng.uniform(math.log(5e3), math.log(2e5)))),
                    dx=round(rng.uniform(0.0015, 0.004), 5), boxes_seed=rng.randrange(1 << 20), steps=10)
    steps = rng.choice((5, 10, 20))
    if kind in ("sdf", "closure"):
        lx, ly, lz = (round(rng.uniform(0.09, 0.16), 4) for _ in range(3))
        fill = round(lz * rng.uniform(0.6, 0.85), 4)
        n = math.exp(rng.uniform(math.log(4e3), math.log(4e5)))
        return dict(kind=kind, dx=round((lx * ly * fill / n) ** (1 / 3), 6), lx=lx, ly=ly, lz=lz, fill=fill,
                    radius=round(rng.uniform(0.012, 0.02), 4), steps=steps)
    bx, by, bz = (round(rng.uniform(0.06, 0.2), 4) for _ in range(3))
    n = math.exp(rng.uniform(math.log(600), math.log(3e4 if kind == "host" else 1e6)))
    return dict(kind=kind, dx=round((bx * by * bz / n) ** (1 / 3), 6), steps=steps, bx=bx, by=by, bz=bz,
                lx=round(bx * rng.uniform(1.3, 4.0), 4), ly=by, lz=round(bz * rng.uniform(1.0, 1.5), 4), sphere=False,
                morton=rng.random() < 0.15)


def spacings(case, key):
    """A length of the case in whole particle spacings."""
    return max(1, round(case[key] / case["dx"]))


def scenarios(case, seed):
    """The scenarios of a simulation case: their sizes from the case, the particles' jitter from the seed."""
    if case["kind"] == "batch":
        scs = domain.batch_boxes(case["boxes"], seed=case["boxes_seed"], dx=case["dx"], lo=case["lo"], hi=case["hi"],
                                 draw="loguniform")
        rng = np.random.default_rng(seed)
        for sc in scs:  # batch_boxes draws sizes and jitter together: the jitter of this seed on top
            for a in (sc.particles.x, sc.particles.y, sc.particles.z):
                a += rng.uniform(-0.01 * case["dx"], 0.01 * case["dx"], a.shape).astype(np.float32)
        return scs
    if case["kind"] in ("sdf", "closure"):
        dx = case["dx"]
        # whole spacings, so that the lattice meets every wall half a spacing from it
        lx, ly, lz, fill = (spacings(case, k) * dx * (1 - 1e-6) for k in ("lx", "ly", "lz", "fill"))
        sc = domain.tank_with_sphere(dx, domain_max=(lx, ly, lz), center=(0.5 * lx, 0.45 * ly, 0.5 * fill),
                                     radius=case["radius"], fill_height=fill, seed=seed, hydrostatic=True,
                                     geometry="lattice", velocity=(0.2, 0.0, 0.0))
        return [sc]
    dx = case["dx"]
    return [domain.dam_break(dx, seed=seed, sphere=case["sphere"],
                             block=tuple((spacings(case, k) - 0.25) * dx for k in ("bx", "by", "bz")),
                             domain_max=tuple(spacings(case, k) * dx for k in ("lx", "ly", "lz")), with_sdf=False)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, t = samples(case["n"], seed)
        return dict(case=case, net=ClosureNet(seed=seed), x=x, t=t, seed=seed)
    scs = scenarios(case, seed)
    sc = scs[0]
    if kind == "batch":
        k = CudaBatch(scs)
    elif kind == "sdf":
        k = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta, boundary_mode=BOUNDARY_SDF,
                       sdf=sc.obstacle_sdf)
        k.set_geometry_sdf(sc.obstacle_sdf)
    else:
        k = CudaKernel(*sc.kernel_args(), alpha=sc.alpha, beta=sc.beta,
                       cell_order=CELL_ORDER_MORTON if case.get("morton") else CELL_ORDER_ROWS)
        if kind == "closure":
            k.set_feature_sdf(sc.sdf)
            k.set_closure(2, np.load(WEIGHTS))
    ex = sc.extras
    return dict(case=case, k=k, frame=0, nb=len(sc.boundary), body=ex.get("n_geometry_boundary", 0))


def samples(n, seed):
    """Closure samples: features of the ranges that near-wall particles have, targets with the spread of the paired
    runs' differences."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.0, 1.0, (n, 16)).astype(np.float32)
    x[:, 0] = 2.0 * np.abs(x[:, 0])
    x[:, 15] = 1.0
    w = rng.normal(0.0, 0.5, (16, 4))
    t = (np.tanh(x @ w) + rng.normal(0.0, 0.3, (n, 4))).astype(np.float32)
    return x, t


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        net = state["net"]
        losses = net.train(state["x"], state["t"], batch=case["batch"], epochs=1, seed=state["seed"])
        return dict(losses=losses, params=net.params())
    k = state["k"]
    out = {}
    if kind == "host":
        dts, metrics = [], []
        for _ in range(case["steps"]):
            dts.append(k.compute_timestep())
            k.step(dts[-1])
            metrics.append(k.error_metrics())
        out["dt"] = np.array(dts, np.float32)
        out["variation"] = np.array([m.max_density_variation for m in metrics], np.float32)
        out["energy"] = np.array([m.energy_conservation for m in metrics], np.float32)
    elif kind == "optimistic":
        stats = k.run_optimistic(case["steps"])
        out["dt"] = stats["last_dt"]
        out["frame"] = np.frombuffer(k.pack_frame(10000, state["frame"], 0.0), np.uint8)
    elif kind == "batch":
        k.step_auto(case["steps"], want_dt=False)
        out["dt"] = k.timesteps()
    else:
        out["dt"] = k.step_auto(case["steps"])
    if kind == "sdf":
        f = k.surface_forces()
        out["force"], out["moment"] = f["force"], f["moment"]
    if case.get("sphere"):
        f = k.body_force(state["nb"] - state["body"], state["body"])
        out["force"] = f["pressure_force"] + f["repulsion_force"]
    p = k.particles()
    out.update({f: getattr(p, f) for f in FIELDS})
    return out


def count(case):
    """Fluid particles of a simulation case."""
    if case["kind"] in ("sdf", "closure"):
        return (spacings(case, "lx") * spacings(case, "ly") * spacings(case, "fill")
                - round(4.19 * (case["radius"] / case["dx"]) ** 3))
    if case["kind"] == "batch":  # log-uniform counts in [lo, hi]
        return int(case["boxes"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]))
    return spacings(case, "bx") * spacings(case, "by") * spacings(case, "bz")


def work(case):
    if case["kind"] == "train":
        # samples in, parameters out; forward and both backward products of 16 x 64 + 64 x 64 + 64 x 4 weights
        return dict(bytes=case["n"] * 80 + 2 * 4 * 5508, flops=case["n"] * 6 * (16 * 64 + 64 * 64 + 64 * 4))
    n = count(case)
    return dict(bytes=n * case["steps"] * 2 * STATE_BYTES, flops=n * case["steps"] * NEIGHBOURS * PAIR_FLOPS)


# ---------------------------------------------------------------------------
# the same pass in 64-bit arithmetic
# ---------------------------------------------------------------------------

def exact(case, seed):
    if case["kind"] not in ("host", "auto", "optimistic", "batch") or count(case) * case["steps"] > 8_000_000:
        return None
    runs = [Sim64(sc) for sc in scenarios(case, seed)]
    out = {}
    if case["kind"] == "host":
        dts, var = [], []
        for _ in range(case["steps"]):
            dts.append(runs[0].timestep())
            runs[0].step(dts[-1])
            var.append(runs[0].variation())
        out = dict(dt=np.array(dts), variation=np.array(var), energy=None)
    elif case["kind"] == "optimistic":
        out = dict(dt=None, frame=None)
        cooldown = 0
        for _ in range(case["steps"]):
            dt, s = runs[0].timestep(), runs[0]
            if cooldown:
                cooldown -= 1
                s.step(dt)
                continue
            saved = (s.x, s.v, s.a, s.rho, s.p)
            s.step(1.5 * dt)
            if s.variation() > 0.03:
                s.x, s.v, s.a, s.rho, s.p = saved
                s.step(dt)
                cooldown = 10
    else:
        dts = []
        for s in runs:
            for _ in range(case["steps"]):
                dt = s.timestep()
                s.step(dt)
            dts.append(s.timestep() if case["kind"] == "batch" else dt)
        out = dict(dt=np.array(dts) if case["kind"] == "batch" else dts[0])
    for i, f in enumerate(("x", "y", "z")):
        out[f] = np.concatenate([s.x[:, i].cpu().numpy() for s in runs])
        out["v" + f] = np.concatenate([s.v[:, i].cpu().numpy() for s in runs])
        out["a" + f] = np.concatenate([s.a[:, i].cpu().numpy() for s in runs])
    out["density"] = np.concatenate([s.rho.cpu().numpy() for s in runs])
    out["pressure"] = np.concatenate([s.p.cpu().numpy() for s in runs])
    out["mass"] = np.concatenate([s.m.cpu().numpy() for s in runs])
    return out


def pairs64(a, b, radius, same):
    """Indices (i, j) of the points of a and b closer than radius (i != j where both are the same set)."""
    lo = b.min(0).values
    cells = ((b - lo) / radius).floor().long()
    dims = cells.max(0).values + 3  # a border of empty cells on both sides
    lin = lambda c: ((c[..., 0] + 1) * dims[1] + c[..., 1] + 1) * dims[2] + c[..., 2] + 1  # noqa: E731
    key, order = lin(cells).sort()
    total = int(dims.prod())
    counts = torch.bincount(key, minlength=total)
    start = counts.cumsum(0) - counts
    most = int(counts.max())
    off = torch.stack(torch.meshgrid(*[torch.arange(-1, 2, device=a.device)] * 3, indexing="ij"), -1).reshape(-1, 3)
    slot = torch.arange(most, device=a.device)
    ii, jj = [], []
    chunk = max(1, 40_000_000 // (27 * most))
    for at in range(0, len(a), chunk):
        q = a[at:at + chunk]
        c = ((q - lo) / radius).floor().long()[:, None, :] + off
        inside = ((c >= -1) & (c <= dims - 2)).all(-1)
        k = lin(torch.where(inside[..., None], c, torch.zeros_like(c)))
        ok = inside[..., None] & (slot < counts[k][..., None])
        j = order[torch.where(ok, start[k][..., None] + slot, torch.zeros_like(slot))]
        d2 = sum((q[:, None, None, x] - b[j, x]) ** 2 for x in range(3))
        ok &= d2 < radius * radius
        i = torch.arange(at, at + len(q), device=a.device)[:, None, None].expand_as(j)
        if same:
            ok &= i != j
        ii.append(i[ok])
        jj.append(j[ok])
    return torch.cat(ii), torch.cat(jj)


class Sim64:
    """One simulation of water particles between wall particles: weakly compressible SPH with the Wendland C2 kernel,
    density diffusion, wall pressure by extrapolation, Monaghan viscosity, XSPH and kick-drift-kick."""

    def __init__(self, sc):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda *v: torch.from_numpy(np.stack(v, -1).astype(np.float64)).to(dev)  # noqa: E731
        p, b = sc.particles, sc.boundary
        self.x, self.v, self.a = t(p.x, p.y, p.z), t(p.vx, p.vy, p.vz), t(p.ax, p.ay, p.az)
        self.rho, self.p, self.m = t(p.density)[:, 0], t(p.pressure)[:, 0], t(p.mass)[:, 0]
        self.bx, self.bm = t(b.x, b.y, b.z), t(b.mass)[:, 0]
        f = lambda v: float(np.float32(v))  # noqa: E731
        self.h, self.c, self.cfl = f(sc.h), f(sc.speed_of_sound), f(sc.cfl_number)
        self.alpha, self.beta = f(sc.alpha), f(sc.beta)
        self.g = t(np.float32(sc.gravity[0]), np.float32(sc.gravity[1]), np.float32(sc.gravity[2]))
        self.lo, self.hi = t(*map(np.float32, sc.domain_min)), t(*map(np.float32, sc.domain_max))
        self.first = True
        self.ff = None

    def kernel(self, r):
        q = r / self.h
        return 21 / (16 * math.pi) / self.h ** 3 * (1 - 0.5 * q).clamp(min=0) ** 4 * (1 + 2 * q)

    def slope(self, d, r):
        """The kernel's gradient along d = x_i - x_j."""
        q = r / self.h
        dw = 21 / (16 * math.pi) / self.h ** 4 * (-5 * q) * (1 - 0.5 * q).clamp(min=0) ** 3
        return (dw / r)[:, None] * d

    def total(self, i, values):
        return torch.zeros((len(self.x),) + values.shape[1:], dtype=values.dtype, device=values.device).index_add_(
            0, i, values)

    def compute_forces(self, dt):
        h, rho0 = self.h, 1000.0
        self.ff = i, j = pairs64(self.x, self.x, 2 * h, True)
        wi, wj = pairs64(self.x, self.bx, 2 * h, False)
        d = self.x[i] - self.x[j]
        r = d.norm(dim=1)
        grad = self.slope(d, r)
        old = self.rho
        rho = self.m * self.kernel(torch.zeros_like(self.m)) + self.total(i, self.m[j] * self.kernel(r))
        wd = self.x[wi] - self.bx[wj]
        wr = wd.norm(dim=1)
        ww = self.kernel(wr)
        rho = rho + self.total(wi, self.bm[wj] * ww)
        eta = 0.01 * h * h
        diff = self.m[j] / old[j] * (old[i] - old[j]) * 2 * (d * grad).sum(1) / (r * r + eta)
        rho = rho + 0.1 * h * self.c * self.total(i, diff) * dt
        p = (rho0 * self.c ** 2 / 7 * ((rho / rho0) ** 7 - 1)).clamp(min=0)
        self.rho, self.p = rho, p
        wall = lambda v: torch.zeros(len(self.bx), dtype=v.dtype, device=v.device).index_add_(0, wj, v)  # noqa: E731
        weight = wall(ww)
        pb = wall(ww * (p[wi] - rho[wi] * (wd @ self.g.reshape(3))))
        pb = torch.where(weight > 1e-12, (pb / weight.clamp(min=1e-300)).clamp(min=0), torch.zeros_like(pb))
        acc = self.total(i, -(self.m[j] * (p[i] / rho[i] ** 2 + p[j] / rho[j] ** 2))[:, None] * grad)
        vr = ((self.v[i] - self.v[j]) * d).sum(1)
        mu = h * vr / (r * r + eta)
        pi = (-self.alpha * self.c * mu + self.beta * mu * mu) / (0.5 * (rho[i] + rho[j]))
        acc += self.total(i, torch.where(vr < 0, -self.m[j] * pi, torch.zeros_like(pi))[:, None] * grad)
        acc += self.total(wi, -(self.bm[wj] * (p[wi] / rho[wi] ** 2 + pb[wj] / rho0 ** 2))[:, None]
                          * self.slope(wd, wr))
        r0 = 0.5 * h
        rep = 10 * 9.81 * 0.01 * (1 - wr / r0).clamp(min=0) ** 2 / r0
        acc += self.total(wi, (rep / wr)[:, None] * wd)
        self.a = acc + self.g

    def step(self, dt):
        if self.first:
            self.compute_forces(dt)
            self.first = False
        v = self.v + 0.5 * dt * self.a
        i, j = self.ff
        r = (self.x[i] - self.x[j]).norm(dim=1)
        f = self.m[j] / (0.5 * (self.rho[i] + self.rho[j])).clamp(min=1) * self.kernel(r)
        dv = self.total(i, f[:, None] * (v[j] - v[i]))
        x = self.x + (v + 0.5 * dv) * dt
        below, above = x < self.lo, x > self.hi
        x = torch.minimum(torch.maximum(x, self.lo), self.hi)
        self.v = torch.where((below & (v < 0)) | (above & (v > 0)), -0.2 * v, v)
        self.x = x
        self.compute_forces(dt)
        self.v = self.v + 0.5 * dt * self.a

    def timestep(self):
        signal = max(self.c, float((self.v.norm(dim=1) + self.c).max()))
        accel = float(self.a.norm(dim=1).max())
        dt = min(self.cfl * self.h / signal, 0.25 * math.sqrt(self.h / accel) if accel > 1e-12 else 0.01)
        return min(max(dt, 1e-8), 0.01)

    def variation(self):
        return float(((self.rho - 1000.0).abs() / 1000.0).max())
