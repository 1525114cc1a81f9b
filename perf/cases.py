"""The calls whose time matters to a user of this framework, as cases that a timing harness can run.

A pass hands the handle its inputs from page-locked host buffers, advances it the number of steps
between two looks at the data, and reads the results back into page-locked host buffers: the loop
that a program around the library runs (inputs up, steps, results down).  The handles, their
CUDA graphs and the host buffers are made once, in prepare().

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  handle, host inputs and host outputs
  run(state)           one pass; returns the outputs (the state's own buffers)
  work(case)           bytes and flops that one pass cannot do without
  exact(case, seed)    what run() returns, in 64 bits by plain torch
"""
import math

import numpy as np
import torch

from prestige_gb300 import ParticleSystem, make_config

G = 9.81
MODES = {"ieee": 0, "fast": 1}


# ------------------------------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # The smallest system in everyday use: the 2D dam break at dx = 0.02 (6,518 particles),
        # graph-replayed, 200 steps between two frames; bound by the latency of its launches.
        {"name": "dam_break_fast", "kind": "dam", "nx": 50, "ny": 100, "mode": "fast", "steps": 200},
        # The same in the default arithmetic (IEEE double, bit-exact with the CPU).
        {"name": "dam_break_ieee", "kind": "dam", "nx": 50, "ny": 100, "mode": "ieee", "steps": 100},
        # 3D lattice, double-word arithmetic: the smallest size of the benchmark's sweep ...
        {"name": "lattice_fast_256k", "kind": "lattice", "n": 262144, "precision": "f64", "mode": "fast",
         "mult": 0.5, "block": 0, "mom_block": 0, "steps": 40},
        # ... and the headline size, with the tuning that the autotuner picks there.
        {"name": "lattice_fast_4m", "kind": "lattice", "n": 4096000, "precision": "f64", "mode": "fast",
         "mult": 0.5, "block": 64, "mom_block": 256, "steps": 8},
        # 3D lattice in IEEE double (the default mode), a size that fills no tile or block evenly.
        {"name": "lattice_ieee_1m", "kind": "lattice", "n": 1000003, "precision": "f64", "mode": "ieee",
         "mult": 0.5, "block": 0, "mom_block": 0, "steps": 6},
        # 3D lattice in single precision with the library's default cell size, ragged.
        {"name": "lattice_f32_700k", "kind": "lattice", "n": 700001, "precision": "f32", "mode": "fast",
         "mult": 1.0, "block": 0, "mom_block": 0, "steps": 25},
        # Many small systems in one handle: 512 dam breaks of 500 to 50,000 fluid particles
        # (6.1 M particles with their walls), graph-replayed.
        {"name": "batch_512_fast", "kind": "batch", "systems": 512, "nmin": 500, "nmax": 50000, "mode": "fast",
         "steps": 20},
        # Differentiable runs: a checkpointed forward run and its backward pass, in both modes.
        {"name": "adjoint_fast_100k", "kind": "adjoint", "n": 100000, "mode": "fast", "steps": 40, "every": 10},
        {"name": "adjoint_ieee_50k", "kind": "adjoint", "n": 50000, "mode": "ieee", "steps": 20, "every": 5},
        # DEM: 200,000 loose spheres (free fall, hardly a contact), and a contact-dense packing.
        {"name": "dem_settling_200k", "kind": "dem_loose", "nx": 42, "ny": 42, "nz": 114, "steps": 150},
        {"name": "dem_dense_200k", "kind": "dem_dense", "nx": 58, "ny": 59, "nz": 58, "steps": 30},
        # The reference's own equation (force[i] += mass[j]) over the neighbour set, with the
        # neighbour counts: one call each on new positions.
        {"name": "equation_gather_500k", "kind": "gather", "n": 500009, "dim": 3, "mult": 1.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lattice", "lattice", "lattice", "dam", "dam", "batch", "adjoint", "dem_loose", "dem_dense",
                       "gather"])
    if kind == "lattice":
        precision, mode = rng.choice([("f64", "fast"), ("f64", "fast"), ("f64", "ieee"), ("f32", "fast"),
                                      ("f32", "ieee")])
        n = _log_int(rng, 10000, 1200000 if precision == "f64" and mode == "ieee" else 3000000)
        cost = 60 if precision == "f64" and mode == "ieee" else 12 if precision == "f64" else 8  # about us per 1000
        steps = max(2, min(60, int(40e3 / (cost * n / 1000.0 * 0.15 + 60))))
        return {"kind": kind, "n": n, "precision": precision, "mode": mode, "mult": rng.choice([0.5, 1.0]),
                "block": rng.choice([0, 0, 64, 256]), "mom_block": rng.choice([0, 0, 256]), "steps": steps}
    if kind == "dam":
        nx = rng.randint(20, 150)
        return {"kind": kind, "nx": nx, "ny": 2 * nx + rng.randint(-3, 3), "mode": rng.choice(["fast", "ieee"]),
                "steps": rng.randint(40, 120)}
    if kind == "batch":
        return {"kind": kind, "systems": _log_int(rng, 5, 300), "nmin": 500, "nmax": rng.choice([5000, 20000, 50000]),
                "mode": rng.choice(["fast", "fast", "ieee"]), "steps": rng.randint(6, 16)}
    if kind == "adjoint":
        every = rng.randint(3, 8)
        return {"kind": kind, "n": _log_int(rng, 4000, 60000), "mode": rng.choice(["fast", "ieee"]),
                "steps": every * rng.randint(2, 3) + rng.randint(0, 2), "every": every}
    if kind in ("dem_loose", "dem_dense"):
        side = rng.randint(16, 52)
        return {"kind": kind, "nx": side, "ny": side + rng.randint(-4, 4), "nz": side + rng.randint(-3, 9),
                "steps": rng.randint(20, 60) if kind == "dem_loose" else rng.randint(10, 30)}
    return {"kind": kind, "n": _log_int(rng, 5000, 900000), "dim": rng.choice([2, 3]), "mult": rng.choice([0.5, 1.0])}


# ------------------------------------------------------------------------------------------
# Inputs (plain torch on the GPU, from the seed alone)
# ------------------------------------------------------------------------------------------
class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda", dtype=torch.float64) * (hi - lo) + lo

    def normal(self, std, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float64) * std


def _side(n):
    s = int(round(n ** (1.0 / 3.0)))
    while s ** 3 < n:
        s += 1
    return s


def _lattice(n, seed, precision="f64", mode="fast", mult=0.5, block=0, fourier=False):
    """Jittered cubic lattice, dx = 0.01, h = 1.3 dx, random velocities and densities (fourier: the
    smooth velocity field of the differentiable runs, at rest density)."""
    dx, rho0, c0, rnd = 0.01, 1000.0, 10.0, _Random(seed)
    s = _side(n)
    idx = torch.arange(n, device="cuda")
    pos = torch.stack([idx % s, (idx // s) % s, idx // (s * s)], 1).double() * dx + 0.5 * dx
    pos += rnd.uniform(-0.2 * dx, 0.2 * dx, n, 3)
    if fourier:
        host = np.random.default_rng(seed)
        vel = torch.zeros_like(pos)
        for _ in range(8):
            kvec = host.integers(1, 4, size=3) * (2.0 * math.pi / (s * dx)) * host.choice([-1, 1], size=3)
            d = host.normal(size=3)
            phase = pos @ torch.tensor(kvec, device="cuda") + host.uniform(0.0, 2.0 * math.pi)
            vel += 0.05 / 8 * torch.outer(torch.sin(phase), torch.tensor(d / np.linalg.norm(d), device="cuda"))
        rho = torch.full((n,), rho0, device="cuda", dtype=torch.float64)
    else:
        vel = rnd.normal(0.1, n, 3)
        rho = rho0 * (1.0 + rnd.uniform(-0.01, 0.01, n))
    h = 1.3 * dx
    pad = 4.0 * h
    cfg = dict(model=0, dim=3, precision=1 if precision == "f64" else 0, gamma=7, n_fluid=-1, domain_lo=[-pad] * 3,
               domain_hi=[s * dx + pad] * 3, cell_multiplier=mult, h=h, rho0=rho0, c0=c0, alpha=0.1, eps_av=0.01,
               tait_B=rho0 * c0 * c0 / 7.0, gravity=[0.0, 0.0, 0.0], dt=0.25 * h / c0, f64_mode=MODES[mode],
               block_size=block)
    fields = {"pos": pos, "vel": vel, "rho": rho, "mass": torch.full((n,), rho0 * dx ** 3, device="cuda",
                                                                     dtype=torch.float64)}
    if precision == "f32":
        fields = {k: v.float() for k, v in fields.items()}
    return cfg, fields


def _dam(nx, ny, height, mode, rnd, precision=1):
    """2D dam break: nx x ny fluid particles of a column of this height in a tank of 2 x 1.5 of its
    height with three layers of fixed wall particles; the fluid is in motion (a jittered lattice with
    random velocities up to a tenth of sqrt(g H)), as it is throughout a run."""
    dx, layers, rho0 = height / ny, 3, 1000.0
    i = torch.arange(nx * ny, device="cuda")
    fluid = torch.stack([(i // ny).double() + 0.5, (i % ny).double() + 0.5], 1) * dx
    fluid += rnd.uniform(-0.05 * dx, 0.05 * dx, nx * ny, 2)
    ncol, nrow = int(round(2.0 * height / dx)), int(round(1.5 * height / dx))
    walls = []
    c = (torch.arange(-layers, ncol + layers, device="cuda").double() + 0.5) * dx
    r = (torch.arange(nrow, device="cuda").double() + 0.5) * dx
    for k in range(layers):
        off = (k + 0.5) * dx
        walls.append(torch.stack([c, torch.full_like(c, -off)], 1))
        walls.append(torch.stack([torch.full_like(r, -off), r], 1))
        walls.append(torch.stack([torch.full_like(r, ncol * dx + off), r], 1))
    pos = torch.cat([fluid] + walls)
    nf, n = nx * ny, pos.shape[0]
    h, c0 = 1.2 * dx, 10.0 * math.sqrt(2.0 * G * height)
    B = rho0 * c0 * c0 / 7
    vel = torch.zeros_like(pos)
    vel[:nf] = rnd.uniform(-1.0, 1.0, nf, 2) * (0.1 * math.sqrt(G * height))
    rho = torch.full((n,), rho0, device="cuda", dtype=torch.float64)
    rho[:nf] = rho0 * (1.0 + rho0 * G * (height - fluid[:, 1]).clamp_min(0.0) / B) ** (1.0 / 7.0)
    edge = layers * dx + 2.0 * h
    cfg = dict(model=0, dim=2, precision=precision, gamma=7, n_fluid=nf, domain_lo=[-edge, -edge, 0.0],
               domain_hi=[ncol * dx + edge, 1.5 * height + 2.0 * h, 0.0], cell_multiplier=1.0, h=h, rho0=rho0, c0=c0,
               alpha=0.1, eps_av=0.01, tait_B=B, gravity=[0.0, -G, 0.0], dt=0.25 * h / c0, f64_mode=MODES[mode])
    mass = torch.full((n,), rho0 * dx * dx, device="cuda", dtype=torch.float64)
    return cfg, {"pos": pos, "vel": vel, "rho": rho, "mass": mass}


def _batch_shapes(case):
    """Fluid columns (nx, ny) and heights of a batch: sizes log-uniform, a column twice as high as wide."""
    r = np.random.default_rng(3)
    ns = np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), size=case["systems"]))
    hs = r.uniform(0.5, 2.0, size=case["systems"])
    return [(max(4, int(round(math.sqrt(m / 2)))), max(8, int(round(math.sqrt(m * 2)))), float(h))
            for m, h in zip(ns, hs)]


def _batch(case, seed):
    rnd = _Random(seed)
    parts = [_dam(nx, ny, h, case["mode"], rnd) for nx, ny, h in _batch_shapes(case)]
    fields = {k: torch.cat([p[1][k] for p in parts]) for k in ("pos", "vel", "rho", "mass")}
    return [p[0] for p in parts], [p[1]["rho"].shape[0] for p in parts], fields


def _spheres(case, seed):
    """DEM: loose spheres of radii U[0.5, 1.0] mm at the density of a random sequential insertion of
    200,000 in 0.1 x 0.1 x 0.3 m (a jittered lattice without overlaps), or a lattice of 0.5 mm
    spheres compressed by 2 % with random velocities and spins, every contact path active."""
    rnd, side = _Random(seed), (case["nx"], case["ny"], case["nz"])
    idx = torch.stack(torch.meshgrid(*[torch.arange(k, device="cuda").double() for k in side], indexing="ij"),
                      -1).reshape(-1, 3)
    n = idx.shape[0]
    if case["kind"] == "dem_loose":
        gap, rmax = 2.4e-3, 1.0e-3
        radius = rnd.uniform(0.5e-3, 1.0e-3, n)
        pos = (idx + 0.5) * gap + rnd.uniform(-0.19e-3, 0.19e-3, n, 3)
        vel, omega = rnd.normal(0.01, n, 3), rnd.normal(1.0, n, 3)
        box = [k * gap for k in side]
        wall_hi = box
    else:
        rmax = 0.5e-3
        gap = 2 * rmax * 0.98
        radius = rmax * (1.0 - rnd.uniform(0.0, 0.05, n))
        pos = (idx + 0.5) * gap + rnd.uniform(-0.05, 0.05, n, 3) * rmax
        vel, omega = rnd.normal(0.05, n, 3), rnd.normal(50.0, n, 3)
        box = [k * gap for k in side]
        wall_hi = [b - 0.01 * rmax for b in box]
    mass = 2600.0 * 4.0 / 3.0 * math.pi * radius ** 3
    cfg = dict(model=1, dim=3, precision=1, domain_lo=[-2e-3] * 3, domain_hi=[b + 2e-3 for b in box],
               cell_multiplier=1.0, gravity=[0.0, 0.0, -G], dt=1e-6, kn=1e5, restitution=0.9, mu=0.3,
               kt=1e5 * 2.0 / 7.0, r_max=rmax, wall_lo=[0.0, 0.0, 0.0], wall_hi=wall_hi, contact_capacity=16)
    return cfg, {"pos": pos, "vel": vel, "omega": omega, "radius": radius, "mass": mass}


def _gather(case, seed):
    n, dim, rnd = case["n"], case["dim"], _Random(seed)
    dx = 0.01
    s = _side(n) if dim == 3 else int(math.ceil(math.sqrt(n)))
    idx = torch.arange(n, device="cuda")
    cols = [idx % s, (idx // s) % s, idx // (s * s)][:dim]
    pos = torch.stack(cols, 1).double() * dx + rnd.uniform(0.3 * dx, 0.7 * dx, n, dim)
    h = 1.3 * dx
    cfg = dict(model=0, dim=dim, precision=1, n_fluid=-1, domain_lo=[-4 * h] * 3, domain_hi=[s * dx + 4 * h] * 3,
               cell_multiplier=case["mult"], h=h, f64_mode=0)
    return cfg, {"pos": pos, "force": rnd.normal(1.0, n), "mass": rnd.uniform(0.5, 1.5, n)}


def _system_inputs(case, seed):
    kind = case["kind"]
    if kind == "lattice":
        return _lattice(case["n"], seed, case["precision"], case["mode"], case["mult"], case["block"])
    if kind == "dam":
        return _dam(case["nx"], case["ny"], 2.0, case["mode"], _Random(seed))
    if kind == "adjoint":
        return _lattice(case["n"], seed, "f64", case["mode"], 1.0, fourier=True)
    if kind == "gather":
        return _gather(case, seed)
    return _spheres(case, seed)


def _target(case, seed, pos):
    """Final positions that a differentiable run is to reach."""
    return pos + _Random(seed + 7919).normal(0.05 * 0.01, *pos.shape)


# ------------------------------------------------------------------------------------------
# A pass
# ------------------------------------------------------------------------------------------
def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        cfgs, counts, fields = _batch(case, seed)
        system = ParticleSystem.batch(cfgs, counts)
    else:
        cfg, fields = _system_inputs(case, seed)
        system = ParticleSystem(make_config(**cfg), fields["pos"].shape[0])
    st = {"kind": kind, "system": system, "steps": case.get("steps", 0), "every": case.get("every", 0)}
    inputs = {k: _pinned(v) for k, v in fields.items()}
    if kind in ("dem_loose", "dem_dense"):  # properties of the spheres, not of a run
        system.set("radius", inputs.pop("radius").numpy())
        system.set("mass", inputs.pop("mass").numpy())
    if kind == "gather":
        system.set("force", inputs["force"].numpy())  # creates the slice
    st["inputs"] = inputs
    out = {"gather": ("force",), "adjoint": ("pos",), "dem_loose": ("pos", "vel", "omega"),
           "dem_dense": ("pos", "vel", "omega")}.get(kind, ("pos", "vel", "rho"))
    st["outputs"] = {k: torch.empty(inputs[k].shape, dtype=inputs[k].dtype, pin_memory=True) for k in out}
    if kind == "adjoint":
        st["target"] = _pinned(_target(case, seed, fields["pos"]))
    if kind == "lattice" and case["mom_block"]:
        system.set_momentum_block(case["mom_block"])
    if kind in ("dam", "batch", "dem_loose", "dem_dense"):
        system.enable_graph(True)
    return st


def _load(system, inputs, put):
    for name, h in inputs.items():
        put(name, h.data_ptr(), h.numel(), h.dtype == torch.float64)


def _store(system, outputs):
    for name, h in outputs.items():
        system.get_ptr_async(name, h.data_ptr(), h.numel(), h.dtype == torch.float64)
    system.wait_io()


def run(state):
    system, kind = state["system"], state["kind"]
    # the differentiable run starts from inputs that are in place; the others upload beside their steps
    _load(system, state["inputs"], system.set_ptr if kind == "adjoint" else system.set_ptr_async)
    if kind == "gather":
        counts = system.count_neighbors()
        system.gather_sum("force", "mass")
        _store(system, state["outputs"])
        return {"counts": counts, "force": state["outputs"]["force"]}
    if kind == "adjoint":
        system.forward_checkpointed(state["steps"], state["every"])
        _store(system, state["outputs"])
        pos = state["outputs"]["pos"]
        dL = (pos - state["target"]) * (2.0 / system.n)
        dalpha, dB, dv0 = system.backward(dL.numpy())
        return {"pos": pos, "dalpha": dalpha, "dB": dB, "dv0": dv0}
    system.step_async(state["steps"])
    _store(system, state["outputs"])
    out = dict(state["outputs"])
    if kind in ("dem_loose", "dem_dense"):
        out["contacts"] = system.dem_contacts()
    return out


# ------------------------------------------------------------------------------------------
# Work
# ------------------------------------------------------------------------------------------
def work(case):
    """Bytes: the particle state read once and written once per step.  Flops: those of the method
    (24.9 per pair in the continuity sum, 34.4 in the momentum sum, 28 per particle; a contact about
    130), with the mean neighbour counts of these lattices (74 in 3D, 20 in 2D)."""
    kind, steps = case["kind"], case.get("steps", 1)
    if kind in ("lattice", "adjoint"):
        eb = 4 if case.get("precision") == "f32" else 8
        passes = 3 if kind == "adjoint" else 1  # forward, and a reverse sweep of about twice its work
        return {"bytes": passes * steps * case["n"] * 15 * eb, "flops": passes * steps * case["n"] * (74 * 59.3 + 28)}
    if kind in ("dam", "batch"):
        shapes = [(case["nx"], case["ny"], 2.0)] if kind == "dam" else _batch_shapes(case)
        n = sum(nx * ny + 3 * (2 * ny + 6 + 2 * int(round(1.5 * ny))) for nx, ny, _ in shapes)
        return {"bytes": steps * n * 11 * 8, "flops": steps * n * (20 * 59.3 + 28)}
    if kind in ("dem_loose", "dem_dense"):
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": steps * n * 160, "flops": steps * n * (30 + (2.5 * 130 if kind == "dem_dense" else 0))}
    n, dim = case["n"], case["dim"]
    nbr = 74 if dim == 3 else 21
    return {"bytes": n * (8 * dim + 8 + 16 + 4), "flops": n * nbr * (3 * dim + 1)}


# ------------------------------------------------------------------------------------------
# The same results in 64 bits, by plain torch
# ------------------------------------------------------------------------------------------
_PAIRS = 60_000_000  # candidate pairs held at a time


def _pairs(pos, support, group=None, self_pairs=False):
    """Lists of index tensors (i, j) of all pairs with |x_i - x_j| < support[i], i ascending;
    support: one value per particle; group: particles of different groups are no pairs."""
    n, dim = pos.shape
    lo = pos.min(0).values
    if group is None:
        cell = ((pos - lo) / support.max()).long() + 1
        top = cell.max(0).values + 2
        key = cell[:, 0]
        stride = int(top[0])
        strides = [stride]
        for d in range(1, dim):
            key = key + cell[:, d] * stride
            stride *= int(top[d])
            strides.append(stride)
    else:
        cell = ((pos - lo) / support[:, None]).long() + 1  # one support per group
        top = [int(v) + 2 for v in cell.max(0).values]
        key = cell[:, 0] + cell[:, 1] * top[0] + group * (top[0] * top[1])
        strides = [top[0]]
    skey, order = torch.sort(key, stable=True)
    rows = [0]
    for d in range(dim - 1):
        rows = [r + o * strides[d] for r in rows for o in (-1, 0, 1)]
    out = []
    chunk = max(1, n // max(1, math.ceil(n * 30.0 * len(rows) / _PAIRS)))
    xs, ss = pos[order], support[order] ** 2
    for a in range(0, n, chunk):
        b = min(n, a + chunk)
        ii, jj = [], []
        for r in rows:
            k = skey[a:b] + r
            first = torch.searchsorted(skey, k - 1)
            count = torch.searchsorted(skey, k + 1, right=True) - first
            i = torch.repeat_interleave(torch.arange(b - a, device="cuda"), count)
            j = torch.arange(i.shape[0], device="cuda") - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
            j = j + first[i]
            i = i + a
            d2 = ((xs[i] - xs[j]) ** 2).sum(1)
            keep = (d2 < ss[i]) if self_pairs else (d2 < ss[i]) & (d2 > 0)
            ii.append(order[i[keep]])
            jj.append(order[j[keep]])
        out.append((torch.cat(ii), torch.cat(jj)))
    return out


class _Fluid:
    """Parameters of the SPH systems, one value per particle (or a number for a single system)."""

    def __init__(self, cfgs, counts):
        self.dim = cfgs[0]["dim"]
        single = len(cfgs) == 1

        def per(f):
            if single:
                return float(f(cfgs[0]))
            v = torch.tensor([f(c) for c in cfgs], dtype=torch.float64, device="cuda")
            return torch.repeat_interleave(v, torch.tensor(counts, device="cuda"))

        self.h = per(lambda c: c["h"])
        self.rho0, self.c0, self.B = per(lambda c: c["rho0"]), per(lambda c: c["c0"]), per(lambda c: c["tait_B"])
        self.dt, self.eps = per(lambda c: c["dt"]), per(lambda c: c["eps_av"])
        self.alpha = float(cfgs[0]["alpha"])
        self.gravity = torch.tensor(cfgs[0]["gravity"][:self.dim], dtype=torch.float64, device="cuda")
        n = sum(counts)
        self.support = 2.0 * self.h * torch.ones(n, dtype=torch.float64, device="cuda")
        self.group = None if single else torch.repeat_interleave(torch.arange(len(cfgs), device="cuda"),
                                                                 torch.tensor(counts, device="cuda"))
        fluid = [torch.arange(m, device="cuda") < (m if c["n_fluid"] < 0 else c["n_fluid"])
                 for c, m in zip(cfgs, counts)]
        self.fluid = torch.cat(fluid)[:, None]


def _at(v, i):
    return v if isinstance(v, float) else v[i]


def _per_row(v):
    return v if isinstance(v, float) else v[:, None]


def _sph_step(p, pairs, pos, vel, rho, mass, alpha, B):
    """rho' = rho + dt C(x, v); v' = v + dt (M(x, v, rho') + g); x' = x + dt v'."""
    sigma_h = 10.0 / (7.0 * math.pi) if p.dim == 2 else 1.0 / math.pi

    def geometry(i, j):
        d = pos[i] - pos[j]
        r2 = (d * d).sum(1)
        r = r2.sqrt()
        h = _at(p.h, i)
        q = r / h
        sigma = sigma_h / h ** p.dim
        F = torch.where(q < 1.0, sigma / h ** 2 * (2.25 * q - 3.0), -0.75 * sigma / h * (2.0 - q) ** 2 / r)
        w = ((vel[i] - vel[j]) * d).sum(1)
        return d, r2, F, w, h

    drho = torch.zeros_like(rho)
    for i, j in pairs:
        _, _, F, w, _ = geometry(i, j)
        drho = drho.index_add(0, i, mass[j] * w * F)
    rho = rho + p.dt * drho
    P = B * ((rho / p.rho0) ** 7 - 1.0) / rho ** 2
    acc = torch.zeros_like(vel)
    for i, j in pairs:
        d, r2, F, w, h = geometry(i, j)
        visc = -2.0 * alpha * _at(p.c0, i) * h * w / ((r2 + _at(p.eps, i) * h * h) * (rho[i] + rho[j]))
        visc = torch.where(w < 0, visc, torch.zeros_like(visc))
        acc = acc.index_add(0, i, -(mass[j] * (P[i] + P[j] + visc) * F)[:, None] * d)
    dt = _per_row(p.dt)
    nv = torch.where(p.fluid, vel + dt * (acc + p.gravity), vel)
    return torch.where(p.fluid, pos + dt * nv, pos), nv, rho


def _exact_sph(cfgs, counts, fields, steps):
    p = _Fluid(cfgs, counts)
    pos, vel, rho, mass = (fields[k].double() for k in ("pos", "vel", "rho", "mass"))
    for _ in range(steps):
        pos, vel, rho = _sph_step(p, _pairs(pos, p.support, p.group), pos, vel, rho, mass, p.alpha, p.B)
    return {"pos": pos, "vel": vel, "rho": rho}


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint

    cfg, fields = _system_inputs(case, seed)
    p = _Fluid([cfg], [case["n"]])
    alpha = torch.tensor(p.alpha, dtype=torch.float64, device="cuda", requires_grad=True)
    B = torch.tensor(p.B, dtype=torch.float64, device="cuda", requires_grad=True)
    v0 = fields["vel"].clone().requires_grad_(True)
    pos, vel, rho, mass = fields["pos"], v0, fields["rho"], fields["mass"]

    def step(pos, vel, rho, alpha, B):
        with torch.no_grad():
            pairs = _pairs(pos.detach(), p.support)
        return _sph_step(p, pairs, pos, vel, rho, mass, alpha, B)

    for _ in range(case["steps"]):
        pos, vel, rho = checkpoint(step, pos, vel, rho, alpha, B, use_reentrant=False)
    dL = (pos.detach() - _target(case, seed, fields["pos"])) * (2.0 / case["n"])
    da, db, dv0 = torch.autograd.grad(pos, (alpha, B, v0), dL)
    return {"pos": pos.detach(), "dalpha": float(da), "dB": float(db), "dv0": dv0}


def _contact(cfg, n, delta, vr, meff, xi):
    """Force on the particle, its tangential part and the new spring of contacts with normals n."""
    le = math.log(cfg["restitution"])
    vn = (vr * n).sum(1, keepdim=True)
    vt = vr - vn * n
    gn = (-2.0 * le / math.sqrt(math.pi ** 2 + le * le)) * (meff * cfg["kn"]).sqrt()[:, None]
    fn = cfg["kn"] * delta[:, None] - gn * vn
    xi = xi - (xi * n).sum(1, keepdim=True) * n + vt * cfg["dt"]
    ft = -cfg["kt"] * xi - gn * vt
    size = (ft * ft).sum(1, keepdim=True).sqrt()
    lim = cfg["mu"] * fn.abs()
    slip = size > lim
    ft = torch.where(slip, ft * (lim / size.clamp_min(1e-300)), ft)
    xi = torch.where(slip, -(ft + gn * vt) / cfg["kt"], xi)
    return fn * n + ft, ft, xi


def _exact_dem(case, seed):
    cfg, f = _spheres(case, seed)
    pos, vel, omega, radius, mass = (f[k] for k in ("pos", "vel", "omega", "radius", "mass"))
    n, dt = pos.shape[0], cfg["dt"]
    g = torch.tensor(cfg["gravity"], dtype=torch.float64, device="cuda")
    reach = torch.full((n,), 2.0 * cfg["r_max"], dtype=torch.float64, device="cuda")
    keys, springs = torch.empty(0, dtype=torch.long, device="cuda"), torch.empty(0, 3, dtype=torch.float64, device="cuda")
    wall = torch.zeros(6, n, 3, dtype=torch.float64, device="cuda")
    contacts = 0
    for _ in range(case["steps"]):
        F, T = torch.zeros_like(pos), torch.zeros_like(pos)
        pairs = _pairs(pos, reach)
        i, j = torch.cat([a for a, _ in pairs]), torch.cat([b for _, b in pairs])
        d = pos[i] - pos[j]
        touch = (d * d).sum(1) < (radius[i] + radius[j]) ** 2
        i, j, d = i[touch], j[touch], d[touch]
        contacts = int(i.shape[0])
        key = i * n + j
        dist = (d * d).sum(1).sqrt()
        nrm = d / dist[:, None]
        spin = radius[i, None] * omega[i] + radius[j, None] * omega[j]
        vr = vel[i] - vel[j] - torch.linalg.cross(spin, nrm)
        xi = torch.zeros_like(d)
        if keys.shape[0] and key.shape[0]:
            at = torch.searchsorted(keys, key).clamp_max(keys.shape[0] - 1)
            xi = torch.where((keys[at] == key)[:, None], springs[at], xi)
        fc, ft, xi = _contact(cfg, nrm, radius[i] + radius[j] - dist, vr, mass[i] * mass[j] / (mass[i] + mass[j]), xi)
        F.index_add_(0, i, fc)
        T.index_add_(0, i, -radius[i, None] * torch.linalg.cross(nrm, ft))
        keys, order = torch.sort(key)
        springs = xi[order]
        for face in range(6):
            ax, hi = face // 2, face % 2
            gap = cfg["wall_hi"][ax] - pos[:, ax] if hi else pos[:, ax] - cfg["wall_lo"][ax]
            k = torch.nonzero(gap < radius)[:, 0]
            nrm = torch.zeros(k.shape[0], 3, dtype=torch.float64, device="cuda")
            nrm[:, ax] = -1.0 if hi else 1.0
            vr = vel[k] - torch.linalg.cross(radius[k, None] * omega[k], nrm)
            fc, ft, xi = _contact(cfg, nrm, radius[k] - gap[k], vr, mass[k], wall[face][k])
            F[k] += fc
            T[k] -= radius[k, None] * torch.linalg.cross(nrm, ft)
            wall[face].zero_()
            wall[face][k] = xi
        vel = vel + dt * (F / mass[:, None] + g)
        pos = pos + dt * vel
        omega = omega + dt * T / (0.4 * mass * radius ** 2)[:, None]
    return {"pos": pos, "vel": vel, "omega": omega, "contacts": contacts}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        cfgs, counts, fields = _batch(case, seed)
        return _exact_sph(cfgs, counts, fields, case["steps"])
    if kind in ("lattice", "dam"):
        cfg, fields = _system_inputs(case, seed)
        return _exact_sph([cfg], [fields["pos"].shape[0]], fields, case["steps"])
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind in ("dem_loose", "dem_dense"):
        return _exact_dem(case, seed)
    cfg, f = _gather(case, seed)
    n = case["n"]
    support = torch.full((n,), 2.0 * cfg["h"], dtype=torch.float64, device="cuda")
    force, counts = f["force"].clone(), torch.zeros(n, dtype=torch.long, device="cuda")
    for i, j in _pairs(f["pos"], support, self_pairs=True):
        force.index_add_(0, i, f["mass"][j])
        counts += torch.bincount(i, minlength=n)
    return {"counts": None, "force": force}
