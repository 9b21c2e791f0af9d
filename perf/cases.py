"""Performance cases: the work that users of pysph_gb300 have it do.

A case is a dict of plain values.  ``listed()`` returns the named ones,
``draw(rng)`` another one of the same ranges, ``prepare(case, seed)`` what a
program has in hand before the call, ``run(state)`` one pass through the
public entry points, ``work(case)`` the bytes and operations a pass cannot do
without and ``exact(case, seed)`` the pass's results in 64 bits by plain
torch.

Kinds of case
-------------
* ``cube``    -- one time step of a 3D block of fluid (jittered lattice,
  SPHRho + Tait + pressure gradient + Monaghan viscosity): the throughput
  configuration, from 16^3 to 161^3 particles.
* ``drop``    -- one time step of the 2D elliptical drop (summation density,
  XSPH), with one smoothing length or with a smoothing length per particle
  (symmetric neighbour lists).
* ``patch``   -- one time step of the 2D fluid-solver patch: continuity
  density rate, MomentumEquation, XSPH.
* ``dam``     -- one time step of the 2D dam break: fluid and wall arrays,
  boundary force, gravity.
* ``batch``   -- one time step of many independent drops advanced together.
* ``fresh``   -- a snapshot whose positions are new: neighbour structure from
  scratch, then the summation density (post-processing, start-up, fast flows).
* ``closure`` -- the learned closure's evaluation on a dam-break state:
  neighbour features, then the network.
* ``forward`` -- the closure network on samples already extracted.
* ``train``   -- one training step of the closure network: forward, backward,
  Adam.

The step cases advance a simulation that runs on from pass to pass, so light
neighbour refreshes and full neighbour builds come in the proportion in which
a simulation has them; after ``STEPS`` steps the program starts its
simulation again from the initial state.
"""
import math

import numpy as np
import torch

import pysph_gb300
from pysph_gb300 import learned, workloads
from pysph_gb300.batch import SimulationBatch

# steps of one simulation before it starts again (a batch's particles may
# not be put back by more than a cell, so its runs are shorter)
STEPS = 128
BATCH_STEPS = 16

# dam break: reference sound speed 10 sqrt(2 g H), H = 2, and rest density
GRAVITY = -9.81
DAM_C0 = 10.0 * math.sqrt(2.0 * 9.81 * 2.0)
DAM_RHO0 = 1000.0


def listed():
    return [
        # the smallest simulation anyone runs: the reference's own drop
        # example (5 025 particles, Euler), where latency and launches count
        dict(name="drop_5k", kind="drop", dx=0.025, integrator="euler", variable_h=False),
        # per-particle smoothing lengths: symmetric lists
        dict(name="drop_varh_31k", kind="drop", dx=0.01, integrator="rk2", variable_h=True),
        # the reference's FluidSolver recipe (continuity density), RK2
        dict(name="patch_20k", kind="patch", dx=0.0125, integrator="rk2"),
        # dam break of the closure's training runs: 20 000 fluid particles
        # and three layers of wall
        dict(name="dam_23k", kind="dam", dx=0.01, integrator="rk2"),
        # an ordinary 3D run
        dict(name="cube_64k", kind="cube", side=40, integrator="rk2"),
        # the headline throughput configuration
        dict(name="cube_1m", kind="cube", side=100, integrator="rk2"),
        # the largest
        dict(name="cube_4m", kind="cube", side=161, integrator="rk2"),
        # a new snapshot of an ordinary 3D run, an odd size
        dict(name="fresh_275k", kind="fresh", side=65),
        # 256 independent drops of seeded radius and spacing, 2 M particles
        dict(name="batch_256", kind="batch", count=256, layout=0, dxmin=0.01, integrator="euler"),
        # closure on the 80 000-particle dam break
        dict(name="closure_80k", kind="closure", dx=0.005),
        # the network over a million recorded samples
        dict(name="forward_1m", kind="forward", samples=1 << 20),
        # the minibatch that the closure is trained with
        dict(name="train_8k", kind="train", samples=8192),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("cube", "cube", "drop", "drop", "patch", "dam", "batch", "fresh",
                       "closure", "forward", "train"))
    if kind == "cube":
        return dict(kind=kind, side=int(round(_log_uniform(rng, 4.1e3, 4.1e6) ** (1.0 / 3.0))),
                    integrator=rng.choice(("rk2", "rk2", "euler", "pc")))
    if kind == "drop":
        return dict(kind=kind, dx=round(_log_uniform(rng, 0.0045, 0.04), 6),
                    integrator=rng.choice(("euler", "rk2", "rk4")),
                    variable_h=rng.choice((False, False, True)))
    if kind == "patch":
        return dict(kind=kind, dx=round(_log_uniform(rng, 0.006, 0.04), 6),
                    integrator=rng.choice(("rk2", "pc", "euler")))
    if kind == "dam":
        return dict(kind=kind, dx=round(1.0 / rng.randint(50, 220), 9),
                    integrator=rng.choice(("rk2", "rk2", "euler")))
    if kind == "batch":
        return dict(kind=kind, count=int(round(_log_uniform(rng, 16, 256))),
                    layout=rng.randint(0, 99), dxmin=rng.choice((0.01, 0.015, 0.02)),
                    integrator=rng.choice(("euler", "rk2")))
    if kind == "fresh":
        return dict(kind=kind, side=int(round(_log_uniform(rng, 4.1e3, 1.1e6) ** (1.0 / 3.0))))
    if kind == "closure":
        return dict(kind=kind, dx=round(1.0 / rng.randint(60, 220), 9))
    if kind == "forward":
        return dict(kind=kind, samples=int(_log_uniform(rng, 1000, 1.05e6)))
    return dict(kind=kind, samples=int(_log_uniform(rng, 1000, 2.6e5)))


# ---------------------------------------------------------------------------
# inputs (NumPy, FP64, from the seed alone)
# ---------------------------------------------------------------------------

def _cube_props(case, seed):
    side = case["side"]
    dx = 1.0 / side
    rng = np.random.default_rng([1, seed, side])
    a = (np.arange(side) + 0.5) * dx
    z, y, x = np.meshgrid(a, a, a, indexing="ij")
    n = side ** 3
    pos = [c.ravel() + rng.uniform(-0.1 * dx, 0.1 * dx, n) for c in (x, y, z)]
    vel = [rng.normal(0.0, 0.01, n) for _ in range(3)]
    return dict(x=pos[0], y=pos[1], z=pos[2], u=vel[0], v=vel[1], w=vel[2],
                m=np.full(n, dx ** 3), h=np.full(n, 1.2 * dx), rho=np.ones(n), cs=np.zeros(n))


def _disc(radius, dx):
    a = np.arange(-1.05 * radius, 1.05 * radius + 1e-4, dx)
    x, y = (c.ravel() for c in np.meshgrid(a, a, indexing="ij"))
    keep = np.sqrt(x * x + y * y) <= radius + 1e-10
    return x[keep], y[keep]


def _drop_props(radius, dx, rng, variable_h=False):
    x, y = _disc(radius, dx)
    n = x.size
    x = x + rng.uniform(-0.02 * dx, 0.02 * dx, n)
    y = y + rng.uniform(-0.02 * dx, 0.02 * dx, n)
    h = np.full(n, 1.3 * dx)
    if variable_h:
        h *= 1.0 + rng.uniform(-0.25, 0.25, n)
    return dict(x=x, y=y, u=-100.0 * x, v=100.0 * y, m=np.full(n, dx * dx), h=h,
                rho=np.ones(n), cs=np.full(n, 100.0))


def _patch_props(case, seed):
    dx = case["dx"]
    rng = np.random.default_rng([3, seed])
    p = _drop_props(1.0, dx, rng)
    p["h"] = np.full_like(p["h"], 2.0 * dx)
    p["p"] = 0.5 * 100.0 ** 2 * (1.0 - (p["x"] ** 2 + p["y"] ** 2))
    return p


def _dam_props(case, seed, jitter=0.02):
    dx = case["dx"]
    rng = np.random.default_rng([4, seed])
    fluid, wall = workloads.dam_break(dx=dx)
    n = fluid["x"].size
    fluid["x"] = fluid["x"] + rng.uniform(-jitter * dx, jitter * dx, n)
    fluid["y"] = fluid["y"] + rng.uniform(-jitter * dx, jitter * dx, n)
    return fluid, wall


def _batch_props(case, seed):
    lay = np.random.default_rng([5, case["layout"]])
    radii = lay.uniform(0.5, 1.5, case["count"])
    dxs = lay.uniform(case["dxmin"], 4.0 * case["dxmin"], case["count"])
    rng = np.random.default_rng([6, seed])
    return [_drop_props(float(r), float(d), rng) for r, d in zip(radii, dxs)]


def _closure_props(case, seed):
    """A dam-break state in motion: jittered column, velocities of a few per
    cent of c0, density within 1 % and its Tait pressure."""
    fluid, wall = _dam_props(case, seed, jitter=0.15)
    rng = np.random.default_rng([7, seed])
    n = fluid["x"].size
    fluid["u"] = rng.normal(0.0, 0.03 * DAM_C0, n)
    fluid["v"] = rng.normal(0.0, 0.03 * DAM_C0, n)
    ratio = 1.0 + rng.normal(0.0, 0.01, n)
    fluid["rho"] = DAM_RHO0 * ratio
    fluid["p"] = DAM_C0 ** 2 * DAM_RHO0 / 7.0 * (ratio ** 7 - 1.0)
    fluid["cs"] = DAM_C0 * ratio ** 3
    return fluid, wall


def _closure_scaling():
    """Per-channel feature mean and standard deviation of those states."""
    b = DAM_C0 ** 2 * DAM_RHO0 / 7.0
    mean = [0.0, 0.0, 0.0, 0.0, DAM_RHO0, 0.02 * b]
    std = [1.1, 1.1, 0.042, 0.042, 0.01 * DAM_RHO0, 0.07 * b]
    return mean, std


def _net_params(seed):
    rng = np.random.default_rng([8, seed])
    w1 = rng.uniform(-1, 1, 128 * 192) / np.sqrt(192)
    b1 = rng.uniform(-0.1, 0.1, 128)
    w2 = rng.uniform(-1, 1, 128 * 128) / np.sqrt(128)
    b2 = rng.uniform(-0.1, 0.1, 128)
    w3 = rng.uniform(-1, 1, 2 * 128) / np.sqrt(128)
    b3 = rng.uniform(-0.1, 0.1, 2)
    return np.concatenate([w1, b1, w2, b2, w3, b3]).astype(np.float32)


def _samples(n, count, seed):
    """``count`` minibatches of n standardised samples and targets; the last
    neighbours of a sample are missing (zero rows) as at a free surface."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 + seed)
    x = torch.randn((count * n, 32, 6), generator=g, device="cuda", dtype=torch.bfloat16)
    nbr = torch.randint(12, 33, (count * n, 1, 1), generator=g, device="cuda")
    x *= torch.arange(32, device="cuda").view(1, 32, 1) < nbr
    x = x.view(count * n, 192)
    t = torch.randn((count * n, 2), generator=g, device="cuda")
    return x, t


def _minibatches(n):
    return max(2, (1 << 18) // n)


def _time_step(case):
    if case["kind"] == "cube":
        return 0.01 / case["side"]      # 1e-4 at 100^3, half the sound-speed limit or less
    if case["kind"] == "dam":
        return 2.5e-3 * case["dx"]
    return min(1e-5, 1e-3 * case["dx"])


# ---------------------------------------------------------------------------
# one pass through the public entry points
# ---------------------------------------------------------------------------

FIELDS = {2: ("x", "y", "u", "v", "rho", "p", "cs"),
          3: ("x", "y", "z", "u", "v", "w", "rho", "p", "cs")}


def prepare(case, seed):
    api = pysph_gb300.api()
    kind = case["kind"]
    st = dict(kind=kind)
    if kind in ("cube", "drop", "patch", "dam"):
        if kind == "cube":
            s, parts = workloads.setup_cube(api, _cube_props(case, seed),
                                            integrator=case["integrator"])
        elif kind == "drop":
            rng = np.random.default_rng([2, seed])
            props = _drop_props(1.0, case["dx"], rng, case["variable_h"])
            s, parts = workloads.setup_drop(api, props, c0=100.0, integrator=case["integrator"],
                                            variable_h=case["variable_h"])
        elif kind == "patch":
            s, parts = workloads.setup_fluid_solver(api, _patch_props(case, seed),
                                                    integrator=case["integrator"])
        else:
            fluid, wall = _dam_props(case, seed)
            s, parts = workloads.setup_dam_break(api, fluid, wall, case["dx"], DAM_C0,
                                                 integrator=case["integrator"])
        pa = parts.arrays[0]
        st.update(solver=s, particles=parts, fluid=pa, dt=_time_step(case), done=0,
                  fields=FIELDS[3 if kind == "cube" else 2],
                  start={f: pa.get_device(f).clone() for f in FIELDS[3]})
    elif kind == "batch":
        b = SimulationBatch(_batch_props(case, seed), dim=2, dt=1e-5, co=100.0,
                            integrator=case["integrator"])
        st.update(batch=b, done=0,
                  start={f: b.arrays[f].clone() for f in ("x", "y", "u", "v")})
    elif kind == "fresh":
        props = _cube_props(case, seed)
        pa = api.base.get_particle_array(name="fluid", **props)
        parts = api.base.Particles(arrays=[pa])
        kernel = api.base.CubicSplineKernel(dim=3)
        calc = api.sph.SPHCalc(parts, [pa], pa, kernel, [api.sph.SPHRho.get_func(pa, pa)],
                               ["rho"])
        st.update(particles=parts, fluid=pa, calc=calc,
                  snapshot={c: pa.get_device(c).clone() for c in "xyz"})
    elif kind == "closure":
        fluid, wall = _closure_props(case, seed)
        s, parts = workloads.setup_dam_break(api, fluid, wall, case["dx"], DAM_C0)
        mean, std = _closure_scaling()
        model = learned.MomentumMLP()
        model.set_params(_net_params(seed))
        st.update(solver=s, particles=parts, fluid=parts.arrays[0], model=model,
                  norm=learned.Normalisation(DAM_C0, mean, std))
    else:
        n = case["samples"]
        model = learned.MomentumMLP()
        model.set_params(_net_params(seed))
        x, t = _samples(n, _minibatches(n) if kind == "train" else 1, seed)
        st.update(model=model, x=x, t=t, n=n, next=0)
    return st


def run(st):
    kind = st["kind"]
    if "solver" in st and kind != "closure":
        if st["done"] == STEPS:         # the next simulation of the same flow
            st["fluid"].set(**st["start"])
            st["particles"].cell_manager.rebuild(check_jump=False)
            st["done"] = 0
        st["solver"].integrator.integrate(st["dt"])
        st["done"] += 1
        return {f: st["fluid"].get_device(f) for f in st["fields"]}
    if kind == "batch":
        b = st["batch"]
        if st["done"] == BATCH_STEPS:
            b.set(**st["start"])
            st["done"] = 0
        b.step(1)
        st["done"] += 1
        return {f: b.arrays[f] for f in FIELDS[2]}
    if kind == "fresh":
        st["fluid"].set(**st["snapshot"])
        st["particles"].cell_manager.rebuild(check_jump=False)
        st["calc"].sph("rho")
        return st["fluid"].get_device("rho")
    model = st["model"]
    if kind == "closure":
        x = learned.features(st["particles"].cell_manager, st["fluid"], st["norm"])
        return {"features": x, "y": model.forward(x)}
    if kind == "forward":
        return model.forward(st["x"])
    n, a = st["n"], st["next"]
    st["next"] = a + n if a + 2 * n <= st["x"].shape[0] else 0
    x, t = st["x"][a:a + n], st["t"][a:a + n]
    y, cache = model.forward(x, save=True)
    model.backward(x, cache, y, t)
    model.adam(1e-3)
    return {"y": y, "loss": model.loss, "grad": model.grad, "params": model.params,
            "m": model.m, "v": model.v}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

EVALUATIONS = {"euler": 1, "rk2": 2, "pc": 2, "rk4": 4}
NET_FLOPS = 2.0 * (192 * 128 + 128 * 128 + 128 * 2)
# FLOP per neighbour pair of the density and of the rates sums
DENSITY_FLOPS, RATES_FLOPS = 24.0, 72.0


def work(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        n = case["samples"]
        if kind == "forward":
            return {"bytes": n * (384 + 8) + 84e3, "flops": NET_FLOPS * n}
        return {"bytes": n * (384 + 16) + 41474 * 4 * 7, "flops": 3 * NET_FLOPS * n}
    if kind in ("cube", "fresh"):
        n = case["side"] ** 3
        pairs = 4.0 / 3.0 * math.pi * 2.4 ** 3 * n
        if kind == "fresh":
            return {"bytes": 48.0 * n, "flops": DENSITY_FLOPS * pairs}
        return {"bytes": (64 + 72) * n,
                "flops": EVALUATIONS[case["integrator"]] * (DENSITY_FLOPS + RATES_FLOPS) * pairs}
    if kind in ("dam", "closure"):
        n = int(round(2.0 / case["dx"] ** 2))
        pairs = math.pi * 2.4 ** 2 * n
        if kind == "closure":
            return {"bytes": n * (8 * 8 + 384 + 8), "flops": NET_FLOPS * n + 12.0 * pairs}
    elif kind == "batch":
        lay = np.random.default_rng([5, case["layout"]])
        radii = lay.uniform(0.5, 1.5, case["count"])
        dxs = lay.uniform(case["dxmin"], 4.0 * case["dxmin"], case["count"])
        n = float(np.sum(math.pi * radii ** 2 / dxs ** 2))
        pairs = math.pi * 2.6 ** 2 * n
    else:
        n = math.pi / case["dx"] ** 2
        pairs = math.pi * (4.0 if kind == "patch" else 2.6) ** 2 * n
    ev = EVALUATIONS[case["integrator"]]
    return {"bytes": (48 + 56) * n, "flops": ev * (DENSITY_FLOPS + RATES_FLOPS) * pairs}


# ---------------------------------------------------------------------------
# the same results in 64 bits, plain torch
# ---------------------------------------------------------------------------

def _gpu(props):
    return {k: torch.as_tensor(np.asarray(v, np.float64), device="cuda")
            for k, v in props.items()}


def _pairs(d, s, symmetric=False, chunk=1 << 16):
    """Neighbour pairs (i, j) of destinations ``d`` among sources ``s``
    (|r_ij| < 2 h_i; symmetric: or < 2 h_j), chunk by chunk."""
    n = d["x"].numel()
    cell = 2.0 * float(torch.maximum(d["h"].max(), s["h"].max()))
    lo = [float(torch.minimum(d[c].min(), s[c].min())) for c in "xyz"]
    hi = [float(torch.maximum(d[c].max(), s[c].max())) for c in "xyz"]
    dims = [int((b - a) / cell) + 4 for a, b in zip(lo, hi)]

    def key(q, ox=0, oy=0, oz=0):
        c = [((q[k] - a) / cell).floor().long() + 1 for k, a in zip("xyz", lo)]
        return ((c[2] + oz) * dims[1] + c[1] + oy) * dims[0] + c[0] + ox

    skey, order = torch.sort(key(s))
    flat = hi[2] == lo[2]
    rows = [(oy, oz) for oz in ((0,) if flat else (-1, 0, 1)) for oy in (-1, 0, 1)]
    for a in range(0, n, chunk):
        q = {k: d[k][a:a + chunk] for k in ("x", "y", "z", "h")}
        k0 = key(q)
        first, last = [], []
        for oy, oz in rows:
            k = k0 + (oz * dims[1] + oy) * dims[0]
            first.append(torch.searchsorted(skey, k - 1))
            last.append(torch.searchsorted(skey, k + 1, right=True))
        first = torch.stack(first, 1).reshape(-1)
        count = torch.stack(last, 1).reshape(-1) - first
        ends = count.cumsum(0)
        row = torch.repeat_interleave(torch.arange(count.numel(), device="cuda"), count)
        j = order[torch.arange(row.numel(), device="cuda") - (ends - count)[row] + first[row]]
        i = row // len(rows)
        r2 = sum((q[c][i] - s[c][j]) ** 2 for c in "xyz")
        hit = r2 < (2.0 * q["h"][i]) ** 2
        if symmetric:
            hit |= r2 < (2.0 * s["h"][j]) ** 2
        yield i[hit] + a, j[hit]


def _spline(r, h, dim):
    """W and (dW/dr)/r of the cubic spline."""
    fac = {2: 10.0 / (7.0 * math.pi), 3: 1.0 / math.pi}[dim] / h ** dim
    q = r / h
    near = q < 1.0
    two = (2.0 - q).clamp(min=0.0)
    w = torch.where(near, 1.0 - 1.5 * q * q * (1.0 - 0.5 * q), 0.25 * two ** 3)
    g = torch.where(near, 3.0 * (0.75 * q - 1.0) / (h * h),
                    -0.75 * two ** 2 / (h * r.clamp(min=1e-300)))
    g = torch.where(q > 1e-14, g, torch.zeros_like(g))
    return w * fac, g * fac


def _density(a, dim, symmetric):
    rho = torch.zeros_like(a["x"])
    for i, j in _pairs(a, a, symmetric):
        r = sum((a[c][i] - a[c][j]) ** 2 for c in "xyz").sqrt()
        w, _ = _spline(r, 0.5 * (a["h"][i] + a["h"][j]), dim)
        rho.index_add_(0, i, a["m"][j] * w)
    return rho


def _tait(a, c0, rho0):
    ratio = a["rho"] / rho0
    a["p"] = c0 * c0 * rho0 / 7.0 * (ratio ** 7 - 1.0)
    a["cs"] = c0 * ratio ** 3


def _rates(a, dim, alpha, eta=0.0, eps=0.0, drho=False, symmetric=False):
    """Accelerations, XSPH-corrected velocities (and the density rate)."""
    k = {c: torch.zeros_like(a["x"]) for c in ("u", "v", "w", "rho")}
    k.update({c: a[v].clone() for c, v in zip("xyz", "uvw")})
    for i, j in _pairs(a, a, symmetric):
        r = [a[c][i] - a[c][j] for c in "xyz"]
        v = [a[c][i] - a[c][j] for c in "uvw"]
        r2 = sum(c * c for c in r)
        h = 0.5 * (a["h"][i] + a["h"][j])
        w, g = _spline(r2.sqrt(), h, dim)
        m = a["m"][j]
        dot = sum(x * y for x, y in zip(r, v))
        rho = 0.5 * (a["rho"][i] + a["rho"][j])
        mu = h * dot.clamp(max=0.0) / torch.where(dot < 0, r2 + eta * eta * h * h,
                                                  torch.ones_like(r2))
        visc = -alpha * 0.5 * (a["cs"][i] + a["cs"][j]) * mu / rho
        f = -m * g * (a["p"][i] / a["rho"][i] ** 2 + a["p"][j] / a["rho"][j] ** 2 + visc)
        for c, rc in zip("uvw", r):
            k[c].index_add_(0, i, f * rc)
        if eps:
            for c, vc in zip("xyz", v):
                k[c].index_add_(0, i, -eps * m * w / rho * vc)
        if drho:
            k["rho"].index_add_(0, i, m * g * dot)
    return k


def _boundary(a, b, dx, k):
    for i, j in _pairs(a, b):
        r = [a[c][i] - b[c][j] for c in "xy"]
        x = (r[0] * b["tx"][j] + r[1] * b["ty"][j]).abs()
        y = r[0] * b["nx"][j] + r[1] * b["ny"][j]
        q = y / a["h"][i]
        n = torch.where(q <= 2.0 / 3.0, torch.full_like(q, 2.0 / 3.0),
                        torch.where(q <= 1.0, 2.0 * q * (1.0 - 0.75 * q), 0.5 * (2.0 - q) ** 2))
        on = (q > 0.0) & (q <= 2.0) & (x <= dx)
        ma, mb = a["m"][i], b["m"][j]
        f = mb / (ma + mb) * n * (1.0 - x / dx) * 0.02 * a["cs"][i] ** 2 / torch.where(
            on, y, torch.ones_like(y))
        f = torch.where(on, f, torch.zeros_like(f))
        k["u"].index_add_(0, i, f * b["nx"][j])
        k["v"].index_add_(0, i, f * b["ny"][j])


def _evaluate(case, a, wall):
    kind = case["kind"]
    sym = bool(case.get("variable_h", False))
    if kind in ("cube", "drop", "batch"):
        dim = 3 if kind == "cube" else 2
        a["rho"] = _density(a, dim, sym)
        _tait(a, 1.0 if kind == "cube" else 100.0, 1.0)
        if kind == "cube":
            return _rates(a, 3, 0.1)
        return _rates(a, 2, 0.01, eps=0.5, symmetric=sym)
    if kind == "patch":
        _tait(a, 100.0, 1.0)
        return _rates(a, 2, 0.01, eta=0.1, eps=0.1, drho=True)
    _tait(a, DAM_C0, DAM_RHO0)
    a["rho"] = _density(a, 2, False)
    k = _rates(a, 2, 0.1)
    _boundary(a, wall, case["dx"], k)
    k["v"] += GRAVITY
    return k


def _step(case, props, wall, dt):
    a = _gpu(props)
    n = a["x"].numel()
    for c in "zuvwp":
        a.setdefault(c, torch.zeros(n, dtype=torch.float64, device="cuda"))
    b = None if wall is None else _gpu(wall)
    if b is not None:
        b["z"] = torch.zeros_like(b["x"])
    moved = ("x", "y", "z", "u", "v", "w") + (("rho",) if case["kind"] == "patch" else ())
    x0 = {c: a[c].clone() for c in moved}

    def to(k, f):
        for c in moved:
            a[c] = x0[c] + f * k[c]

    k1 = _evaluate(case, a, b)
    how = case["integrator"]
    if how == "euler":
        to(k1, dt)
    elif how == "rk2":
        to(k1, dt)
        k2 = _evaluate(case, a, b)
        to({c: k1[c] + k2[c] for c in moved}, 0.5 * dt)
    elif how == "pc":
        to(k1, 0.5 * dt)
        to(_evaluate(case, a, b), dt)
    else:
        to(k1, 0.5 * dt)
        k2 = _evaluate(case, a, b)
        to(k2, 0.5 * dt)
        k3 = _evaluate(case, a, b)
        to(k3, dt)
        k4 = _evaluate(case, a, b)
        to({c: k1[c] + 2.0 * k2[c] + 2.0 * k3[c] + k4[c] for c in moved}, dt / 6.0)
    return a


def _nearest(a, mean, std):
    """Standardised features: the 32 nearest neighbours in 2D."""
    n = a["x"].numel()
    out = torch.zeros((n, 32, 6), dtype=torch.float64, device="cuda")
    mean = torch.tensor(mean, dtype=torch.float64, device="cuda")
    std = torch.tensor(std, dtype=torch.float64, device="cuda")
    for i, j in _pairs(a, a):
        r2 = (a["x"][i] - a["x"][j]) ** 2 + (a["y"][i] - a["y"][j]) ** 2
        o = torch.sort(r2, stable=True)[1]
        o = o[torch.sort(i[o], stable=True)[1]]
        i, j = i[o], j[o]
        base = int(i[0])
        count = torch.bincount(i - base)
        rank = torch.arange(i.numel(), device="cuda") - (count.cumsum(0) - count)[i - base]
        near = rank < 32
        i, j, rank = i[near], j[near], rank[near]
        h = a["h"][i]
        raw = torch.stack([(a["x"][i] - a["x"][j]) / h, (a["y"][i] - a["y"][j]) / h,
                           (a["u"][j] - a["u"][i]) / DAM_C0, (a["v"][j] - a["v"][i]) / DAM_C0,
                           a["rho"][j], a["p"][j]], 1)
        out[i, rank] = (raw - mean) / std
    return out.view(n, 192)


def _weights(params):
    p = torch.as_tensor(params, device="cuda").double()
    o = np.cumsum([0, 128 * 192, 128, 128 * 128, 128, 256, 2])
    w1, b1, w2, b2, w3, b3 = (p[a:b] for a, b in zip(o[:-1], o[1:]))
    return w1.view(128, 192), b1, w2.view(128, 128), b2, w3.view(2, 128), b3


def _network(x, weights):
    w1, b1, w2, b2, w3, b3 = weights
    act = torch.nn.functional.gelu
    h = act(x @ w1.T + b1, approximate="tanh")
    return act(h @ w2.T + b2, approximate="tanh") @ w3.T + b3


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cube", "drop", "patch", "dam"):
        wall = None
        if kind == "cube":
            props = _cube_props(case, seed)
        elif kind == "drop":
            props = _drop_props(1.0, case["dx"], np.random.default_rng([2, seed]),
                                case["variable_h"])
        elif kind == "patch":
            props = _patch_props(case, seed)
        else:
            props, wall = _dam_props(case, seed)
        a = _step(case, props, wall, _time_step(case))
        return {f: a[f] for f in FIELDS[3 if kind == "cube" else 2]}
    if kind == "batch":
        each = [_step(case, p, None, 1e-5) for p in _batch_props(case, seed)]
        return {f: torch.cat([a[f] for a in each]) for f in FIELDS[2]}
    if kind == "fresh":
        return _density(_gpu(_cube_props(case, seed)), 3, False)
    weights = _weights(_net_params(seed))
    if kind == "closure":
        a = _gpu(_closure_props(case, seed)[0])
        a["z"] = torch.zeros_like(a["x"])
        x = _nearest(a, *_closure_scaling())
        return {"features": x, "y": _network(x, weights)}
    n = case["samples"]
    if kind == "forward":
        x, _ = _samples(n, 1, seed)
        return torch.cat([_network(c.double(), weights) for c in x.split(1 << 17)])
    x, t = _samples(n, _minibatches(n), seed)
    x, t = x[:n].double(), t[:n].double()
    weights = [w.requires_grad_() for w in weights]
    y = _network(x, weights)
    loss = 0.5 / n * ((y - t) ** 2).sum()
    grad = torch.cat([g.reshape(-1) for g in torch.autograd.grad(loss, weights)])
    p = torch.cat([w.detach().reshape(-1) for w in weights])
    m, v = 0.1 * grad, 0.001 * grad * grad
    p = p - 1e-3 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
    return {"y": y.detach(), "loss": loss.detach().reshape(1), "grad": grad, "params": p,
            "m": m, "v": v}
