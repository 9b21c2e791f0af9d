"""The brick-staged pair passes against the list-streaming ones and the oracle.

With one source of uniform h, ``sph_density`` (SPHRho + Tait) and
``sph_rates`` (PGrad + Monaghan AV, + XSPH) stage each brick of cells'
neighbour records in shared memory and stream 16-bit lists into that
staging.  The same step must match the list-streaming kernels
(``PYSPH_GB300_BRICKS=0``) within FP32 rounding and the FP64 oracle within
the 1e-5 normwise tolerance of every step-parity test, for every cell
subdivision, in 2D and 3D, with non-real destinations, and on the paths for
over-full lists and for bricks whose sources are read from global memory.
"""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import oracle
import pysph_gb300
from golden_util import normwise, rel_percentiles
from pysph_gb300 import workloads as W

pytestmark = pytest.mark.gpu

API = pysph_gb300.api()
TOL = 1e-5          # normwise, against the FP64 oracle
SAME = 5e-6         # normwise, brick-staged against list-streaming kernels (FP32
                    # rounding; Tait amplifies that of rho about 7-fold in p)
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def _cube_step(props, bricks, monkeypatch, steps=1, dt=1e-4):
    monkeypatch.setenv("PYSPH_GB300_BRICKS", "1" if bricks else "0")
    s, particles = W.setup_cube(API, props)
    for _ in range(steps):
        s.integrator.integrate(dt)
    pa = particles.arrays[0]
    out = {p: pa.get(p) for p in ("x", "y", "z", "u", "v", "w", "rho", "p", "cs")}
    return out, particles.cell_manager.brick_pass_count()


@pytest.mark.parametrize("n,subdiv", [(32768, 1), (32768, 2), (64000, 3)])
def test_cube_step_bricks_match_lists_and_oracle(n, subdiv, monkeypatch):
    _need_gpu()
    monkeypatch.setenv("PYSPH_GB300_SUBDIV", str(subdiv))
    props = W.cube_lattice(n, seed=21)
    got, nb = _cube_step(props, True, monkeypatch)
    ref_list, nl = _cube_step(props, False, monkeypatch)
    assert nb == 4 and nl == 0          # 2 density + 2 rates passes per RK2 step
    prob = oracle.Problem({"fluid": props}, oracle.cube_ops(), dim=3)
    prob.integrate_rk2(1e-4)
    ref = prob.arrays["fluid"]
    for p in ("rho", "p", "cs"):
        assert normwise(got[p], ref_list[p]) < SAME, p
        assert normwise(got[p], ref[p]) < TOL, p
    for p in ("x", "y", "z", "u", "v", "w"):
        assert normwise(got[p] - props[p], ref_list[p] - props[p]) < SAME, p
        assert normwise(got[p] - props[p], ref[p] - props[p]) < TOL, p
    p50, p99, mx, cnt = rel_percentiles(got["rho"], ref["rho"])
    print("rho per-particle relative error p50 %.2e p99 %.2e max %.2e over %d" % (p50, p99, mx, cnt))
    assert mx < 1e-5


def test_drop_euler_step_with_xsph(monkeypatch):
    """2D: PGrad + AV + XSPH in one brick-staged rates pass (the drop)."""
    _need_gpu()
    props = W.elliptical_drop(dx=0.0125, c0=100.0)
    outs = {}
    for bricks in (True, False):
        monkeypatch.setenv("PYSPH_GB300_BRICKS", "1" if bricks else "0")
        s, particles = W.setup_drop(API, props, c0=100.0)
        s.integrator.integrate(1e-5)
        pa = particles.arrays[0]
        outs[bricks] = {p: pa.get(p) for p in ("x", "y", "u", "v", "rho", "p")}
        assert (particles.cell_manager.brick_pass_count() > 0) == bricks
    prob = oracle.Problem({"fluid": props}, oracle.drop_ops(c0=100.0), dim=2)
    prob.integrate_euler(1e-5)
    ref = prob.arrays["fluid"]
    for p in ("rho", "p"):
        assert normwise(outs[True][p], outs[False][p]) < SAME, p
        assert normwise(outs[True][p], ref[p]) < TOL, p
    for p in ("x", "y", "u", "v"):
        assert normwise(outs[True][p] - props[p], outs[False][p] - props[p]) < SAME, p
        assert normwise(outs[True][p] - props[p], ref[p] - props[p]) < TOL, p


def test_cube_step_mixed_masses(monkeypatch):
    """A block whose sources share one mass reads two records per pair in
    the rates pass (cs from rho through Tait), any other block three.  Masses
    2 % heavier in one corner of the cube mix both kinds of block in one
    pass: the step matches the list-streaming kernels and the oracle."""
    _need_gpu()
    props = W.cube_lattice(32768, seed=25)
    corner = (props["x"] < 0.3) & (props["y"] < 0.3)
    props["m"] = np.where(corner, 1.02 * props["m"], props["m"])
    got, nb = _cube_step(props, True, monkeypatch)
    ref_list, _ = _cube_step(props, False, monkeypatch)
    assert nb == 4
    prob = oracle.Problem({"fluid": props}, oracle.cube_ops(), dim=3)
    prob.integrate_rk2(1e-4)
    ref = prob.arrays["fluid"]
    for p in ("rho", "p", "cs"):
        assert normwise(got[p], ref_list[p]) < SAME, p
        assert normwise(got[p], ref[p]) < TOL, p
    for p in ("x", "y", "z", "u", "v", "w"):
        assert normwise(got[p] - props[p], ref_list[p] - props[p]) < SAME, p
        assert normwise(got[p] - props[p], ref[p] - props[p]) < TOL, p


def test_light_refresh_trajectory_matches_list_kernels(monkeypatch):
    """Twenty RK2 steps with the list skin (light refreshes between full
    builds): the brick-staged and list-streaming trajectories agree."""
    _need_gpu()
    props = W.cube_lattice(32768, seed=22)
    a, _ = _cube_step(props, True, monkeypatch, steps=20)
    b, _ = _cube_step(props, False, monkeypatch, steps=20)
    for p in ("rho", "p"):
        assert normwise(a[p], b[p]) < 1e-5, p
    for p in ("x", "y", "z", "u", "v", "w"):
        assert normwise(a[p] - props[p], b[p] - props[p]) < 1e-5, p


def test_non_real_destinations_get_zero_in_bricks(monkeypatch):
    _need_gpu()
    monkeypatch.setenv("PYSPH_GB300_BRICKS", "1")
    base, sph = API.base, API.sph
    props = W.cube_lattice(8000, seed=23)
    n = len(props["x"])
    tag = np.zeros(n, np.int64)
    tag[::5] = 1
    pa = base.get_particle_array(name="fluid", **props)
    pa.add_property({"name": "tag", "data": tag, "type": "long"})
    pa.align_particles()
    particles = base.Particles(arrays=[pa])
    k3 = base.CubicSplineKernel(dim=3)
    sph.SPHCalc(particles, [pa], pa, k3, [sph.SPHRho.get_func(pa, pa)], ["rho"]).sph("rho")
    assert particles.cell_manager.brick_pass_count() == 1
    rho = pa.get("rho", only_real_particles=False)
    t = pa.get("tag", only_real_particles=False)
    assert np.all(rho[t != 0] == 0)
    host = {k: pa.get(k, only_real_particles=False) for k in ("x", "y", "z", "h", "m")}
    host["tag"] = t
    off, idx = oracle.neighbors(host, host, particles.cell_manager.cell_size, same=True)
    ref = oracle.pair_sum("rho", host, host, off, idx, 3)[0]
    assert normwise(rho, ref) < TOL


_SUB = r'''
import sys
sys.path.insert(0, ".")
import oracle, pysph_gb300
from pysph_gb300 import workloads as W
from tests.golden_util import normwise
api = pysph_gb300.api()
props = W.cube_lattice(32768, seed=24)
s, particles = W.setup_cube(api, props)
s.integrator.integrate(1e-4)
assert particles.cell_manager.brick_pass_count() >= 4
pa = particles.arrays[0]
prob = oracle.Problem({"fluid": props}, oracle.cube_ops(), dim=3)
prob.integrate_rk2(1e-4)
for p in ("rho", "p"):
    assert normwise(pa.get(p), prob.arrays["fluid"][p]) < 1e-5, p
for p in ("x", "u", "w"):
    assert normwise(pa.get(p) - props[p], prob.arrays["fluid"][p] - props[p]) < 1e-5, p
props = W.elliptical_drop(dx=0.025, c0=100.0)
s, particles = W.setup_drop(api, props, c0=100.0)
s.integrator.integrate(1e-5)
assert particles.cell_manager.brick_pass_count() > 0
pa = particles.arrays[0]
prob = oracle.Problem({"fluid": props}, oracle.drop_ops(c0=100.0), dim=2)
prob.integrate_euler(1e-5)
for p in ("rho", "p"):
    assert normwise(pa.get(p), prob.arrays["fluid"][p]) < 1e-5, p
for p in ("x", "y", "u", "v"):
    assert normwise(pa.get(p) - props[p], prob.arrays["fluid"][p] - props[p]) < 1e-5, p
print("ok")
'''


@pytest.mark.parametrize("env", [{"SPH_BRICK_UNSTAGED": "1"}, {"SPH_LIST_CAP": "9"},
                                 {"SPH_BRICK_UNSTAGED": "1", "SPH_LIST_CAP": "9"},
                                 {"SPH_BRICK_TWO_RECORDS": "0"}],
                         ids=["global-records", "over-full-lists", "both", "three-records"])
def test_brick_fallback_paths_match_oracle(env):
    """Records read from global memory (bricks too populous for shared
    memory), lists shorter than the neighbour counts (completed by
    re-traversal) and the rates pass's three records per pair in every
    block, forced on small sets in a fresh process."""
    _need_gpu()
    e = dict(os.environ, PYSPH_GB300_BRICKS="1", **env)
    r = subprocess.run([sys.executable, "-c", _SUB], cwd=ROOT, env=e, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-3000:]


_HASH = r'''
import sys, hashlib
sys.path.insert(0, ".")
import pysph_gb300
from pysph_gb300 import workloads as W
api = pysph_gb300.api()
h = hashlib.sha256()
def add(particles, names):
    for a in particles.arrays:
        for f in names:
            h.update(a.get(f).tobytes())
for n in (343, 4096, 32768):
    s, particles = W.setup_cube(api, W.cube_lattice(n, seed=31))
    for _ in range(3):
        s.integrator.integrate(1e-4)
    assert particles.cell_manager.brick_pass_count() > 0
    add(particles, ("x", "y", "z", "u", "v", "w", "rho", "p", "cs"))
for dx in (0.2, 0.03):
    s, particles = W.setup_drop(api, W.elliptical_drop(dx=dx, c0=100.0), c0=100.0)
    for _ in range(4):
        s.integrator.integrate(1e-5)
    add(particles, ("x", "y", "u", "v", "rho", "p", "cs"))
print(h.hexdigest())
'''


@pytest.mark.parametrize("subdiv", [1, 2, 3])
def test_lanes_and_rounds_give_the_same_bits(subdiv):
    """One, two or four threads per destination, and destinations past a
    block's threads (64 threads per block), fold the same batches in the same
    order: the steps agree bit for bit."""
    _need_gpu()
    seen = set()
    for env in ({"SPH_BRICK_LANES": "1"}, {"SPH_BRICK_LANES": "2"}, {"SPH_BRICK_LANES": "4"},
                {"SPH_BRICK_LANES": "1", "SPH_BRICK_MAX_THREADS": "64"}):
        e = dict(os.environ, PYSPH_GB300_BRICKS="1", PYSPH_GB300_SUBDIV=str(subdiv), **env)
        r = subprocess.run([sys.executable, "-c", _HASH], cwd=ROOT, env=e, capture_output=True,
                           text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1


_HASH_LISTS = r'''
import sys, hashlib
sys.path.insert(0, ".")
import numpy as np, pysph_gb300
from pysph_gb300 import workloads as W
api = pysph_gb300.api()
h = hashlib.sha256()
def run(s, particles, dt, names, steps=3):
    for _ in range(steps):
        s.integrator.integrate(dt)
    for a in particles.arrays:
        for f in names:
            h.update((a.get(f) + 0.0).tobytes())
names = ("x", "y", "u", "v", "w", "rho", "p", "cs")
for dx in (0.5, 0.04):
    drop = W.elliptical_drop(dx=dx, c0=100.0)
    run(*W.setup_drop(api, W.jitter_h(drop), c0=100.0, variable_h=True), 1e-5, names)
    run(*W.setup_fluid_solver(api, W.circular_patch(dx=dx)), 1e-5, names)
strip = W.periodic_strip(dx=0.05, nx=31, ny=7, jitter=0.1)
run(*W.setup_drop(api, strip, c0=10.0, periodic_domain=api.base.PeriodicDomain(0.0, 1.55)), 1e-4,
    names)
fluid, wall = W.dam_break(dx=0.04)
rng = np.random.default_rng(3)
fluid["u"], fluid["v"] = rng.normal(0, 1, (2, fluid["x"].size))
run(*W.setup_dam_break(api, fluid, wall, 0.04, W.dam_break_c0()), 2.5e-5, names)
print(h.hexdigest())
'''


@pytest.mark.parametrize("cap", ["", "9"], ids=["lists", "over-full-lists"])
def test_list_rates_lanes_give_the_same_bits(cap):
    """One, two or eight threads per destination of the list-streaming rates
    pass fold the same batches in the same order: variable-h, periodic,
    continuity and boundary-force steps agree bit for bit, also where lists
    overflow and the rest comes from a traversal."""
    _need_gpu()
    seen = set()
    for lanes in ("1", "2", "8"):
        e = dict(os.environ, SPH_PAIR_LANES=lanes)
        if cap:
            e["SPH_LIST_CAP"] = cap
        r = subprocess.run([sys.executable, "-c", _HASH_LISTS], cwd=ROOT, env=e,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1

@pytest.mark.parametrize("cap", ["", "9"], ids=["lists", "over-full-lists"])
def test_four_list_lanes_give_the_same_bits(cap):
    """Four threads per destination of the list builds and the rates pass:
    the bits of one."""
    _need_gpu()
    seen = set()
    for lanes in ("1", "4"):
        e = dict(os.environ, SPH_PAIR_LANES=lanes)
        if cap:
            e["SPH_LIST_CAP"] = cap
        r = subprocess.run([sys.executable, "-c", _HASH_LISTS], cwd=ROOT, env=e,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1


@pytest.mark.parametrize("n", [65534, 65535, 70001])
def test_crowded_destination_with_a_sparse_source(n, monkeypatch):
    """Sample points so many that no block could stage them (65 535 and more
    around one brick) among the particles of another, sparse array: their
    blocks' destinations are those of the build, first and after a move that
    crowds them.  Density and momentum rates against the oracle."""
    _need_gpu()
    monkeypatch.setenv("PYSPH_GB300_BRICKS", "1")
    base, sph = API.base, API.sph
    rng = np.random.default_rng(n)
    h, m = 0.05, 400

    def state(k, x, y):
        return dict(x=x, y=y, u=rng.normal(0, 1, k), v=rng.normal(0, 1, k),
                    m=rng.uniform(0.5, 1.5, k), h=np.full(k, h), rho=rng.uniform(1.0, 2.0, k),
                    p=rng.uniform(1.0, 2.0, k), cs=rng.uniform(1.0, 2.0, k), ax=np.zeros(k),
                    ay=np.zeros(k))

    sp = state(m, rng.uniform(0, 0.3, m), rng.uniform(0, 0.3, m))
    dp = state(n, rng.uniform(0, 4.0, n), rng.uniform(0, 4.0, n))
    src = base.get_particle_array(name="fluid", **sp)
    dst = base.get_particle_array(name="samples", **dp)
    particles = base.Particles(arrays=[src, dst])
    cm = particles.cell_manager
    kern = base.CubicSplineKernel(dim=2)
    for crowded in (False, True):
        if crowded:
            dp["x"], dp["y"] = 0.075 * dp["x"], 0.075 * dp["y"]
            dst.set(x=dp["x"], y=dp["y"])
            cm.rebuild(check_jump=False)
        passes = cm.brick_pass_count()
        sph.SPHCalc(particles, [src], dst, kern, [sph.SPHRho.get_func(src, dst)], ["rho"]).sph("rho")
        got = dst.get("rho")
        dst.set(rho=dp["rho"])
        mom = sph.MomentumEquation.withargs(alpha=0.5, beta=0.5, dim=2)
        sph.SPHCalc(particles, [src], dst, kern, [mom.get_func(src, dst)], ["ax", "ay"]).sph("ax", "ay")
        assert cm.brick_pass_count() == passes + 2
        off, idx = oracle.neighbors(dp, sp, 2.0 * h)
        assert normwise(got, oracle.pair_sum("rho", dp, sp, off, idx, 2, nout=1)[0]) < TOL
        ax, ay = oracle.pair_sum("momentum", dp, sp, off, idx, 2,
                                 dict(alpha=0.5, beta=0.5, eta=0.1), nout=2)[:2]
        assert normwise(dst.get("ax"), ax) < TOL and normwise(dst.get("ay"), ay) < TOL


_HASH_MASSES = r'''
import sys, hashlib
sys.path.insert(0, ".")
import numpy as np, pysph_gb300
from pysph_gb300 import workloads as W
api = pysph_gb300.api()
h = hashlib.sha256()
def run(s, particles, dt, names):
    for _ in range(3):
        s.integrator.integrate(dt)
    assert particles.cell_manager.brick_pass_count() > 0
    for f in names:
        h.update(particles.arrays[0].get(f).tobytes())
for n in (1000, 13824):
    props = W.cube_lattice(n, seed=41)
    run(*W.setup_cube(api, props), 1e-4, ("x", "y", "z", "u", "v", "w", "rho", "p", "cs"))
    props["m"] = np.where(props["x"] < 0.3, 1.02 * props["m"], props["m"])
    run(*W.setup_cube(api, props), 1e-4, ("x", "y", "z", "u", "v", "w", "rho", "p", "cs"))
drop = W.elliptical_drop(dx=0.03, c0=100.0)
run(*W.setup_drop(api, drop, c0=100.0), 1e-5, ("x", "y", "u", "v", "rho", "p", "cs"))
print(h.hexdigest())
'''


def _hash_masses(**env):
    e = dict(os.environ, PYSPH_GB300_BRICKS="1", **env)
    r = subprocess.run([sys.executable, "-c", _HASH_MASSES], cwd=ROOT, env=e, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return r.stdout.split()[-1]


@pytest.mark.parametrize("env", [{}, {"PYSPH_GB300_SKIN": "0"}, {"SPH_LIST_CAP": "9"},
                                 {"SPH_BRICK_UNSTAGED": "1"},
                                 {"SPH_BRICK_UNSTAGED": "1", "SPH_LIST_CAP": "9",
                                  "PYSPH_GB300_SKIN": "0"}],
                         ids=["staged", "no-skin", "over-full", "global-records", "all"])
def test_records_found_from_rows_give_the_same_bits(env):
    """A build without the table of staged entries (too many of them, or no
    memory for it) finds every record from the rows of cells: the same bits,
    with one mass and with two, in 3D and 2D."""
    _need_gpu()
    rows = _hash_masses(SPH_BRICK_STAGE_TABLE="0", **env)
    assert rows == _hash_masses(**env)


def _with_far_particles(props, far):
    """Four particles of a 2D set moved far out, one to each quadrant."""
    out = {k: v.copy() for k, v in props.items()}
    for j, (sx, sy) in enumerate(((1, 1), (-1, 1), (1, -1), (-1, -1))):
        out["x"][7 * j], out["y"][7 * j] = sx * far * (1 + 0.01 * j), sy * far * (1 + 0.01 * j)
        out["u"][7 * j] = out["v"][7 * j] = 0.0
    return out


def _best_us(f, passes=20, rounds=8):
    import time
    f()
    best = float("inf")
    for _ in range(rounds):
        torch.cuda.synchronize()
        t = time.perf_counter()
        for _ in range(passes):
            f()
        torch.cuda.synchronize()
        best = min(best, (time.perf_counter() - t) / passes * 1e6)
    return best


def test_a_box_of_empty_bricks(monkeypatch):
    """Four particles far from a drop make a box of 43 000 bricks, nearly all
    empty: the step is the oracle's, and the empty bricks cost less than the
    rest of it (a build under three times, a step under four times that of the
    drop by itself)."""
    _need_gpu()
    monkeypatch.setenv("PYSPH_GB300_BRICKS", "1")
    drop = W.elliptical_drop(dx=0.025, c0=100.0)
    build, step = [], []
    for props in (drop, _with_far_particles(drop, 40.0)):
        s, particles = W.setup_drop(API, props, c0=100.0)
        s.integrator.integrate(1e-6)
        assert particles.cell_manager.brick_pass_count() > 0
        pa = particles.arrays[0]
        prob = oracle.Problem({"fluid": props}, oracle.drop_ops(c0=100.0), dim=2)
        prob.integrate_euler(1e-6)
        ref = prob.arrays["fluid"]
        for p in ("rho", "p"):
            assert normwise(pa.get(p), ref[p]) < TOL, p
        for p in ("u", "v"):
            assert normwise(pa.get(p) - props[p], ref[p] - props[p]) < TOL, p
        step.append(_best_us(lambda: s.integrator.integrate(1e-7)))
        build.append(_best_us(lambda: particles.cell_manager.rebuild(check_jump=False)))
    print("build us %s, step us %s" % (build, step))
    assert build[1] < 3.0 * build[0]
    assert step[1] < 4.0 * step[0]


_HASH_WIDE = r'''
import sys, hashlib
sys.path.insert(0, ".")
import pysph_gb300
from pysph_gb300 import workloads as W
api = pysph_gb300.api()
h = hashlib.sha256()
def run(s, particles, dt, names):
    for _ in range(2):
        s.integrator.integrate(dt)
    particles.cell_manager.rebuild(check_jump=False)
    s.integrator.integrate(dt)
    assert particles.cell_manager.brick_pass_count() > 0
    for f in names:
        h.update(particles.arrays[0].get(f).tobytes())
for hdx in (1.7, 2.2, 4.0):
    run(*W.setup_drop(api, W.elliptical_drop(dx=0.02, hdx=hdx, c0=100.0), c0=100.0), 1e-6,
        ("x", "y", "u", "v", "rho", "p", "cs"))
run(*W.setup_cube(api, W.cube_lattice(8000, hdx=2.0, seed=5)), 1e-5,
    ("x", "y", "z", "u", "v", "w", "rho", "p", "cs"))
print(h.hexdigest())
'''


_ONE = {"SPH_BRICK_LANES": "1"}


@pytest.mark.parametrize("records,envs", [
    ("1", [_ONE, dict(_ONE, SPH_BRICK_MAX_THREADS="64"), dict(_ONE, SPH_BRICK_MAX_THREADS="512")]),
    ("0", [{}, _ONE, dict(_ONE, SPH_BRICK_MAX_THREADS="64"),
           dict(_ONE, SPH_BRICK_MAX_THREADS="512"), {"SPH_BRICK_LANES": "2"}])],
    ids=["threads", "threads-and-lanes"])
def test_wide_supports_give_the_same_bits(records, envs):
    """Bricks with more destinations than the block has threads -- a few more,
    and several times as many -- in rounds of a thread each and of four lanes:
    the same bits whatever the block's threads, and its lanes (with three
    records per pair: a part of a brick can be small enough to stage, and so
    read two, where the brick is not)."""
    _need_gpu()
    seen = set()
    for env in envs:
        e = dict(os.environ, PYSPH_GB300_BRICKS="1", SPH_BRICK_TWO_RECORDS=records, **env)
        r = subprocess.run([sys.executable, "-c", _HASH_WIDE], cwd=ROOT, env=e,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1


_HASH_1D = r'''
import sys, hashlib
sys.path.insert(0, ".")
import numpy as np, pysph_gb300
api = pysph_gb300.api()
base, sph, solver = api.base, api.sph, api.solver
Fluid = base.ParticleType.Fluid
h = hashlib.sha256()
for n, hdx in ((1, 1.2), (50, 1.2), (700, 2.0), (4000, 3.0)):
    x = (np.arange(n) + 0.5) / n
    pa = base.get_particle_array(name="gas", type=Fluid, x=x, m=np.full(n, 1.0 / n),
                                 h=np.full(n, hdx / n), rho=np.ones(n), u=0.1 * np.sin(20 * x),
                                 cs=np.ones(n))
    particles = base.Particles(arrays=[pa])
    s = solver.Solver(dim=1, integrator_type=solver.RK2Integrator)
    s.add_operation(solver.SPHOperation(sph.SPHRho.withargs(), on_types=[Fluid],
                                        from_types=[Fluid], updates=["rho"], id="density"))
    s.add_operation(solver.SPHOperation(sph.TaitEquation.withargs(co=1.0, ro=1.0),
                                        on_types=[Fluid], updates=["p", "cs"], id="eos"))
    s.add_operation(solver.SPHIntegration(sph.SPHPressureGradient.withargs(dim=1),
                                          on_types=[Fluid], from_types=[Fluid], updates=["u"],
                                          id="pgrad"))
    s.add_operation(solver.SPHIntegration(
        sph.MonaghanArtificialVsicosity.withargs(alpha=0.1, beta=0.0), on_types=[Fluid],
        from_types=[Fluid], updates=["u", "v", "w"], id="avisc"))
    s.add_operation_step([Fluid])
    s.setup_integrator(particles)
    for _ in range(4):
        s.integrator.integrate(0.05 / n)
    assert particles.cell_manager.brick_pass_count() > 0
    for f in ("x", "u", "rho", "p", "cs"):
        h.update(pa.get(f).tobytes())
print(h.hexdigest())
'''


def test_lanes_in_1d_give_the_same_bits():
    """1D sets, of one particle upwards: as they come, and with one, two and
    four threads per destination."""
    _need_gpu()
    seen = set()
    for env in ({}, {"SPH_BRICK_LANES": "1"}, {"SPH_BRICK_LANES": "2"}, {"SPH_BRICK_LANES": "4"}):
        e = dict(os.environ, PYSPH_GB300_BRICKS="1", **env)
        r = subprocess.run([sys.executable, "-c", _HASH_1D], cwd=ROOT, env=e,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1


@pytest.mark.parametrize("env", [{"SPH_BRICK_UNSTAGED": "1"}, {"SPH_LIST_CAP": "9"},
                                 {"SPH_BRICK_UNSTAGED": "1", "SPH_LIST_CAP": "9"},
                                 {"SPH_BRICK_TWO_RECORDS": "0"}],
                         ids=["global-records", "over-full-lists", "both", "three-records"])
def test_one_lane_fallback_paths_match_oracle(env):
    """The fallback paths with a thread per destination, which larger sets
    have (these small ones would get two and four)."""
    _need_gpu()
    e = dict(os.environ, PYSPH_GB300_BRICKS="1", SPH_BRICK_LANES="1", **env)
    r = subprocess.run([sys.executable, "-c", _SUB], cwd=ROOT, env=e, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-3000:]


@pytest.mark.parametrize("env", [{"SPH_LIST_CAP": "9"}, {"SPH_BRICK_UNSTAGED": "1"},
                                 {"SPH_LIST_CAP": "9", "SPH_BRICK_UNSTAGED": "1"}],
                         ids=["over-full-lists", "global-records", "both"])
def test_lanes_give_the_same_bits_on_fallback_paths(env):
    """One, two or four threads per destination agree bit for bit where lists
    overflow and where records are read from global memory."""
    _need_gpu()
    seen = set()
    for lanes in ("1", "2", "4"):
        e = dict(os.environ, PYSPH_GB300_BRICKS="1", SPH_BRICK_LANES=lanes, **env)
        r = subprocess.run([sys.executable, "-c", _HASH], cwd=ROOT, env=e, capture_output=True,
                           text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1


_HASH_LISTS_3D = r'''
import sys, hashlib
sys.path.insert(0, ".")
import numpy as np, pysph_gb300
from pysph_gb300 import workloads as W
api = pysph_gb300.api()
base, sph, solver = api.base, api.sph, api.solver
Fluid = base.ParticleType.Fluid
h = hashlib.sha256()
def run(s, particles, dt, names):
    for _ in range(2):
        s.integrator.integrate(dt)
    for a in particles.arrays:
        for f in names:
            h.update((a.get(f) + 0.0).tobytes())
def cube(props, split, variable_h):
    m = np.arange(len(props["x"])) % 4 == 0
    parts = [props] if not split else [{k: v[~m] for k, v in props.items()},
                                       {k: v[m] for k, v in props.items()}]
    arrays = [base.get_particle_array(name="f%d" % i, type=Fluid, **p) for i, p in enumerate(parts)]
    particles = base.Particles(arrays=arrays, variable_h=variable_h)
    s = solver.Solver(dim=3, integrator_type=solver.RK2Integrator)
    s.add_operation(solver.SPHOperation(sph.SPHRho.withargs(), on_types=[Fluid],
                                        from_types=[Fluid], updates=["rho"], id="density"))
    s.add_operation(solver.SPHOperation(sph.TaitEquation.withargs(co=1.0, ro=1.0),
                                        on_types=[Fluid], updates=["p", "cs"], id="eos"))
    s.add_operation(solver.SPHIntegration(sph.SPHPressureGradient.withargs(dim=3),
                                          on_types=[Fluid], from_types=[Fluid],
                                          updates=["u", "v", "w"], id="pgrad"))
    s.add_operation(solver.SPHIntegration(
        sph.MonaghanArtificialVsicosity.withargs(alpha=0.1, beta=0.0), on_types=[Fluid],
        from_types=[Fluid], updates=["u", "v", "w"], id="avisc"))
    s.add_operation_step([Fluid])
    s.setup_integrator(particles)
    return s, particles
names = ("x", "y", "z", "u", "v", "w", "rho", "p", "cs")
for n in (64, 4913):
    props = W.cube_lattice(n, seed=9, vel_std=0.1)
    run(*cube(props, True, False), 1e-4, names)
    run(*cube(W.jitter_h(props), False, True), 1e-4, names)
drop = W.elliptical_drop(dx=0.06, c0=100.0)
run(*W.setup_drop(api, W.jitter_h(drop), c0=100.0, variable_h=True), 1e-5, names)
run(*W.setup_fluid_solver(api, W.circular_patch(dx=0.06)), 1e-5, names)
strip = W.periodic_strip(dx=0.05, nx=31, ny=7, jitter=0.1)
run(*W.setup_drop(api, strip, c0=10.0, periodic_domain=base.PeriodicDomain(0.0, 1.55)), 1e-4, names)
print(h.hexdigest())
'''


@pytest.mark.parametrize("subdiv", [1, 2, 3])
def test_list_lanes_give_the_same_bits_over_half_widths(subdiv):
    """One, two, four or eight threads per destination of the list builds and
    the list-streaming passes, with stencils of one to three cells, in 3D (two
    arrays; variable h) and in 2D: bit for bit the same."""
    _need_gpu()
    seen = set()
    for lanes in ("1", "2", "4", "8"):
        e = dict(os.environ, SPH_PAIR_LANES=lanes, PYSPH_GB300_SUBDIV=str(subdiv))
        r = subprocess.run([sys.executable, "-c", _HASH_LISTS_3D], cwd=ROOT, env=e,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1


_SPARSE_3D = r'''
import sys, hashlib
sys.path.insert(0, ".")
import numpy as np, oracle, pysph_gb300
from pysph_gb300 import workloads as W
from tests.golden_util import normwise
api = pysph_gb300.api()
props = W.cube_lattice(4096, seed=6)
rng = np.random.default_rng(8)
for c in "xyz":                 # a tenth of the cube scattered over a box 3 wide
    props[c][::10] = rng.uniform(-1.0, 2.0, props[c][::10].size)
s, particles = W.setup_cube(api, props)
s.integrator.integrate(1e-4)
assert particles.cell_manager.brick_pass_count() >= 4
pa = particles.arrays[0]
prob = oracle.Problem({"fluid": props}, oracle.cube_ops(), dim=3)
prob.integrate_rk2(1e-4)
for p in ("rho", "p"):
    assert normwise(pa.get(p), prob.arrays["fluid"][p]) < 1e-5, p
for p in ("x", "u", "w"):
    assert normwise(pa.get(p) - props[p], prob.arrays["fluid"][p] - props[p]) < 1e-5, p
h = hashlib.sha256()
for f in ("x", "y", "z", "u", "v", "w", "rho", "p", "cs"):
    h.update(pa.get(f).tobytes())
print(h.hexdigest())
'''


def test_blocks_of_few_occupied_rows():
    """Bricks of which only some rows of cells, not the first ones, hold
    anything, beside empty and full ones: the oracle's step, and the same
    bits with the staged entries from their table and from the rows, with one
    to four lanes."""
    _need_gpu()
    seen = set()
    for env in ({}, {"SPH_BRICK_STAGE_TABLE": "0"}, {"SPH_BRICK_LANES": "1"},
                {"SPH_BRICK_LANES": "2"}, {"SPH_BRICK_LANES": "4"}):
        e = dict(os.environ, PYSPH_GB300_BRICKS="1", **env)
        r = subprocess.run([sys.executable, "-c", _SPARSE_3D], cwd=ROOT, env=e,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
        seen.add(r.stdout.split()[-1])
    assert len(seen) == 1
