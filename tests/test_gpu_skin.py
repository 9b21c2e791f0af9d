"""Neighbour lists with a skin: light refreshes between full builds keep
every result of the reference's path (neighbour sets, trajectories)."""
import numpy as np
import pytest
import torch

import oracle
import pysph_gb300
from golden_util import csr_sets, normwise
from pysph_gb300 import workloads as W

pytestmark = pytest.mark.gpu
API = pysph_gb300.api()


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def test_light_refresh_keeps_neighbour_sets_exact():
    _need_gpu()
    props = W.cube_lattice(32768, seed=3, vel_std=0.5)
    s, particles = W.setup_cube(API, props)
    for _ in range(3):
        s.integrator.integrate(1e-4)
    cm = particles.cell_manager
    full, light = cm.build_stats()
    assert light > 0, (full, light)
    pa = particles.arrays[0]
    loc = particles.nnps_manager.get_neighbor_particle_locator(pa, pa, 2.0)
    off, idx = loc.neighbour_csr()
    host = {k: pa.get(k) for k in ("x", "y", "z", "h")}
    ro, ri = oracle.neighbors(host, host, 2.0 * host["h"].max(), 2.0, same=True)
    assert csr_sets(off, idx) == csr_sets(ro, ri)


def _drop_run(steps, monkeypatch, skin):
    monkeypatch.setenv("PYSPH_GB300_SKIN", str(skin))
    props = W.elliptical_drop(dx=0.025, c0=100.0)
    s, particles = W.setup_drop(API, props, c0=100.0)
    for _ in range(steps):
        s.integrator.integrate(1e-5)
    pa = particles.arrays[0]
    out = {k: pa.get(k) for k in ("x", "y", "u", "v", "rho", "p")}
    return props, out, particles.cell_manager.build_stats()


def test_skin_trajectory_matches_exact_lists(monkeypatch):
    """40 Euler steps of the fast drop with and without a skin: light
    refreshes and forced rebuilds both occur, the results agree to FP32
    summation-order differences."""
    _need_gpu()
    props, a, st_a = _drop_run(40, monkeypatch, 0.05)
    _, b, st_b = _drop_run(40, monkeypatch, 0.0)
    assert st_a[1] > 0 and st_a[0] > 1, st_a       # light refreshes and full builds
    assert st_b[1] == 0, st_b
    for p in ("x", "y", "u", "v"):
        assert normwise(a[p] - props[p], b[p] - props[p]) < 1e-5, p
    for p in ("rho", "p"):
        assert normwise(a[p], b[p]) < 1e-5, p


def test_skin_drop_matches_oracle(monkeypatch):
    _need_gpu()
    props, a, st = _drop_run(10, monkeypatch, 0.05)
    assert st[1] > 0
    prob = oracle.Problem({"fluid": props}, oracle.drop_ops(c0=100.0), dim=2)
    for _ in range(10):
        prob.integrate_euler(1e-5)
    ref = prob.arrays["fluid"]
    for p in ("x", "y", "u", "v"):
        assert normwise(a[p] - props[p], ref[p] - props[p]) < 1e-4, p
    assert normwise(a["rho"], ref["rho"]) < 1e-5


@pytest.mark.parametrize("sizes", [(600,), (600, 150), (40, 0, 600), (300, 20, 1, 270),
                                   (90, 0, 300, 20, 70, 110)])
def test_light_refresh_of_several_arrays(sizes, monkeypatch):
    """One launch refreshes up to four arrays, of any lengths (none included):
    after a move inside the skin every array's density over all arrays is the
    oracle's at the new positions."""
    _need_gpu()
    monkeypatch.setenv("PYSPH_GB300_SKIN", "0.05")
    rng = np.random.default_rng(len(sizes))
    base, sph = API.base, API.sph
    h = 0.05
    props = [{"x": rng.uniform(0, 1, n), "y": rng.uniform(0, 1, n), "h": np.full(n, h),
              "m": rng.uniform(0.5, 1.5, n), "rho": np.ones(n)} for n in sizes]
    arrays = [base.get_particle_array(name="a%d" % k, type=base.ParticleType.Fluid, **p)
              for k, p in enumerate(props)]
    particles = base.Particles(arrays=arrays)
    kern = base.CubicSplineKernel(dim=2)
    for step in range(2):
        if step:
            for pa, p in zip(arrays, props):
                for c in "xy":
                    p[c] = p[c] + 0.001 * rng.uniform(-1, 1, len(p[c]))
                pa.set(x=p["x"], y=p["y"])
            particles.update()
        for pa, p in zip(arrays, props):
            if len(p["x"]) == 0:
                continue
            calc = sph.SPHCalc(particles, arrays, pa, kern,
                               [sph.SPHRho.get_func(s, pa) for s in arrays], ["rho"])
            calc.sph("rho")
            want = np.zeros(len(p["x"]))
            for q in props:
                if len(q["x"]) == 0:
                    continue
                off, idx = oracle.neighbors(p, q, 2.0 * h, same=q is p)
                want += oracle.pair_sum("rho", p, q, off, idx, 2, nout=1)[0]
            assert normwise(pa.get("rho"), want) < 1e-5
    full, light = particles.cell_manager.build_stats()
    assert light >= 1, (full, light)
