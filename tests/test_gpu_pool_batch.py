"""Particle kernels of a pool's step, one launch over all runs: runs of
different particle counts, stencils and options (no particles, one, more than
a block of threads, thermostat, obstacles, no Lennard-Jones pairs) advance in
the pool as they do alone.  FP64; the only difference left is the order of the
atomics where three or more profiles overlap a cell (1e-12)."""
import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.serve import Pool
from kapsel3_b200.spm import SPMRun, unpack_particles
from kapsel3_b200.udf import SPMConfig, make_particles

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _cfgs(side):
    base = dict(npx=side, npy=side, npz=side + 1, a_xi=2.0, dt=0.05)
    return [SPMConfig(n_particles=0, a=4.0, **base),
            SPMConfig(n_particles=1, a=4.0, kbt=1e-4, **base),
            SPMConfig(n_particles=150, a=1.5, lj_truncate="NONE", **base),
            SPMConfig(n_particles=5, a=3.0, janus_axis="Z", janus_propulsion="OBSTACLE", kbt=1e-4, **base),
            SPMConfig(n_particles=7, a=2.5, body_force=(1e-3, 0.0, 0.0), rotation=False, **base)]


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("order", [(0, 1, 2, 3, 4), (2,), (0,), (4, 3, 1)])
def test_pool_runs_match_lone_runs(gpu, order, use_graph):
    cfgs = [_cfgs(5)[i] for i in order]
    parts = [make_particles(c, seed=40 + i, v_sd=1e-3, random_orientation=True) for i, c in zip(order, cfgs)]
    want = []
    for i, c, p in zip(order, cfgs, parts):
        with SPMRun(c, mt_seed=i) as run:
            run.initialize(p)
            run.step(3)
            want.append((run.particles(), run.velocity()))
    with Pool(cfgs[0], precision=N.SPM_PREC_FP64, capacity=2) as pool:
        runs = [pool.admit(c, p, mt_seed=i) for i, c, p in zip(order, cfgs, parts)]
        pool.step(3, use_graph=use_graph)
        pool.synchronize()
        for r, c, (p, u) in zip(runs, cfgs, want):
            got = unpack_particles(pool.particles(r, c.n_particles))
            for k in ("x", "v", "omega", "q", "f_hydro_previous", "fr_previous"):
                assert rel(got[k], p[k]) <= 1e-12, (c.n_particles, k)
            assert rel(pool.velocity(r, c.shape), u) <= 1e-12, c.n_particles


@pytest.mark.parametrize("shape", [(3, 5, 5), (5, 5, 3)])
def test_pool_without_a_cell_list(gpu, shape):
    """An axis of 8 points (no Lennard-Jones forces there): the body forces, one launch per run."""
    cfgs = [SPMConfig(npx=shape[0], npy=shape[1], npz=shape[2], n_particles=n, a=1.0, a_xi=1.0, dt=0.05,
                      lj_truncate="NONE", body_force=(1e-3, 0.0, 0.0)) for n in (0, 9, 2)]
    parts = [make_particles(c, seed=50 + i, v_sd=1e-3) for i, c in enumerate(cfgs)]
    with Pool(cfgs[0], precision=N.SPM_PREC_FP64, capacity=3) as pool:
        runs = [pool.admit(c, p) for c, p in zip(cfgs, parts)]
        pool.step(3)
        pool.synchronize()
        got = [unpack_particles(pool.particles(r, c.n_particles)) for r, c in zip(runs, cfgs)]
    for c, p, g in zip(cfgs, parts, got):
        with SPMRun(c) as run:
            run.initialize(p)
            run.step(3)
            want = run.particles()
        for k in ("x", "v", "f_hydro_previous", "fr_previous"):
            assert rel(g[k], want[k]) <= 1e-12, (c.n_particles, k)
