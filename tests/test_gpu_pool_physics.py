"""Runs of a pool with different viscosities, densities and time steps advance
as they do alone, in the fused update and in the separate one, whatever their
order (a pool holds runs of one grid; only the grid, DX and the precision are
shared).  FP64, the same operations per run: 1e-12."""
import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.serve import Pool
from kapsel3_b200.spm import SPMRun, unpack_particles
from kapsel3_b200.udf import SPMConfig, make_particles

pytestmark = pytest.mark.gpu
BASE = dict(npx=5, npy=4, npz=5, n_particles=2, a=2.0, a_xi=1.0)
CFGS = [SPMConfig(dt=0.05, **BASE), SPMConfig(dt=0.02, eta=2.0, **BASE), SPMConfig(dt=0.02, eta=2.0, rho=0.5, **BASE)]


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("no_tma", [False, True])
@pytest.mark.parametrize("order", [(1,), (0, 1), (1, 1, 0), (0, 2, 2, 1, 0)])
def test_each_run_keeps_its_constants(gpu, order, no_tma, monkeypatch):
    monkeypatch.setenv("SPM_NO_TMA", "1" if no_tma else "0")
    parts = [make_particles(CFGS[i], seed=k, v_sd=1e-2, random_orientation=True) for k, i in enumerate(order)]
    want = []
    for i, p in zip(order, parts):
        with SPMRun(CFGS[i]) as run:
            run.initialize(p)
            run.step(4)
            want.append((run.particles(), run.velocity()))
    with Pool(CFGS[0], precision=N.SPM_PREC_FP64, capacity=len(order)) as pool:
        runs = [pool.admit(CFGS[i], p) for i, p in zip(order, parts)]
        pool.step(3)
        pool.step(1, use_graph=False)
        pool.synchronize()
        for r, i, (p, u) in zip(runs, order, want):
            got = unpack_particles(pool.particles(r, 2))
            for k in ("x", "v", "omega", "f_hydro_previous"):
                assert _rel(got[k], p[k]) <= 1e-12, (i, k)
            assert _rel(pool.velocity(r, CFGS[i].shape), u) <= 1e-12, i
