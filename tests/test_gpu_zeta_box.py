"""Zeta outside the 2/3 box, set from outside a step: the next step drops it
(the reference truncates zeta at the start of every step, fluid_solver.cxx:
313-374), whichever entry point wrote it.  Through spm_set_zeta, a state saved
and loaded before its first step, and U_k2zeta_k; every equation that truncates
in the step, every mode compared."""
import os

import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.spm import SPMRun
from kapsel3_b200.udf import EQ_EL, EQ_NS, EQ_SNS, SPMConfig, make_particles

pytestmark = pytest.mark.gpu
EL = dict(kbt=1.0, dt=0.005, salt=True, valency=(1.0, -1.0), onsager=(1.0, 1.0), debye_length=4.0, surface_charge=-8.0)
RUNS = [(EQ_NS, N.SPM_PREC_FP64, {}), (EQ_NS, N.SPM_PREC_FP32_MIXED, {}),
        (EQ_SNS, N.SPM_PREC_FP64, dict(shear_rate=0.01)), (EQ_EL, N.SPM_PREC_FP64, EL)]


def _case(eq, more):
    cfg = SPMConfig(**{**dict(npx=4, npy=5, npz=4, n_particles=1, a=3.0, a_xi=2.0, dt=0.05, equation=eq), **more})
    nx, ny, nz = cfg.shape
    rng = np.random.default_rng(7)
    k = np.fft.rfftn(1e-2 * rng.normal(size=(3, nx, ny, nz)), axes=(1, 2, 3))
    kx, ky = (np.array([i - n if i > n // 2 else i for i in range(n)]) for n in (nx, ny))
    box = ((abs(kx) < (nx + 2) // 3)[:, None, None] & (abs(ky) < (ny + 2) // 3)[None, :, None]
           & (np.arange(nz // 2 + 1) < (nz + 2) // 3))
    return cfg, make_particles(cfg, seed=2, v_sd=1e-3), k, box


def _same(a, b, tol=1e-12):
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("eq,prec,more", RUNS)
def test_state_saved_before_its_first_step(gpu, eq, prec, more, steps, tmp_path):
    cfg, parts, k, box = _case(eq, more)
    path = os.path.join(tmp_path, "s.ck")
    with SPMRun(cfg, precision=prec) as a, SPMRun(cfg, precision=prec) as b:
        a.initialize(parts)
        a.set_zeta(k[:2], np.zeros(3))
        a.save_state(path)
        b.initialize(parts)
        b.load_state(path)
        a.step(steps)
        b.step(steps)
        (za, _), (zb, _) = a.zeta(), b.zeta()
        ua, ub = a.velocity(), b.velocity()
    assert not za[:, ~box].any() and not zb[:, ~box].any()
    _same(zb, za)
    _same(ub, ua)


@pytest.mark.parametrize("eq,prec,more", RUNS)
def test_zeta_of_a_velocity(gpu, eq, prec, more):
    cfg, parts, k, box = _case(eq, more)
    with SPMRun(cfg, precision=prec) as run:
        run.initialize(parts)
        run.step(1)
        z, dc = run.U_k2zeta_k(k)
        assert z[:, ~box].any()
        assert np.array_equal(run.zeta()[0], z)  # no compensation left of the zeta before
        run.step(2)
        got, _ = run.zeta()
    assert not got[:, ~box].any()
