"""Solenoidal_u in one X pass (x_fused_kernel, kXSole) in the squirmers' slip
loop and in the Electrolyte step (which also takes zeta from it), against the
separate passes (SPM_NO_TMA=1), three steps: the same operations in another
order.  A hydrodynamic force is a difference of nearly equal velocities: with up
to 10^3 of cancellation and some 10^2 roundings a mode, FP64 stays below 1e-11
and FP32 below 2e-4 of the norm."""
import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.spm import SPMRun
from kapsel3_b200.udf import EQ_EL, SPMConfig, make_particles
from kernel_names import step_kernels

pytestmark = pytest.mark.gpu


def _run(cfg, parts, no_tma, monkeypatch, prec):
    monkeypatch.setenv("SPM_NO_TMA", "1" if no_tma else "0")
    with SPMRun(cfg, precision=prec) as run:
        run.initialize(parts)
        run.step(3)
        out = run.particles(), run.velocity()
        fused = not no_tma and cfg.shape[0] <= (256 if prec == N.SPM_PREC_FP64 else 512)
        assert ("x_solenoidal" in step_kernels(run)) == fused
        return out


def _close(cfg, monkeypatch, prec, tol):
    parts = make_particles(cfg, seed=3, v_sd=1e-3, random_orientation=True)
    (p, u), (q, w) = (_run(cfg, parts, t, monkeypatch, prec) for t in (False, True))
    for k in ("x", "v", "f_hydro_previous"):
        assert np.linalg.norm(p[k] - q[k]) <= tol * np.linalg.norm(q[k]), k
    assert np.linalg.norm(u - w) <= tol * np.linalg.norm(w)


SHAPES = [(4, 4, 4), (5, 4, 6), (6, 5, 4), (7, 4, 5), (8, 4, 4), (9, 4, 4)]
PREC = [(N.SPM_PREC_FP64, 1e-11), (N.SPM_PREC_FP32_MIXED, 2e-4)]


@pytest.mark.parametrize("prec,tol", PREC)
@pytest.mark.parametrize("shape", SHAPES)
def test_squirmers(gpu, shape, prec, tol, monkeypatch):
    cfg = SPMConfig(npx=shape[0], npy=shape[1], npz=shape[2], n_particles=3, a=2.0, a_xi=1.0, dt=0.1, janus_axis="Z",
                    janus_propulsion="SQUIRMER", slip_vel=0.015, slip_mode=1.0, slip_tol=0.0, slip_iter=3)
    _close(cfg, monkeypatch, prec, tol)


@pytest.mark.parametrize("prec,tol", PREC)
@pytest.mark.parametrize("shape", SHAPES)
def test_electrolyte(gpu, shape, prec, tol, monkeypatch):
    cfg = SPMConfig(npx=shape[0], npy=shape[1], npz=shape[2], n_particles=2, a=2.0, a_xi=1.0, dt=0.005, kbt=1.0,
                    equation=EQ_EL, salt=True, valency=(1.0, -1.0), onsager=(1.0, 1.0), debye_length=2.0,
                    surface_charge=-5.0, e_field="DC", e_ext=(0.05, 0.0, 0.0))
    _close(cfg, monkeypatch, prec, tol)
