"""Fused X passes of the step (csrc/spm_xfuse.cuh): whole Navier_Stokes steps
of a random flow against the oracle at every axis length the fused passes
serve (FP32 up to 512 points in two TMA boxes a tile, FP64 up to 256), at an
FP64 axis of 512 points (the separate passes), and with the separate passes
forced.  The names of the launched kernels say which passes ran.

FP64: one step is a chain of unnormalised transforms of length n and a
pointwise update, rounding error about log2(n) 2^-53 of the field; FP32 the
same with 2^-24 (log2(n) <= 22 here, some tens of operations per mode)."""
import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.spm import SPMRun
from kapsel3_b200.udf import SPMConfig
from kernel_names import step_kernels
from oracle.spm_oracle import OracleSPM

pytestmark = pytest.mark.gpu
SHAPES = [(3, 3, 3), (4, 3, 5), (5, 4, 3), (6, 3, 4), (7, 3, 3), (8, 3, 4), (9, 3, 3), (3, 8, 5), (4, 9, 3)]


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _flow(shape, no_tma, monkeypatch, prec, steps=2, dx=1.0):
    cfg = SPMConfig(npx=shape[0], npy=shape[1], npz=shape[2], n_particles=0, lj_truncate="NONE", dt=0.05 * dx * dx,
                    dx=dx, fix_cell=(True, False, True))
    none = dict(x=np.zeros((0, 3)), v=np.zeros((0, 3)), omega=np.zeros((0, 3)), q=np.zeros((0, 4)))
    oracle = OracleSPM(cfg, none)
    rng = np.random.default_rng(sum(shape))
    u = rng.normal(size=(3,) + cfg.shape)
    oracle.zeta, oracle.uk_dc = oracle.u_k2zeta_k(oracle.solenoidal_uk(oracle.truncate(oracle.fft(u))))
    monkeypatch.setenv("SPM_NO_TMA", "1" if no_tma else "0")
    with SPMRun(cfg, precision=prec) as run:
        run.initialize(none)
        run.set_zeta(oracle.zeta, oracle.uk_dc)
        run.step(steps)
        zeta, dc = run.zeta()
        fused = not no_tma and cfg.shape[0] <= (256 if prec == N.SPM_PREC_FP64 else 512)
        names = step_kernels(run)
        assert ({"x_zeta_u", "x_ns_update", "x_project"} & names) == (
            {"x_zeta_u", "x_ns_update", "x_project"} if fused else set())
        assert ("k_ns_update" in names) != fused
    for _ in range(steps):
        oracle.step()
    return rel(zeta, oracle.truncate(oracle.zeta)), dc, oracle.uk_dc


@pytest.mark.parametrize("no_tma", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_flow_step_fp64(gpu, shape, no_tma, monkeypatch):
    err, dc, want = _flow(shape, no_tma, monkeypatch, N.SPM_PREC_FP64)
    assert err <= 1e-13
    assert np.abs(dc - want).max() <= 1e-13 * (1.0 + np.abs(want).max())


@pytest.mark.parametrize("dx", [1e-3, 37.0])
@pytest.mark.parametrize("prec,tol", [(N.SPM_PREC_FP64, 1e-13), (N.SPM_PREC_FP32_MIXED, 3e-6)])
def test_flow_step_other_spacing(gpu, prec, tol, dx, monkeypatch):
    """k^2 far from 1 (the reciprocal of the fused passes starts from an FP32 seed)."""
    err, _, _ = _flow((5, 4, 3), False, monkeypatch, prec, dx=dx)
    assert err <= tol


@pytest.mark.parametrize("shape", SHAPES)
def test_flow_step_fp32(gpu, shape, monkeypatch):
    err, _, _ = _flow(shape, False, monkeypatch, N.SPM_PREC_FP32_MIXED)
    assert err <= 3e-6
