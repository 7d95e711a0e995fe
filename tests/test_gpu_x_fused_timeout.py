"""Bounded waits of the fused X passes: with three passes told to issue no tile
load (spm_debug_skip_tma_loads) the step's two Y passes and its fused update
run out of their 1 ms waits with nothing in flight and stop; the next
synchronising call reports the timeout and the context steps on."""
import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.spm import SPMRun
from kapsel3_b200.udf import SPMConfig, make_particles
from kernel_names import step_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [N.SPM_PREC_FP64, N.SPM_PREC_FP32_MIXED])
def test_fused_wait_runs_out(gpu, prec):
    cfg = SPMConfig(npx=5, npy=5, npz=5, n_particles=2, a=4.0, a_xi=2.0, dt=0.05)
    parts = make_particles(cfg, seed=7, v_sd=1e-3, random_orientation=True)
    with SPMRun(cfg, precision=prec) as run:
        run.initialize(parts)
        assert "x_ns_update" in step_kernels(run)  # the third pass is the fused one
        run.initialize(parts)
        run.step(3)
        want = run.particles()
        assert run.L.spm_set_wait_limit(run.h, 1e-3) == 0
        assert run.L.spm_debug_skip_tma_loads(run.h, 3) == 0
        run.step(1)
        with pytest.raises(N.SpmError, match="TMA pipeline wait timed out"):
            run.synchronize()
        assert run.L.spm_set_wait_limit(run.h, 1.0) == 0
        run.initialize(parts)
        run.step(3)
        got = run.particles()
    for k in ("x", "v", "omega", "q"):
        assert np.linalg.norm(got[k] - want[k]) <= 1e-12 * np.linalg.norm(want[k]), k
