"""Block sums of the Lees-Edwards step (k_le_finish_reduction,
k_le_stress_finish): the stress line against the oracle for particle counts
below, at and above one block of 1024 threads.

FP64 sums of n terms in another order differ by at most about n 2^-53 of the
terms' absolute sum; with n = 1100 particles and the cancellation between
them the columns agree to 1e-10 of the largest one."""
import numpy as np
import pytest

from kapsel3_b200.spm import SPMRun
from kapsel3_b200.udf import EQ_LE, SPMConfig, make_particles
from oracle.spm_oracle import OracleSPMLE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side", [(1, 5), (31, 5), (1024, 6), (1100, 6)])
def test_stress_sums(gpu, n, side):
    cfg = SPMConfig(npx=side, npy=side, npz=side, n_particles=n, a=1.0, a_xi=1.0, dt=0.01, equation=EQ_LE,
                    shear_rate=1e-2, lj_truncate="NONE")
    parts = make_particles(cfg, seed=n, v_sd=1e-2, random_orientation=True)
    oracle = OracleSPMLE(cfg, parts)
    with SPMRun(cfg) as run:
        run.initialize(parts)
        for _ in range(2):
            run.step(1)
            oracle.step()
        _, st = run.shear_state()
    want = np.array([oracle.stress[k] for k in ("shear_rate", "strain", "lj", "hydro_old", "hydro_new", "reynolds",
                                                "fluid", "apparent")])
    assert np.abs(st - want).max() <= 1e-10 * np.abs(want).max()
