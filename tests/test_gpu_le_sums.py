"""Block sums of the Lees-Edwards step (k_le_shear_rate,
k_le_step_finish): the stress line against the oracle for particle counts
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


@pytest.mark.parametrize("shape,n", [((4, 5, 4), 0), ((5, 4, 6), 1), ((6, 5, 5), 17)])
def test_step_on_other_boxes(gpu, shape, n):
    """Boxes that are not cubes, across a remap of the strain (|gamma| reaches
    NX / NY), with and without particles: zeta of every mode, FP64."""
    cfg = SPMConfig(npx=shape[0], npy=shape[1], npz=shape[2], n_particles=n, a=2.0, a_xi=1.0, dt=0.1, equation=EQ_LE,
                    shear_rate=1.3, lj_truncate="ON" if n > 1 else "NONE")
    parts = make_particles(cfg, seed=n, v_sd=1e-3, random_orientation=True)
    oracle = OracleSPMLE(cfg, parts)
    rng = np.random.default_rng(5)
    u = 1e-2 * rng.normal(size=(3,) + cfg.shape)
    oracle.zeta, oracle.uk_dc = oracle.u_k2zeta_k(oracle.solenoidal_uk(oracle.truncate(oracle.fft(u))))
    with SPMRun(cfg) as run:
        run.initialize(parts)
        run.set_zeta(oracle.zeta, oracle.uk_dc)
        steps = int(np.ceil(cfg.shape[0] / cfg.shape[1] / 0.13)) + 2
        run.step(steps)
        zeta, _ = run.zeta()
    for _ in range(steps):
        oracle.step()
    assert abs(oracle.gamma) < cfg.shape[0] / cfg.shape[1]
    assert np.linalg.norm(zeta - oracle.zeta) <= 1e-11 * np.linalg.norm(oracle.zeta)
