"""FP32 fields across the C ABI (r_field_widen, r_field_narrow): rows with and
without padding, grids from the smallest up, both halves of the field.
Compensated zeta holds a double as two floats (relative error below 2^-47, an
unevaluated sum of 24 + 24 bits); a plain FP32 field is the rounded double."""
import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.spm import SPMRun
from kapsel3_b200.udf import EQ_LE, EQ_NS, SPMConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (3, 4, 5), (5, 3, 7), (4, 4, 8)])
@pytest.mark.parametrize("eq", [EQ_NS, EQ_LE])
def test_zeta_round_trip(gpu, shape, eq):
    cfg = SPMConfig(npx=shape[0], npy=shape[1], npz=shape[2], n_particles=0, lj_truncate="NONE", equation=eq,
                    shear_rate=1e-3)
    rng = np.random.default_rng(1)
    with SPMRun(cfg, precision=N.SPM_PREC_FP32_MIXED) as run:
        nx, ny, nz = run.shape
        z = rng.normal(size=(2, nx, ny, run.hnz)) + 1j * rng.normal(size=(2, nx, ny, run.hnz))
        dc = rng.normal(size=3)
        run.initialize({k: np.zeros((0, 4 if k == "q" else 3)) for k in ("x", "v", "omega", "q")})
        run.set_zeta(z, dc)
        got, gdc = run.zeta()
    assert np.array_equal(gdc, dc)
    if eq == EQ_LE:
        assert np.array_equal(got, z.astype(np.complex64).astype(np.complex128))
    else:
        v, w = got.view(float), z.view(float)
        assert (np.abs(v - w) <= 2.0 ** -47 * np.abs(w)).all()
