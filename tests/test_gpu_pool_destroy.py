"""Destroying and growing a pool does not wait for the device: the pinned words
of destroyed pools are kept for the next one (zeroed), not unmapped."""
import ctypes as C
import time

import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.serve import Pool
from kapsel3_b200.udf import SPMConfig, make_particles

pytestmark = pytest.mark.gpu
SMALL = SPMConfig(npx=5, npy=5, npz=5, n_particles=1, a=3.0, a_xi=2.0, dt=0.05)


def _small(capacity=1):
    pool = Pool(SMALL, precision=N.SPM_PREC_FP64, capacity=capacity)
    run = pool.admit(SMALL, make_particles(SMALL, seed=0))
    pool.step(1)
    pool.synchronize()
    return pool, run


def test_destroy_beside_a_stepping_pool(gpu):
    cfg = SPMConfig(npx=7, npy=7, npz=7, n_particles=4, a=4.0, a_xi=2.0, dt=0.01)
    with Pool(cfg, precision=N.SPM_PREC_FP64, capacity=2) as busy:
        for i in range(2):
            busy.admit(cfg, make_particles(cfg, seed=i))
        busy.step(1)
        busy.synchronize()
        pools = [_small()[0] for _ in range(4)]
        busy.step(600)  # some 0.2 s on the device
        took = []
        for p in pools:
            t = time.perf_counter()
            p.close()
            took.append(time.perf_counter() - t)
        t = time.perf_counter()
        busy.synchronize()
        left = time.perf_counter() - t
    assert sum(took) < 0.25 * left, (took, left)


def test_kept_words_start_at_zero(gpu):
    """A pool whose run left an error bit in its words, then others that reuse
    them: no error before their first step, and the bound holds for many pools."""
    parts = make_particles(SMALL, seed=0)
    for _ in range(3):
        pool, run = _small()
        rec = pool.particles(run, 1)
        rec[0, 6] = -1e4  # v_x: the next position update leaves the box
        N.check(pool.L.spm_set_particles(run, N.dptr(rec)), "spm_set_particles")
        pool.step(1)
        assert pool.synchronize()[1] != [0]
        pool.close()
        with Pool(SMALL, precision=N.SPM_PREC_FP64, capacity=1) as fresh:
            fresh.admit(SMALL, parts)
            assert fresh.synchronize()[1] == [0]
            fresh.admit(SMALL, parts)  # the arena grows
            assert fresh.synchronize()[1] == [0, 0]
            fresh.step(1)
            assert fresh.synchronize()[1] == [0, 0]
    held = C.c_size_t()
    N.check(N.lib().spm_release_cached_memory(C.byref(held)), "spm_release_cached_memory")
    pool, run = _small(3)
    assert np.isfinite(pool.particles(run, 1)).all()
    pool.close()
