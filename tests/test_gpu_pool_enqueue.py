"""spm_pool_step only enqueues: a second call after a membership change does not
wait for the first call's steps, and a step without graph replay can be recorded
into the caller's own CUDA graph, the first one after a membership change
included (host copies and waits belong to the calls that change the
membership)."""
import ctypes as C
import time

import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200.serve import Pool
from kapsel3_b200.spm import pack_particles, params_from_config, unpack_particles
from kapsel3_b200.udf import SPMConfig, make_particles

pytestmark = pytest.mark.gpu


def test_second_call_does_not_wait(gpu):
    cfg = SPMConfig(npx=7, npy=7, npz=7, n_particles=4, a=4.0, a_xi=2.0, dt=0.01)
    with Pool(cfg, precision=N.SPM_PREC_FP64, capacity=4) as pool:
        for i in range(2):
            pool.admit(cfg, make_particles(cfg, seed=i))
        pool.step(3)
        pool.synchronize()
        pool.admit(cfg, make_particles(cfg, seed=2))
        t0 = time.perf_counter()
        pool.step(300)  # some 0.15 s on the device
        t1 = time.perf_counter()
        pool.step(1)
        t2 = time.perf_counter()
        pool.synchronize()
        t3 = time.perf_counter()
    # the first call captures the step's graph; the device is busy until long after the second
    assert t2 - t1 < 0.25 * (t3 - t0), (t1 - t0, t2 - t1, t3 - t0)


def test_first_step_recorded_by_the_caller(gpu):
    import torch
    cfg = SPMConfig(npx=5, npy=4, npz=5, n_particles=3, a=2.0, a_xi=1.0, dt=0.05, kbt=1e-4)
    parts = [make_particles(cfg, seed=i, v_sd=1e-3, random_orientation=True) for i in range(2)]
    L, got = N.lib(), []
    for record in (False, True):
        stream, pool = torch.cuda.Stream(), C.c_void_p()
        p = params_from_config(cfg, N.SPM_PREC_FP64)
        N.check(L.spm_pool_create(C.byref(p), 2, C.c_void_p(stream.cuda_stream), C.byref(pool)), "spm_pool_create")
        runs = []
        for i, q in enumerate(parts):
            run, rec = C.c_void_p(), pack_particles(q, cfg.n_particles)
            p = params_from_config(cfg, N.SPM_PREC_FP64, mt_seed=i)
            N.check(L.spm_pool_admit(pool, C.byref(p), N.dptr(rec), C.byref(run)), "spm_pool_admit")
            runs.append(run)
        if record:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                N.check(L.spm_pool_step(pool, 1, 0), "spm_pool_step")
            with torch.cuda.stream(stream):
                graph.replay()
                graph.replay()
            stream.synchronize()
        else:
            N.check(L.spm_pool_step(pool, 2, 0), "spm_pool_step")
        rec = np.zeros((cfg.n_particles, N.SPM_PARTICLE_WORDS))
        for run in runs:
            N.check(L.spm_get_particles(run, N.dptr(rec)), "spm_get_particles")
            got.append(unpack_particles(rec.copy()))
        if record:
            del graph
        N.check(L.spm_pool_destroy(pool), "spm_pool_destroy")
    for a, b in zip(got[:2], got[2:]):
        for k in ("x", "v", "omega", "q"):
            assert np.linalg.norm(a[k] - b[k]) <= 1e-12 * np.linalg.norm(a[k]), k
