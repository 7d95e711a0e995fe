"""The fused X passes on every device of a process: the shared-memory limit and
the occupancy of an instance belong to the device that is current when a plan
is created (cudaFuncSetAttribute).  On the host with a stand-in for the two
calls that keeps limits per device; on a machine with two devices with runs on
both."""
import os
import subprocess

import numpy as np
import pytest

from kapsel3_b200 import _native as N
from kapsel3_b200 import build
from kapsel3_b200.spm import SPMRun, device_count
from kapsel3_b200.udf import SPMConfig, make_particles

SRC = r"""
#include <cstdio>
#include <map>
#include <cuda_runtime.h>
static int g_dev = 0, g_refuse = 0;
static std::map<std::pair<int, const void *>, int> g_limit;
template <typename K>
cudaError_t fake_attribute(K kern, cudaFuncAttribute, int bytes) {
    if (g_refuse) return cudaErrorInvalidValue;
    g_limit[{g_dev, (const void *)kern}] = bytes;
    return cudaSuccess;
}
template <typename K>
cudaError_t fake_occupancy(int *n, K kern, int, size_t bytes) {
    auto it = g_limit.find({g_dev, (const void *)kern});
    if (it == g_limit.end() || (size_t)it->second < bytes) return cudaErrorInvalidValue;
    *n = 3 + g_dev;
    return cudaSuccess;
}
#define cudaFuncSetAttribute fake_attribute
#define cudaOccupancyMaxActiveBlocksPerMultiprocessor fake_occupancy
#include "spm_xfuse.cuh"
using namespace spm;
int main() {
    auto occ = [] { return x_fused_occupancy<float, 8, kXZeta, true>(); };
    int bad = 0;
    g_refuse = 1;
    bad += occ() != 0;  // refused: the separate passes, and not for the life of the process
    g_refuse = 0;
    bad += occ() != 3;
    g_dev = 1;
    bad += occ() != 4;
    g_dev = 0;
    bad += occ() != 3;
    int seen[5] = {};
    seen[x_instance(kXZeta, true)]++, seen[x_instance(kXNs, true)]++, seen[x_instance(kXNs, false)]++;
    seen[x_instance(kXProj, false)]++, seen[x_instance(kXSole, true)]++;
    for (int s : seen) bad += s != 1;
    bad += x_instance(kXProj, true) != x_instance(kXProj, false);
    std::printf("%d\n", bad);
    return bad;
}
"""


def test_instances_are_set_up_on_each_device(tmp_path):
    try:
        nvcc = build.nvcc_path()
    except FileNotFoundError:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "devices.cu", tmp_path / "devices"
    src.write_text(SRC)
    subprocess.run([nvcc, *build.ARCH, "--std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                    os.path.join(build.ROOT, "include"), str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [N.SPM_PREC_FP64, N.SPM_PREC_FP32_MIXED])
def test_runs_on_two_devices(gpu, prec):
    if device_count() < 2:
        pytest.skip("needs two devices")
    import torch
    cfg = SPMConfig(npx=7, npy=4, npz=4, n_particles=2, a=2.0, a_xi=1.0, dt=0.05)  # 128 points: more than 48 KB
    parts = make_particles(cfg, seed=1, v_sd=1e-3)
    got = []
    for dev in (0, 1):
        with torch.cuda.device(dev), SPMRun(cfg, precision=prec) as run:
            run.initialize(parts)
            run.step(2)
            got.append(run.particles()["v"])
    assert np.linalg.norm(got[0] - got[1]) <= 1e-12 * np.linalg.norm(got[0])
