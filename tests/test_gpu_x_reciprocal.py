"""x_reciprocal (csrc/spm_xfuse.cuh), 1 / k^2 of the fused X passes from an FP32
seed, against the division on the device: random mantissas over the accepted
range of k^2 (1e-30 to 1e30), its ends and k^2 = 0.  FP64: the last operation
rounds a value within 2^-88 of the quotient, so it is within one unit in the
last place of the rounded quotient (2^-52 relative); FP32: one Newton step from
a seed of relative error 2^-22 at most leaves 2^-44."""
import subprocess

import pytest

from kapsel3_b200 import build

pytestmark = pytest.mark.gpu
SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "spm_xfuse.cuh"
using namespace spm;
__global__ void both(const double *k2, int n, double *f64, double *f32, double *div) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    f64[i] = x_reciprocal<double>(k2[i]), f32[i] = x_reciprocal<float>(k2[i]);
    div[i] = k2[i] > 0.0 ? 1.0 / k2[i] : 0.0;
}
int main() {
    std::mt19937_64                        rng(5);
    std::uniform_real_distribution<double> e(-30.0, 30.0), m(1.0, 2.0);
    std::vector<double>                    k{0.0, 1e-30, 1.0000001e-30, 1e30, 0.999999e30, 1.0, 2.0, 3.0};
    for (int i = 0; i < 1 << 20; i++) k.push_back(i & 1 ? std::pow(10.0, e(rng)) : std::ldexp(m(rng), i % 180 - 90));
    const int           n = (int)k.size();
    std::vector<double> h(3 * (size_t)n);
    double             *d = nullptr;
    if (cudaMalloc(&d, 4 * (size_t)n * sizeof(double)) != cudaSuccess) return 2;
    cudaMemcpy(d, k.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    both<<<(n + 255) / 256, 256>>>(d, n, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n);
    if (cudaMemcpy(h.data(), d + n, 3 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    double worst[2] = {0.0, 0.0};
    for (int i = 0; i < n; i++)
        for (int t = 0; t < 2; t++) {
            const double got = h[(size_t)t * n + i], want = h[2 * (size_t)n + i];
            if (k[i] == 0.0 ? got != 0.0 : !std::isfinite(got)) return 3;
            if (k[i] > 0.0) worst[t] = std::fmax(worst[t], std::fabs(got - want) / want);
        }
    std::printf("%.17g %.17g\n", worst[0], worst[1]);
    return 0;
}
"""


def test_against_the_division(gpu, tmp_path):
    try:
        nvcc = build.nvcc_path()
    except FileNotFoundError:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "reciprocal.cu", tmp_path / "reciprocal"
    src.write_text(SRC)
    subprocess.run([nvcc, *build.ARCH, "-O3", "--std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                    build.ROOT + "/include", str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)
    f64, f32 = (float(v) for v in r.stdout.split())
    assert f64 <= 2.0 ** -52 and f32 <= 2.0 ** -44, (f64, f32)
