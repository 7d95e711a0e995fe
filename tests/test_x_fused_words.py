"""Which words of zeta the threads of a fused X pass load and store
(csrc/spm_xfuse.cuh), walked on the host over every tile, thread and mode with
the kernel's own index functions: a word that one thread stores is loaded by no
other, every mode of the retained box is stored exactly once, and no load or
store leaves the field."""
import os
import subprocess

import pytest

from kapsel3_b200 import build

SRC = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "spm_xfuse.cuh"
using namespace spm;

template <typename T, int N>
int walk(int ny, int nz) {
    using M = XModes<N>;
    constexpr int W = kXCols<T, N>;
    Grid g{};
    g.nx = N, g.ny = ny, g.nz = nz, g.hnz = nz / 2 + 1;
    g.hnzp = sizeof(T) == 8 ? g.hnz : (g.hnz + 1) & ~1;
    const int n3[3] = {N, ny, nz};
    for (int d = 0; d < 3; d++) g.trn[d] = (n3[d] + 2) / 3;
    const size_t   words = g.field_elems_c();
    const unsigned nst   = (unsigned)ny * g.hnzp;
    const int ct_used = (g.trn[2] + W - 1) / W, n_used = outer_count(ny, g.trn[1]);
    std::vector<int> store(words, -1);
    long stored = 0;
    for (int pass = 0; pass < 2; pass++)  // stores first, then the loads against them
        for (int t = 0; t < ct_used * n_used; t++)
            for (int tid = 0; tid < W * M::N1; tid++) {
                const int  kz = (t % ct_used) * W + tid % W, gg = tid / W;
                const int  o  = outer_line(t / ct_used, ny, g.trn[1]);
                const bool col = kz < g.trn[2];
                const int  me  = t * W * M::N1 + tid;
                const unsigned line = x_line(g, o, kz);
                for (int m = 0; m < M::N2; m++) {
                    if (!M::maybe(m)) continue;
                    const int  k   = signed_mode(gg + M::N1 * m, N);
                    const bool box = col && std::abs(k) < g.trn[0];
                    if ((col && M::retained(gg, m)) != box) return std::printf("retained %d %d\n", gg, m), 1;
                    if (pass == 0) {
                        if (!box) continue;
                        const size_t w = (size_t)(gg + M::N1 * m) * nst + line;
                        if (w >= words || store[w] >= 0) return std::printf("store %zu\n", w), 1;
                        store[w] = me;
                        stored++;
                    } else {
                        const size_t w = (size_t)M::zeta_index(gg, m) * nst + line;
                        if (w >= words) return std::printf("load past the field %zu\n", w), 1;
                        if (store[w] >= 0 && store[w] != me) return std::printf("word %zu of thread %d loaded by %d\n", w, store[w], me), 1;
                        if (box && store[w] != me) return std::printf("mode %zu\n", w), 1;
                    }
                }
            }
    return stored == (long)g.box_elems() ? 0 : (std::printf("%ld stored\n", stored), 1);
}
template <typename T, int N>
int axis() {
    for (int ny : {8, 16, 64})
        for (int nz : {8, 16, 32, 128, 256})
            if (walk<T, N>(ny, nz)) return std::printf("N %d ny %d nz %d bytes %zu\n", N, ny, nz, sizeof(T)), 1;
    return 0;
}
int main() {
    return axis<double, 8>() || axis<double, 16>() || axis<double, 32>() || axis<double, 64>() || axis<double, 128>() ||
           axis<double, 256>() || axis<float, 8>() || axis<float, 16>() || axis<float, 32>() || axis<float, 64>() ||
           axis<float, 128>() || axis<float, 256>() || axis<float, 512>();
}
"""


@pytest.fixture(scope="module")
def nvcc():
    try:
        return build.nvcc_path()
    except FileNotFoundError:
        pytest.skip("no nvcc")


def test_no_word_is_loaded_beside_its_store(nvcc, tmp_path):
    src, exe = tmp_path / "words.cu", tmp_path / "words"
    src.write_text(SRC)
    subprocess.run([nvcc, *build.ARCH, "--std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                    os.path.join(build.ROOT, "include"), str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
