"""The FP32 dot products of the mixed solves, four vectors a block.

Every product of two floats is exact in FP64, so widening by integer operations
and shared butterflies must leave the bits of plain conversions and a butterfly
a vector: each thread's sum in stride order, pairs 16, 8, 4, 2, 1 lanes apart,
then the warps in order.  Subnormals, zeros of both signs, infinities and NaN
among the values; vector counts around the four a block; the kernel is compiled
into a program of its own.
"""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "matrix-toolkits-java_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "mixed_ir_phases.cuh"
int main(int argc, char **argv)
{
    const int n = std::atoi(argv[1]), k = std::atoi(argv[2]), G = std::atoi(argv[3]);
    std::vector<float> h((size_t)n * (k + 1));
    if (std::fread(h.data(), sizeof(float), h.size(), stdin) != h.size()) return 1;
    float *v = nullptr;
    double *part = nullptr;
    std::vector<double> out((size_t)k * G);
    if (cudaMalloc(&v, sizeof(float) * h.size()) || cudaMalloc(&part, sizeof(double) * out.size()) ||
        cudaMemcpy(v, h.data(), sizeof(float) * h.size(), cudaMemcpyHostToDevice))
        return 2;
    mtjg::k_ir_vdot<<<dim3(G, (k + mtjg::kIrDots - 1) / mtjg::kIrDots), mtjg::kIrBlock>>>(n, v, n, k, v + (size_t)n * k, part);
    if (cudaMemcpy(out.data(), part, sizeof(double) * out.size(), cudaMemcpyDeviceToHost)) return 3;
    std::fwrite(out.data(), sizeof(double), out.size(), stdout);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("dots")
    (d / "dots.cu").write_text(PROGRAM)
    subprocess.run([os.path.join(CUDA, "bin", "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o", str(d / "dots"),
                    str(d / "dots.cu")], check=True)
    return str(d / "dots")


def _expected(V, w, G):
    k, n = V.shape
    steps = -(-n // (G * 256))
    prod = np.zeros((k, steps * G * 256))
    with np.errstate(all="ignore"):
        prod[:, :n] = V.astype(np.float64) * w.astype(np.float64)
        has = np.arange(steps * G * 256).reshape(steps, G, 256) < n
        prod = prod.reshape(k, steps, G, 256)
        acc = np.zeros((k, G, 256))
        for s in range(steps):
            acc = np.where(has[s], acc + prod[:, s], acc)
        acc = acc.reshape(k, G, 8, 32)
        for o in (16, 8, 4, 2, 1):
            acc = acc[..., :o] + acc[..., o:2 * o]
        out = np.zeros((k, G))
        for q in range(8):
            out = out + acc[:, :, q, 0]
    return out


@pytest.mark.parametrize("special", [False, True], ids=["plain", "special"])
@pytest.mark.parametrize("n,k,G", [(1, 1, 1), (255, 3, 2), (257, 4, 2), (1000, 5, 3), (5000, 8, 3), (5000, 9, 7), (70001, 31, 16)])
def test_bits(program, n, k, G, special):
    rng = np.random.default_rng(n + k)
    V = (rng.uniform(-1, 1, (k + 1, n)) * 2.0 ** rng.integers(-20, 20, (k + 1, n))).astype(np.float32)
    if special:
        V = np.where(rng.random(V.shape) < 0.3, (V.astype(np.float64) * 2.0**-135).astype(np.float32), V)  # subnormals
        V = np.where(rng.random(V.shape) < 0.1, np.where(rng.random(V.shape) < 0.5, -0.0, 0.0).astype(np.float32), V)
        V[0, : n // 2] = np.where(rng.random(n // 2) < 0.01, np.float32(np.finfo(np.float32).max), V[0, : n // 2])
        if k > 1:
            V[1, n // 3] = np.inf
        if k > 2:
            V[2, n // 2] = np.nan
    out = subprocess.run([program, str(n), str(k), str(G)], input=V.tobytes(), check=True, capture_output=True).stdout
    got = np.frombuffer(out, dtype=np.float64).reshape(k, G)
    assert np.array_equal(got, _expected(V[:k], V[k], G), equal_nan=True)
