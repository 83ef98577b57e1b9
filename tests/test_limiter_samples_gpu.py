"""The adjoint's reconstruction (s2_companion3_x) takes the face values that the forward's limiter saw, bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from ugks2d_high_order_b200.build import ARCH, CSRC, NVCC, ROOT

MAIN = r"""
#include <cstdio>
#include <vector>
#include "ugks_s2_math.cuh"
using namespace ugks;
__global__ void k(int n, const double* q, double* o) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double a[5], b[5], f[3], d[3], c[3], g[3];
    for (int m = 0; m < 5; ++m) { a[m] = q[10 * t + m]; b[m] = q[10 * t + 5 + m]; }
    S2Weno w;
    S2WenoX x;
    s2_power_companion3(a, b, f, d, c);
    s2_companion3_x(a, b, g, d, c, w, x);
    for (int m = 0; m < 3; ++m) { o[6 * t + m] = f[m]; o[6 * t + 3 + m] = g[m]; }
}
int main(int, char** argv) {
    const int n = 4096;
    std::vector<double> q(10 * n), o(6 * n);
    FILE* f = std::fopen(argv[1], "rb");
    if (!f || std::fread(q.data(), 8, q.size(), f) != q.size()) return 2;
    std::fclose(f);
    double *dq, *d;
    if (s2_upload_tables() != cudaSuccess || cudaMalloc(&dq, q.size() * 8) != cudaSuccess || cudaMalloc(&d, o.size() * 8) != cudaSuccess) return 3;
    cudaMemcpy(dq, q.data(), q.size() * 8, cudaMemcpyHostToDevice);
    k<<<n / 128, 128>>>(n, dq, d);
    if (cudaMemcpy(o.data(), d, o.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 4;
    f = std::fopen(argv[2], "wb");
    return f && std::fwrite(o.data(), 8, o.size(), f) == o.size() && std::fclose(f) == 0 ? 0 : 5;
}
"""


@pytest.mark.gpu
def test_limiter_samples(tmp_path):
    """Stencils of one size and with neighbours up to 1e40 times the mean, as in the tails of the distribution."""
    if shutil.which(NVCC) is None:
        pytest.skip("no nvcc")
    (tmp_path / "t.cu").write_text(MAIN)
    exe = str(tmp_path / "t")
    subprocess.run([NVCC] + ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                                    "-o", exe, str(tmp_path / "t.cu")], check=True)
    rng = np.random.default_rng(0)
    q = rng.uniform(0.1, 1, (4096, 10))
    q[1024:] *= 10.0 ** rng.uniform(-40, 0, (3072, 10))
    q.tofile(tmp_path / "q")
    subprocess.run([exe, str(tmp_path / "q"), str(tmp_path / "o")], check=True)
    o = np.fromfile(tmp_path / "o").reshape(4096, 2, 3)
    assert np.isfinite(o).all() and np.array_equal(o[:, 0], o[:, 1])
