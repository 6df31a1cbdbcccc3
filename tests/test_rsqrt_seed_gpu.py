"""Bound of the hardware seed behind the FP64 reciprocal square roots (B200).

rsqrt_f64, inv_cube_f64 and exact_inv rest on the relative error of rsqrt.approx.ftz.f64 staying below
2^-20.  Here it is measured: every high word of two octaves (every mantissa that the instruction sees, both
parities of the exponent) with all-zero and all-one low words, and 4096 mantissas of every exponent that
exact_inv takes without IEEE root and division, [2^-894, 2^897).
"""
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include <cuda_runtime.h>
// err[i] = |s y^2 - 1| / 2 for argument i of n, the relative error of y to first order
__global__ void seed_error(int n, int exponents, double* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s;
    if (exponents) {  // 1791 exponents x 4096 mantissas
        const int e = i / 4096 - 894, m = i % 4096;
        s = ldexp(1.0 + (m + 0.37) / 4096.0, e);
    } else {          // 2^21 high words of [1, 4) x two low words
        s = __hiloint2double(0x3ff00000 + (i >> 1), (i & 1) ? 0xffffffff : 0);
    }
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    err[i] = 0.5 * fabs(fma(-s * y, y, 1.0));
}
int main() {
    for (int mode = 0; mode < 2; ++mode) {
        const int n = mode ? 1791 * 4096 : 1 << 22;
        double* d;
        if (cudaMalloc(&d, n * sizeof(double)) != cudaSuccess) return 1;
        seed_error<<<(n + 255) / 256, 256>>>(n, mode, d);
        std::vector<double> h(n);
        if (cudaMemcpy(h.data(), d, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
        double worst = 0.0;
        for (double v : h) worst = v > worst || v != v ? v : worst;
        std::printf("%.17g\n", worst);
        cudaFree(d);
    }
}
"""


def test_seed_error_stays_below_its_bound(tmp_path):
    src = tmp_path / "seed.cu"
    src.write_text(SOURCE)
    exe = tmp_path / "seed"
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", str(src), "-o", str(exe)], check=True)
    worst = [float(v) for v in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()]
    assert len(worst) == 2
    for w in worst:
        assert w * (1.0 + 2.0**-18) < 2.0**-20  # first order, and the rounding of s y
