"""The FP64 solver's reciprocal (recip, flux_kernel.cuh) against exact
rational arithmetic: within two units in the last place, as its comment says,
so |r x - 1| <= 2^-51, over the range of 1 - R rho and far beyond it."""
import ctypes as C
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

from socrates_gb300 import build as B

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include "flux_kernel.cuh"
__global__ void run(const double *x, double *y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = socgpu::recip(x[i]);
}
extern "C" __attribute__((visibility("default"))) int recips(const double *x, double *y, int n) {
  double *dx = nullptr, *dy = nullptr;
  int bad = cudaMalloc(&dx, 8 * n) != cudaSuccess || cudaMalloc(&dy, 8 * n) != cudaSuccess;
  if (!bad) {
    bad = cudaMemcpy(dx, x, 8 * n, cudaMemcpyHostToDevice) != cudaSuccess;
    run<<<(n + 255) / 256, 256>>>(dx, dy, n);
    bad = bad || cudaMemcpy(y, dy, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess;
  }
  cudaFree(dx);
  cudaFree(dy);
  return bad;
}
"""


@pytest.fixture(scope="module")
def recips(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("recip")
    (d / "recip.cu").write_text(PROGRAM)
    subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "-O3", "-shared", "-Xcompiler", "-fPIC", f"-I{B.INCLUDE}", f"-I{B.CSRC}",
                    str(d / "recip.cu"), "-o", str(d / "recip.so")], check=True, capture_output=True)
    lib = C.CDLL(str(d / "recip.so"))

    def call(x):
        x = np.ascontiguousarray(x, np.float64)
        y = np.empty_like(x)
        assert lib.recips(C.c_void_p(x.ctypes.data), C.c_void_p(y.ctypes.data), C.c_int(x.size)) == 0
        return y
    return call


def test_two_units_in_the_last_place(recips):
    rng = np.random.default_rng(7)
    eps = 2.0 ** -52
    x = np.concatenate([
        rng.uniform(0.0, 2.0, 8000),
        2.0 ** rng.uniform(-52.0, 1.0, 8000),                 # nearly conservative layers between bright ones
        1.0 - eps * np.arange(0.0, 200.0), 1.0 + eps * np.arange(0.0, 200.0),
        eps * np.arange(1.0, 200.0), 2.0 ** np.arange(-60.0, 61.0),
        -(2.0 ** rng.uniform(-40.0, 40.0, 2000)), 2.0 ** rng.uniform(-900.0, 900.0, 2000)])
    y = recips(x)
    worst = max(abs(Fraction(float(a)) * Fraction(float(b)) - 1) for a, b in zip(x, y))
    assert worst <= Fraction(1, 2 ** 51), float(worst)
