"""fast_rcp (rg_device.cuh) against CUDA's division."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from recurgreen_gb300 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "rg_device.cuh"
__global__ void both(const double* x, double* fast, double* div, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fast[i] = rg::fast_rcp(x[i]);
  div[i] = 1.0 / x[i];
}
extern "C" int run(const double* x, double* fast, double* div, int n) {
  double* d = nullptr;
  const size_t b = sizeof(double) * n;
  if (cudaMalloc((void**)&d, 3 * b) != cudaSuccess) return 1;
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  both<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n);
  cudaMemcpy(fast, d + n, b, cudaMemcpyDeviceToHost);
  cudaMemcpy(div, d + 2 * n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return cudaGetLastError() != cudaSuccess;
}
"""


def test_within_one_ulp_of_the_division(tmp_path):
    (tmp_path / "rcp.cu").write_text(SRC)
    so = str(tmp_path / "rcp.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC,
                    str(tmp_path / "rcp.cu"), "-o", so], check=True)
    r = np.random.default_rng(3)
    n = 1 << 18
    x = np.ldexp(1 + r.random(n), r.integers(-1021, 1021, n)) * r.choice([-1.0, 1.0], n)
    x[:6] = (1.0, 2.0, 1e-300, 1e300, np.nextafter(2.0, 1.0), np.nextafter(1.0, 2.0))
    fast, div = np.empty(n), np.empty(n)
    f = ctypes.CDLL(so).run
    f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]
    assert f(x.ctypes.data, fast.ctypes.data, div.ctypes.data, n) == 0
    assert np.all(np.abs(fast - div) <= np.spacing(np.abs(div)))
