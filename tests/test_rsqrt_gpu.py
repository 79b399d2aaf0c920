"""rsqrt_normal (csrc/linalg.cuh), which the Cholesky pivots and the Jacobi angles use: within 2 ulp of 1 / sqrt(x) over
the normal range.  The kernel is compiled here and run on every exponent with random mantissas, powers of two and their
neighbours, and a sweep over [1, 4); the reference is x87 extended precision (64-bit mantissa: 2^-11 of an ulp)."""
import ctypes as ct
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = Path(__file__).resolve().parent.parent / "ipeps.jl_b200" / "csrc"

PROGRAM = r"""
#include "linalg.cuh"
__global__ void run(const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = ipeps::rsqrt_normal(x[i]);
}
extern "C" int rsqrt_of(const double* x, double* y, int n) {
  double *dx = nullptr, *dy = nullptr;
  cudaError_t e = cudaMalloc(&dx, size_t(n) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&dy, size_t(n) * 8);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, size_t(n) * 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    run<<<(n + 255) / 256, 256>>>(dx, dy, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(y, dy, size_t(n) * 8, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  return int(e);
}
"""


def test_within_two_ulp(tmp_path):
    src, lib = tmp_path / "r.cu", tmp_path / "r.so"
    src.write_text(PROGRAM)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared", "-I", str(CSRC), str(src), "-o",
                    str(lib)], check=True)
    rng = np.random.default_rng(1)
    e = np.arange(-1022, 1024)
    two = np.ldexp(1.0, e)
    x = np.concatenate([two, np.nextafter(two, np.inf), np.nextafter(two[1:], 0.0), [np.finfo(float).max],
                        np.ldexp(rng.uniform(1.0, 2.0, (200, e.size)), e).ravel(), np.linspace(1.0, 4.0, 1 << 20),
                        rng.uniform(1.0, 4.0, 1 << 20), rng.uniform(0.5, 1.0, 1 << 18)])
    x = np.ascontiguousarray(x[(x >= np.finfo(float).tiny) & np.isfinite(x)])
    y = np.empty_like(x)
    dp = ct.POINTER(ct.c_double)
    assert ct.CDLL(str(lib)).rsqrt_of(x.ctypes.data_as(dp), y.ctypes.data_as(dp), x.size) == 0
    ref = 1 / np.sqrt(x.astype(np.longdouble))
    assert np.finfo(np.longdouble).nmant >= 63
    ulp = np.spacing(ref.astype(float)).astype(np.longdouble)
    err = np.abs(y.astype(np.longdouble) - ref) / ulp
    print("largest error in ulp:", float(err.max()))
    assert err.max() <= 2.0
