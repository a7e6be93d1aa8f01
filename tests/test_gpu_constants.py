"""The gate units' division by constants (a product with a reciprocal in two floats) against the IEEE division by the
constant as a float, which is what the reference's arithmetic holds."""
import ctypes
import subprocess

import numpy as np
import pytest

from infoli_gb300 import build as B

pytestmark = pytest.mark.gpu

CONSTANTS = (13.9, 5.0, 4.2, 8.5, 30.0, 7.3, 5.5, 5.8, 33.0, 10.0, 12.0, 900.0)
SOURCE = r"""
#include "infoli_cell.cuh"
__global__ void run(const float* x, float* q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  using namespace infoli;
  float* o = q + i;
%s}
extern "C" int divide(const float* x, float* q, int n, int constants) {
  float *dx, *dq;
  if (cudaMalloc(&dx, n * sizeof(float)) != cudaSuccess || cudaMalloc(&dq, (size_t)n * constants * sizeof(float)) != cudaSuccess)
    return 1;
  cudaMemcpy(dx, x, n * sizeof(float), cudaMemcpyHostToDevice);
  run<<<(n + 255) / 256, 256>>>(dx, dq, n);
  cudaMemcpy(q, dq, (size_t)n * constants * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dq);
  return cudaGetLastError() != cudaSuccess;
}
""" % "".join(f"  o[(size_t){k} * n] = INFOLI_OVER(x[i], {c!r});\n" for k, c in enumerate(CONSTANTS))


def test_division_by_the_float_constants(tmp_path):
    (tmp_path / "over.cu").write_text(SOURCE)
    subprocess.run(["nvcc", *B.ARCH, "-O3", "-std=c++17", "-I", B.SRC, "-I", B.INC, "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(tmp_path / "over.so"), str(tmp_path / "over.cu")], check=True)
    lib, n = ctypes.CDLL(str(tmp_path / "over.so")), 1 << 20
    x = np.random.default_rng(3).uniform(-250, 250, n).astype(np.float32)
    x[:6] = (0.0, -0.0, np.inf, -np.inf, np.nan, 1e-30)
    q = np.empty((len(CONSTANTS), n), np.float32)
    assert lib.divide(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(q.ctypes.data), n, len(CONSTANTS)) == 0
    for got, c in zip(q, CONSTANTS):
        want = x / np.float32(c)
        special = ~np.isfinite(want)
        assert np.array_equal(got[special], want[special], equal_nan=True)
        # 2^-47 of the result before its one rounding: another float only next to a tie, one in 2^22
        assert np.all(np.abs(got[~special] - want[~special]) <= np.spacing(np.abs(want[~special])))
        assert np.mean(got[~special] != want[~special]) < 1e-5
