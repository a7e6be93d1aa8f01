"""The gate units' branch-free reciprocal and quotient against the IEEE operations, over the whole range of normal
numbers and at what their corrections must leave alone (zeros, infinities, NaN, results below the normal range)."""
import ctypes
import subprocess

import numpy as np
import pytest

from infoli_gb300 import build as B

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "infoli_cell.cuh"
__global__ void run(const float* a, const float* b, float* rec, float* quo, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    rec[i] = infoli::recip(b[i]);
    quo[i] = infoli::quotient(a[i], b[i]);
  }
}
extern "C" int divide(const float* a, const float* b, float* rec, float* quo, int n) {
  float* d[4];
  for (auto& p : d)
    if (cudaMalloc(&p, n * sizeof(float)) != cudaSuccess) return 1;
  cudaMemcpy(d[0], a, n * sizeof(float), cudaMemcpyHostToDevice);
  cudaMemcpy(d[1], b, n * sizeof(float), cudaMemcpyHostToDevice);
  run<<<(n + 255) / 256, 256>>>(d[0], d[1], d[2], d[3], n);
  cudaMemcpy(rec, d[2], n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaMemcpy(quo, d[3], n * sizeof(float), cudaMemcpyDeviceToHost);
  for (auto& p : d) cudaFree(p);
  return cudaGetLastError() != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    where = tmp_path_factory.mktemp("division")
    (where / "division.cu").write_text(SOURCE)
    subprocess.run(["nvcc", *B.ARCH, "-O3", "-std=c++17", "-I", B.SRC, "-I", B.INC, "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(where / "division.so"), str(where / "division.cu")], check=True)
    lib = ctypes.CDLL(str(where / "division.so"))

    def call(a, b):
        rec, quo = np.empty_like(a), np.empty_like(a)
        assert lib.divide(*(ctypes.c_void_p(x.ctypes.data) for x in (a, b, rec, quo)), len(a)) == 0
        return rec, quo

    return call


@pytest.mark.parametrize("low,high", [(-0.01, 0.01), (-20, 20), (-60, 60)])
def test_division_is_within_an_ulp_of_ieee(divide, low, high):
    rng = np.random.default_rng(7)
    a, b = ((2.0 ** rng.uniform(low, high, 1 << 20) * rng.choice([-1, 1], 1 << 20)).astype(np.float32) for _ in range(2))
    for got, want in zip(divide(a, b), (1 / b, a / b)):
        assert np.all(np.abs(got.astype(np.float64) - want) <= np.spacing(np.abs(want)))  # one step of the final addition
        assert np.mean(got == want) > 0.9  # each residual is exact: what is left is that addition's own rounding


def test_division_at_zeros_infinities_and_small_results(divide):
    tiny, big = np.finfo(np.float32).tiny, np.finfo(np.float32).max
    edge = np.array([0.0, -0.0, 1.0, -1.0, 0.1, 3e4, np.inf, -np.inf, np.nan, 8e37, -9e37, big, tiny], np.float32)
    a, b = (x.ravel().copy() for x in np.meshgrid(edge, edge))
    # past 8e37 a reciprocal is below the normal range and counts as 0; the reciprocal's operands are never 0
    large = np.abs(b) > 8e37
    rec, quo = divide(a, b)
    with np.errstate(all="ignore"):
        for got, want, ok in ((rec, 1 / b, b != 0), (quo, a / b, ~(large & (np.abs(a) > 3e4)))):
            got, want, small = got[ok], want[ok], large[ok]
            plain = np.isfinite(want)
            assert np.array_equal(got[~plain], want[~plain], equal_nan=True)
            assert np.all(np.abs(got[plain].astype(np.float64) - want[plain])
                          <= np.maximum(np.spacing(np.abs(want[plain])), np.where(small[plain], 3e4 * tiny, 0)))
