"""The error that a launch reports is the first one that a CTA recorded, in the host's word as in the device's."""
import ctypes
import subprocess

import pytest

from infoli_gb300 import build as B

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "infoli_kernels.cuh"
__global__ void record(infoli::StepArgs a) {  // every thread an error of its own
  infoli::device_error(a, 1 + (int)(blockIdx.x * blockDim.x + threadIdx.x));
}
extern "C" int record_errors(int blocks, int threads, int* words) {  // {device word, host word}
  infoli::StepArgs a = {};
  if (cudaMalloc(&a.err, sizeof(int)) != cudaSuccess || cudaMallocHost(&a.err_host, sizeof(int)) != cudaSuccess) return 1;
  cudaMemset(a.err, 0, sizeof(int));
  *a.err_host = 0;
  record<<<blocks, threads>>>(a);
  cudaMemcpy(words, a.err, sizeof(int), cudaMemcpyDeviceToHost);
  words[1] = *a.err_host;
  cudaFree(a.err);
  cudaFreeHost(a.err_host);
  return cudaGetLastError() != cudaSuccess;
}
"""


def test_the_first_error_stands_in_both_words(tmp_path):
    (tmp_path / "error.cu").write_text(SOURCE)
    subprocess.run(["nvcc", *B.ARCH, "-O3", "-std=c++17", "-I", B.SRC, "-I", B.INC, "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(tmp_path / "error.so"), str(tmp_path / "error.cu")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "error.so"))
    words = (ctypes.c_int * 2)()
    for blocks, threads in ((1, 1), (1, 32), (152, 256)):
        assert lib.record_errors(blocks, threads, words) == 0
        assert words[0] == words[1] > 0
