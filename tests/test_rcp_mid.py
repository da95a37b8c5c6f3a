"""rcp_mid (lux_b200/csrc/common.cuh) against the correctly rounded reciprocal, for every float of its range: both signs, all
mantissas, the exponents of 2^-125 <= |b| < 2^125."""
import ctypes
import os
import subprocess

import pytest

SOURCE = r"""
#include "common.cuh"
__global__ void k_compare(unsigned long long* differ) {
  unsigned long long n = 0;
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < 1u << 23; m += gridDim.x * blockDim.x)
    for (uint32_t e = 2; e <= 251; e++)
      for (uint32_t sign = 0; sign < 2; sign++) {
        const float b = __uint_as_float(sign << 31 | e << 23 | m);
        n += __float_as_uint(lux::rcp_mid(b)) != __float_as_uint(__frcp_rn(b));
      }
  atomicAdd(differ, n);
}
extern "C" int compare(unsigned long long* differ) {
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, sizeof *d) != cudaSuccess || cudaMemset(d, 0, sizeof *d) != cudaSuccess) return 1;
  k_compare<<<148 * 8, 256>>>(d);
  if (cudaMemcpy(differ, d, sizeof *d, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  return cudaFree(d) == cudaSuccess ? 0 : 3;
}
"""


@pytest.mark.gpu
def test_every_float_of_the_range(tmp_path):
    from lux_b200 import build
    src, lib = tmp_path / "rcp_mid.cu", tmp_path / "rcp_mid.so"
    src.write_text(SOURCE)
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xptxas", "-v")]
    subprocess.run([build.nvcc()] + flags + ["-I", build.CSRC, "-shared", "-o", os.fspath(lib), os.fspath(src)], check=True)
    differ = ctypes.c_ulonglong(1)
    assert ctypes.CDLL(os.fspath(lib)).compare(ctypes.byref(differ)) == 0
    assert differ.value == 0
