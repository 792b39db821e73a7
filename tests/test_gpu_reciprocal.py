"""k_pt2's reciprocal against division, over every exponent that it is used for.

The hardware's approximation r0 is taken to be within 2^-19; r0 (1 + e + e^2)
with e = 1 - d r0 then leaves e^3 < 2^-57, and the last fused operation rounds
once: together less than one unit in the last place."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "pt2_epi.cuh"
using namespace cipsi_dev;
__global__ void k(const double* d, double* r, double* e, int* ok, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double r0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(d[i]));
  e[i] = fma(-d[i], r0, 1.0);
  r[i] = recip(d[i]);
  ok[i] = recip_ok(d[i]);
}
extern "C" int reciprocals(const double* d, double* r, double* e, int* ok, int n) {
  double *dd, *dr, *de;
  int* dk;
  if (cudaMalloc(&dd, n * 8) || cudaMalloc(&dr, n * 8) || cudaMalloc(&de, n * 8) || cudaMalloc(&dk, n * 4)) return 1;
  cudaMemcpy(dd, d, n * 8, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(dd, dr, de, dk, n);
  cudaMemcpy(r, dr, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(e, de, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(ok, dk, n * 4, cudaMemcpyDeviceToHost);
  cudaFree(dd), cudaFree(dr), cudaFree(de), cudaFree(dk);
  return cudaGetLastError();
}
"""


def test_reciprocal_within_an_ulp(tmp_path, engine_lib):
    src, lib = tmp_path / "recip.cu", tmp_path / "recip.so"
    src.write_text(SOURCE)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-shared", "-Xcompiler", "-fPIC", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-gencode", "arch=compute_103a,code=sm_103a", "-I", os.path.join(ROOT, "cipsi_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), str(src), "-o", str(lib)], check=True)
    rng = np.random.default_rng(1)
    field = np.arange(2047)
    mantissa = np.concatenate([[0, 1, 2**52 - 1], rng.integers(0, 2**52, 500)]).astype(np.uint64)
    bits = (field[:, None].astype(np.uint64) << np.uint64(52)) | mantissa[None, :]
    d = bits.ravel().view(np.float64)
    d = np.concatenate([d, -d, [np.inf, -np.inf, np.nan]])
    n = len(d)
    r, e, ok = np.zeros(n), np.zeros(n), np.zeros(n, np.int32)
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (d, r, e, ok)]
    assert ctypes.CDLL(str(lib)).reciprocals(*p, n) == 0
    exponent = (np.abs(d).view(np.uint64) >> np.uint64(52)).astype(int)
    assert np.array_equal(ok != 0, (exponent >= 64) & (exponent < 1984))
    use = ok != 0
    assert np.abs(e[use]).max() < 2.0 ** -19
    want = 1.0 / d[use]
    assert np.array_equal(np.sign(r[use]), np.sign(want))
    assert np.abs(np.abs(r[use]).view(np.int64) - np.abs(want).view(np.int64)).max() <= 1
