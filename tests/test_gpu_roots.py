"""GPU: the square root and reciprocal that the FP32 transform forms from an
approximation and one Newton step, against 64 bits: within 2^-23 of the value
for every positive normal argument with a normal reciprocal."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "lgpu_f32x2.cuh"
__global__ void k(const float *x, int n, float *s, float *r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { s[i] = lgpu::sqrt_pos(x[i]); r[i] = lgpu::rcp_pos(x[i]); }
}
extern "C" int roots(const float *x, int n, float *s, float *r) {
  float *d = nullptr;
  const size_t b = sizeof(float) * (size_t)n;
  cudaError_t e = cudaMalloc(&d, 3 * b);
  if (e != cudaSuccess) return (int)e;
  e = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) { k<<<(n + 255) / 256, 256>>>(d, n, d + n, d + 2 * (size_t)n); e = cudaGetLastError(); }
  if (e == cudaSuccess) e = cudaMemcpy(s, d + n, b, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(r, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


def test_roots(tmp_path):
    from letkf_gb300 import _build
    (tmp_path / "roots.cu").write_text(SOURCE)
    lib = str(tmp_path / "roots.so")
    subprocess.check_call([_build._nvcc(), *_build.NVCC_FLAGS, "-shared", "-o", lib, str(tmp_path / "roots.cu")])
    rng = np.random.default_rng(7)
    # every mantissa of two octaves (the square root's period), and random ones over the range
    dense = np.arange(0x3F800000, 0x40800000, dtype=np.uint32).view(np.float32)
    wide = (rng.uniform(1.0, 2.0, 4 << 20) * 2.0 ** rng.integers(-126, 126, 4 << 20)).astype(np.float32)
    edge = np.array([2.0 ** -126, 2.0 ** 126, 1.0, np.nextafter(np.float32(1), np.float32(0))], np.float32)
    x = np.concatenate([dense, wide, edge])
    s, r = np.empty_like(x), np.empty_like(x)
    fp = ctypes.POINTER(ctypes.c_float)
    f = ctypes.CDLL(lib).roots
    assert f(x.ctypes.data_as(fp), len(x), s.ctypes.data_as(fp), r.ctypes.data_as(fp)) == 0
    x64 = x.astype(np.float64)
    assert np.abs(s / np.sqrt(x64) - 1.0).max() <= 2.0 ** -23
    assert np.abs(r * x64 - 1.0).max() <= 2.0 ** -23
