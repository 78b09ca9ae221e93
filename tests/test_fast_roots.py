"""recip_mid and rsqrt_mid (csrc/common.cuh) over their whole range against 64-bit-mantissa arithmetic.
Both end in one rounding after a step whose own error is far below it: 2^-53 relative for the reciprocal, and
half of that more for the root, whose step starts from a rounded v y.  2^-52 is allowed."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parent.parent / "sdpx.rs_b200" / "csrc"
SRC = r"""
#include "common.cuh"
__global__ void k_roots(const double* v, int n, double* r, double* q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = recip_mid(v[i]);
  q[i] = rsqrt_mid(v[i]);
}
extern "C" int roots(const double* v, int n, double* r, double* q) {
  double* g = nullptr;
  const size_t b = (size_t)n * sizeof(double);
  if (cudaMalloc(&g, 3 * b) != cudaSuccess) return 1;
  cudaMemcpy(g, v, b, cudaMemcpyHostToDevice);
  k_roots<<<(n + 255) / 256, 256>>>(g, n, g + n, g + 2 * (size_t)n);
  cudaMemcpy(r, g + n, b, cudaMemcpyDeviceToHost);
  cudaMemcpy(q, g + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  cudaFree(g);
  return cudaGetLastError() != cudaSuccess;
}
"""


def test_error_bounds(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "r.cu").write_text(SRC)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "--expt-relaxed-constexpr", "-I", str(CSRC), str(tmp_path / "r.cu"), "-o",
                    str(tmp_path / "r.so")], check=True)
    lib = C.CDLL(str(tmp_path / "r.so"))
    rng = np.random.default_rng(0)
    m = rng.uniform(1.0, 2.0, 1 << 20)
    m[:4] = 1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5
    ex = rng.integers(-1000, 1000, m.size)
    ex[4:2004] = np.arange(-1000, 1000)
    m[4:2004] = rng.choice(m[:4], 2000)
    v = np.ldexp(m, ex)
    r, q, ptr = np.empty_like(v), np.empty_like(v), C.POINTER(C.c_double)
    assert lib.roots(v.ctypes.data_as(ptr), v.size, r.ctypes.data_as(ptr), q.ctypes.data_as(ptr)) == 0
    assert np.finfo(np.longdouble).nmant >= 63
    x = v.astype(np.longdouble)
    for got, want in ((r, 1 / x), (q, 1 / np.sqrt(x))):
        assert float(np.max(np.abs(got.astype(np.longdouble) / want - 1))) <= 2.0 ** -52
