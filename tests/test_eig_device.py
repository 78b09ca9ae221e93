"""The shared-memory eigenvalue routines of csrc/eig.cuh by themselves, in a kernel of this test: their
results may depend neither on what another kernel left in the scratch memory nor on the order's place in
the register layout."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = Path(__file__).resolve().parent.parent / "sdpx.rs_b200" / "csrc"
EPS = np.finfo(np.float64).eps
SRC = r"""
#include "eig.cuh"
// out: d[64], e[64], every eigenvalue[64], the smallest, whether that one was found
__global__ void __launch_bounds__(SDPXG_EIG_THREADS)
k_eig(const double* A, int n, double fill, double* out, uint32_t* status) {
  extern __shared__ __align__(16) double sm[];
  double* M = sm;
  double* ws = M + SDPXG_LD * SDPXG_NMAX;
  double* sd = ws + SDPXG_TRIDIAG_WORK;
  double* se = sd + SDPXG_NMAX;
  double* eig = se + SDPXG_NMAX;
  int* best = reinterpret_cast<int*>(eig + SDPXG_NMAX);
  for (int i = threadIdx.x; i < SDPXG_TRIDIAG_WORK + 3 * SDPXG_NMAX; i += blockDim.x) ws[i] = fill;
  cta_load_mat(M, A, n);
  __syncthreads();
  cta_tridiagonalize(M, n, sd, se, ws);
  cta_eig_all(sd, se, n, reinterpret_cast<double2*>(ws), eig, status);
  __syncthreads();
  bool ok;
  const double g = cta_eig_min(sd, se, n, reinterpret_cast<double2*>(ws), best, &ok);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    out[i] = sd[i];
    out[64 + i] = i + 1 < n ? se[i] : 0.0;
    out[128 + i] = eig[i];
  }
  if (threadIdx.x == 0) {
    out[192] = g;
    out[193] = ok;
  }
}
extern "C" int eig(const double* A, int n, double fill, double* out, uint32_t* status) {
  const size_t smem = (SDPXG_LD * SDPXG_NMAX + SDPXG_TRIDIAG_WORK + 3 * SDPXG_NMAX + 1) * sizeof(double);
  double* g = nullptr;
  if (cudaMalloc(&g, (64 * 64 + 200) * sizeof(double)) != cudaSuccess) return 1;
  double* o = g + 64 * 64;
  uint32_t* st = reinterpret_cast<uint32_t*>(o + 199);
  cudaFuncSetAttribute(k_eig, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaMemset(o, 0, 200 * sizeof(double));
  cudaMemcpy(g, A, (size_t)n * n * sizeof(double), cudaMemcpyHostToDevice);
  k_eig<<<1, SDPXG_EIG_THREADS, smem>>>(g, n, fill, o, st);
  cudaMemcpy(out, o, 194 * sizeof(double), cudaMemcpyDeviceToHost);
  cudaMemcpy(status, st, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(g);
  return cudaGetLastError() != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("eig")
    (d / "e.cu").write_text(SRC)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "--expt-relaxed-constexpr", "-I", str(CSRC), str(d / "e.cu"), "-o", str(d / "e.so")],
                   check=True)
    return C.CDLL(str(d / "e.so"))


def run(device, X, fill=0.0):
    """(the 64-entry rows d, e, every eigenvalue), the smallest eigenvalue, whether it was found, the status."""
    X = np.asfortranarray(X)
    out, st, ptr = np.zeros(194), C.c_uint32(), C.POINTER(C.c_double)
    assert device.eig(X.ctypes.data_as(ptr), X.shape[0], C.c_double(fill), out.ctypes.data_as(ptr), C.byref(st)) == 0
    return out[:192].reshape(3, 64), out[192], out[193] == 1.0, st.value


@pytest.mark.parametrize("n", range(1, 65))
def test_no_stale_scratch_is_read(device, n):
    """Every eigenvalue against numpy's: the Householder reduction and the Sturm sequences are backward
    stable, 8 n eps |A| allowed.  Scratch full of NaN, of infinities and of zeros gives the same bits."""
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, n))
    X = 0.5 * (X + X.T)
    rows, low, ok, st = run(device, X)
    w = np.linalg.eigvalsh(X)
    assert ok and st == 0
    bound = 8 * n * EPS * np.max(np.abs(w))
    assert np.max(np.abs(rows[2, :n] - w)) <= bound and abs(low - w[0]) <= bound
    for fill in (float("nan"), float("inf")):
        got = run(device, X, fill)
        assert np.array_equal(got[0], rows) and got[1:] == (low, ok, st)


@pytest.mark.parametrize("n", [1, 2, 8, 33, 64])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
def test_a_matrix_that_is_not_finite_is_reported(device, n, value):
    X = np.eye(n)
    X[n - 1, n // 2] = X[n // 2, n - 1] = value
    _, _, ok, st = run(device, X)
    assert not ok and st != 0


@pytest.mark.parametrize("n", [2, 3, 4, 9, 17, 33, 64])
@pytest.mark.parametrize("size", [1e-18, 1e-30, 1e-40, 1e-55])
@pytest.mark.parametrize("kind", ["diagonal", "block"])
def test_eigenvalues_far_below_the_norm(device, kind, size, n):
    """A small block beside a large entry, without coupling: its eigenvalues are found to their own rounding
    (8 n eps of the block's norm), wherever the block stands."""
    rng = np.random.default_rng(n)
    B = np.diag(np.r_[1.0, 1.0, rng.uniform(1.0, 2.0, n)][:n - 1])
    if kind == "block":
        B = rng.standard_normal((n - 1, n - 1))
        B = B @ B.T + np.eye(n - 1)
    for at in (0, n - 1):
        for sign in (1.0, -1.0):
            X = np.zeros((n, n))
            X[at, at] = 1.0
            keep = np.arange(n) != at
            X[np.ix_(keep, keep)] = sign * size * B
            w = sign * size * np.linalg.eigvalsh(B)
            rows, low, ok, st = run(device, X)
            assert ok and st == 0
            got = np.sort(rows[2, :n])[:-1]
            bound = 8 * n * EPS * size * np.linalg.norm(B, 2)
            assert np.max(np.abs(got - np.sort(w))) <= bound and abs(low - np.min(w)) <= bound
