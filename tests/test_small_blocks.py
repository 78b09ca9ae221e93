"""Problems of many small blocks: the one-CTA congruences against the clusters (the same chains of products,
so the same bits), the Schur complement of tiny blocks, and the block kernels on shared memory full of
another kernel's NaNs (their padding ends at the next multiple of eight rows)."""
import ctypes as C
import shutil
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200 import problems as P
from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _tri(n):
    return n * (n + 1) // 2


def _context(orders, m, rng):
    t = sum(_tri(n) for n in orders)
    A = rng.standard_normal((t, m))
    ctx = KernelContext()
    ctx.upload(sp.csc_matrix(A), orders)
    return ctx, A


def _interior(orders, rng):
    def spd(n):
        B = rng.standard_normal((n, n))
        return B @ B.T / n + 0.1 * np.eye(n)
    return tuple(np.concatenate([P.svec(spd(n)) for n in orders]) for _ in range(2))


@pytest.mark.parametrize("orders", [list(range(1, 17)), [16] * 3, [1] * 90, [n for n in range(1, 49)] * 2, [48] * 75,
                                    [64, 57, 3] * 25], ids=["1-16", "16", "1s", "1-48", "48s", "64s"])
def test_congruences_do_not_depend_on_the_launch(orders):
    """The same blocks together (one CTA each) and in groups with a block of order 64 (clusters, at most 64)."""
    rng = np.random.default_rng(len(orders))
    R = [rng.standard_normal((n, n)) for n in orders]
    Ri = [rng.standard_normal((n, n)) for n in orders]
    x = [rng.standard_normal(_tri(n)) for n in orders]

    def apply(part, extra):
        ctx, _ = _context([orders[j] for j in part] + [64] * extra, 1, rng)
        ctx.set_scaling([R[j] for j in part] + [np.eye(64)] * extra, [Ri[j] for j in part] + [np.eye(64)] * extra)
        v = np.concatenate([x[j] for j in part] + [np.zeros(_tri(64))] * extra)
        return [ctx.cone_apply(op, v)[:sum(_tri(orders[j]) for j in part)] for op in range(6)]
    groups = [range(k, min(k + 60, len(orders))) for k in range(0, len(orders), 60)]
    want = [np.concatenate(parts) for parts in zip(*(apply(g, 1) for g in groups))]
    for a, b in zip(apply(range(len(orders)), 0), want):
        assert np.all(np.isfinite(a)) and np.array_equal(a, b)


@pytest.mark.parametrize("orders,m", [([1] * 70, 9), ([2] * 40, 33), ([3, 1, 7] * 12, 40), ([8] * 20, 65), ([9, 16] * 3, 70)])
def test_schur_of_small_blocks(orders, m):
    """H = A' Hs^-1 A against numpy: sums of all rows' products, 4 rows eps |A|^2 |G|^2 allowed."""
    rng = np.random.default_rng(m)
    ctx, A = _context(orders, m, rng)
    R = [np.linalg.qr(rng.standard_normal((n, n)))[0] * rng.uniform(0.5, 2.0, n) for n in orders]
    Ri = [np.linalg.inv(r) for r in R]
    ctx.set_scaling(R, Ri)
    H = ctx.schur()
    T, row = np.empty_like(A), 0
    for n, ri in zip(orders, Ri):
        G = ri.T @ ri
        for c in range(m):
            T[row:row + _tri(n), c] = P.svec(G @ P.smat(A[row:row + _tri(n), c], n) @ G)
        row += _tri(n)
    g = max(np.linalg.norm(ri, 2) for ri in Ri) ** 2
    a = np.max(np.linalg.norm(A, axis=0))
    assert np.array_equal(H, H.T)
    assert np.max(np.abs(H - A.T @ T)) <= 4 * A.shape[0] * EPS * (a * g) ** 2


@pytest.mark.parametrize("orders,m", [([50], k) for k in (1, 15, 16, 17, 63, 64, 65, 112, 127, 128, 129, 191, 250)]
                         + [([33] * 35, 7), ([8] * 400, 33), ([1] * 700, 5)])
def test_constraint_products(orders, m):
    """A x and A' z through the residual with zero right-hand sides and the identity scaling: columns at the
    edges of the forward product's rounds of loads, and more tiles than its sixteen-warp form takes."""
    rng = np.random.default_rng(m)
    ctx, A = _context(orders, m, rng)
    ctx.identity_scaling()
    x, z = rng.standard_normal(m), rng.standard_normal(A.shape[0])
    ex, ez, _ = ctx.residual(np.zeros(m), np.zeros(A.shape[0]), x, z)
    assert np.all(np.abs(-ex - A.T @ z) <= 4 * A.shape[0] * EPS * (np.abs(A.T) @ np.abs(z)))
    assert np.all(np.abs(ez - (z - A @ x)) <= 4 * (m + 8) * EPS * (np.abs(A) @ np.abs(x) + 2 * np.abs(z).max()))


POISON = r"""
#include <cuda_runtime.h>
__global__ void k_poison(int words) {
  extern __shared__ double sm[];
  for (int i = threadIdx.x; i < words; i += blockDim.x) sm[i] = __longlong_as_double(0x7ff8000000000001LL);
  __syncthreads();
  if (sm[words - 1 - (int)threadIdx.x] == 1.0) sm[0] = 0.0;  // never: keeps the stores
}
extern "C" int poison() {
  int bytes = 0, sms = 0;
  cudaDeviceGetAttribute(&bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, 0);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
  cudaFuncSetAttribute(k_poison, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  k_poison<<<sms, 1024, bytes>>>(bytes / 8);
  return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def poison(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("poison")
    (d / "p.cu").write_text(POISON)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", str(d / "p.cu"), "-o", str(d / "p.so")], check=True)
    return C.CDLL(str(d / "p.so")).poison


@pytest.mark.parametrize("orders", [[1], [2], [5], [7, 8, 9], [12], [17, 23], [25, 31, 33], [41], [49, 57], [60, 64],
                                    list(range(1, 65))], ids=str)
def test_no_stale_shared_memory(orders, poison):
    rng = np.random.default_rng(sum(orders))
    ctx, A = _context(orders, 12, rng)
    s, z = _interior(orders, rng)
    dz, ds = (np.concatenate([P.svec((lambda E: E + E.T)(rng.standard_normal((n, n)))) for n in orders])
              for _ in range(2))
    bx, bz = rng.standard_normal(12), rng.standard_normal(A.shape[0])

    def run(before):
        out = []
        for call in (lambda: ctx.nt_scale(s, z), lambda: ctx.step_length(dz, ds, 1e3),
                     lambda: ctx.step_length(1e-9 * dz, 1e-9 * ds, 1.0), lambda: [ctx.schur()],
                     lambda: [ctx.factor(1e-8)], lambda: ctx.kkt_solve(bx, bz)):
            before()
            out += list(call())
        for op in range(6):
            before()
            out.append(ctx.cone_apply(op, s))
        return out
    want = run(lambda: None)
    for w, g in zip(want, run(lambda: poison())):
        assert np.all(np.isfinite(w)) and np.array_equal(w, g)
