"""The per-block cone kernels against numpy at the orders where their layouts change: the NT scaling
(4, 8 or 16 rows per Jacobi warp, 8 x 8 tiles, two-row Cholesky lanes) and the congruences (a cluster of
four CTAs, CTA J with the tile columns J and 7 - J)."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200 import problems as P
from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps
ORDERS = [1, 2, 3, 7, 8, 9, 15, 16, 17, 24, 25, 31, 32, 33, 40, 41, 48, 56, 57, 63, 64]


def _context(n):
    ctx = KernelContext()
    ctx.upload(sp.csc_matrix(np.ones((n * (n + 1) // 2, 1))), [n])
    return ctx


def _smat(v, n):
    X = np.zeros((n, n))
    e = 0
    for j in range(n):
        for i in range(j + 1):
            X[i, j] = X[j, i] = v[e] / (1.0 if i == j else np.sqrt(2.0))
            e += 1
    return X


@pytest.mark.parametrize("n", ORDERS)
def test_nt_scale_of_one_block(n):
    """lambda against the eigenvalues of L1' Z L1 at 1e-12 (conditions of a few hundred), again with S and Z
    scaled so far apart that every Cholesky pivot leaves the range of the fast root, and a failure for
    an indefinite S."""
    rng = np.random.default_rng(n)
    S, Z = ((lambda B: B @ B.T / n + 0.1 * np.eye(n))(rng.standard_normal((n, n))) for _ in range(2))
    L = np.linalg.cholesky(S)
    want = np.sqrt(np.sort(np.linalg.eigvalsh(L.T @ Z @ L))[::-1])
    for power in (0, 1008):
        ctx = _context(n)
        lam, status = ctx.nt_scale(P.svec(np.ldexp(S, -power)), P.svec(np.ldexp(Z, power)))
        assert status == 0
        assert np.allclose(lam, want, rtol=1e-12, atol=0)
    ctx = _context(n)
    bad = S.copy()
    bad[n - 1, n - 1] = -1.0
    _, status = ctx.nt_scale(P.svec(bad), P.svec(Z))
    assert status != 0


@pytest.mark.parametrize("n", ORDERS)
def test_congruences_of_one_block(n):
    """W x, W'x, W^-1 x, W^-T x and the two-congruence Hs x, Hs^-1 x.  A product of n-term sums is off by
    at most n eps times the product of the norms; two (four) products, doubled."""
    rng = np.random.default_rng(100 + n)
    R, Ri = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    X = rng.standard_normal((n, n))
    X = X + X.T
    ctx = _context(n)
    ctx.set_scaling([R], [Ri])
    a, b, x = np.linalg.norm(R), np.linalg.norm(Ri), np.linalg.norm(X)
    W, Wi = R.T @ X @ R, Ri @ X @ Ri.T
    want = {0: (W, a ** 2), 1: (R @ X @ R.T, a ** 2), 2: (Ri.T @ X @ Ri, b ** 2), 3: (Wi, b ** 2),
            4: (R @ W @ R.T, a ** 4), 5: (Ri.T @ Wi @ Ri, b ** 4)}
    for op, (Y, scale) in want.items():
        got = _smat(ctx.cone_apply(op, P.svec(X)), n)
        assert np.max(np.abs(got - Y)) <= 8 * n * EPS * scale * x, (n, op)
