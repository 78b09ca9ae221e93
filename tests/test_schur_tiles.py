"""The ordinary Schur assembly of one block, H = [<A_a, G^-1 A_b G^-1>], against numpy at the edges of its
32 x 32 tiles and 32-row chunks and for every number of CTAs that share a tile's rows (1, 2, 4, 8)."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("n,k", [(1, 1), (7, 5), (8, 33), (15, 31), (16, 32), (16, 65), (22, 64), (23, 33), (32, 97),
                                 (45, 40), (63, 31), (64, 130), (64, 700)])
def test_schur_of_one_dense_block(n, k):
    """Sums of n, n and n(n+1)/2 terms: off by at most their lengths times eps times the product of norms."""
    rng = np.random.default_rng(64 * n + k)
    t = n * (n + 1) // 2
    A = rng.standard_normal((t, k))
    Ri = rng.standard_normal((n, n))
    ctx = KernelContext()
    ctx.upload(sp.csc_matrix(A), [n])
    ctx.set_scaling([np.linalg.inv(Ri)], [Ri])
    H = ctx.schur()
    G = Ri.T @ Ri
    i, j = np.array([(i, j) for j in range(n) for i in range(j + 1)]).T
    w = np.where(i == j, 1.0, np.sqrt(2.0))
    X = np.zeros((k, n, n))
    X[:, i, j] = X[:, j, i] = (A / w[:, None]).T
    T = np.einsum("ab,kbc,cd->kad", G, X, G, optimize=True)
    want = A.T @ (T[:, i, j] * w).T
    bound = 4 * (t + 2 * n) * EPS * np.linalg.norm(G) ** 2 * np.outer(*2 * (np.linalg.norm(A, axis=0),))
    assert np.all(np.abs(H - want) <= bound)
    assert np.array_equal(H, H.T)


@pytest.mark.parametrize("k,bad", [(1, 0), (33, 32), (64, 0), (70, 69), (70, 31)])
def test_one_non_finite_entry_is_found(k, bad):
    """Column `bad` overflows only against itself: one infinite entry, on the diagonal, in any tile."""
    A = np.random.default_rng(k).standard_normal((10, k))
    A[:, bad] *= 1e200
    ctx = KernelContext()
    ctx.upload(sp.csc_matrix(A), [4])
    ctx.identity_scaling()
    with pytest.raises(Exception, match="non-finite"):
        ctx.schur()
    A[:, bad] /= 1e200
    ctx.upload(sp.csc_matrix(A), [4])
    ctx.identity_scaling()
    assert np.all(np.isfinite(ctx.schur()))
