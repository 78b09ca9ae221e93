"""Step lengths of single PSD blocks at the identity scaling against numpy's eigenvalues, at the orders
where the tridiagonalisation's register layout changes (the matrix sits in the last n of 64 positions,
four positions per warp and segments of 16) and on matrices whose columns are already reduced."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200 import problems as P
from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _matrix(kind, n, rng):
    if kind == "random":
        X = rng.standard_normal((n, n))
    elif kind == "diagonal":
        X = np.diag(rng.standard_normal(n))
    elif kind == "rank1":
        u = rng.standard_normal(n)
        X = -np.outer(u, u)
    elif kind == "equal":  # one eigenvalue n times
        X = -2.0 * np.eye(n)
    else:  # "graded": columns over 24 orders of magnitude
        g = 10.0 ** (-24.0 * np.arange(n) / max(n - 1, 1))
        X = rng.standard_normal((n, n)) * np.sqrt(np.outer(g, g))
    X = 0.5 * (X + X.T)
    if np.linalg.eigvalsh(X)[0] >= 0.0:
        X = -X
    return X


@pytest.mark.parametrize("kind", ["random", "diagonal", "rank1", "equal", "graded"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 15, 16, 17, 18, 31, 32, 33, 34, 47, 48, 49, 61, 62, 63, 64])
def test_step_length_of_one_block(n, kind):
    """alpha = -1 / lambda_min.  Tridiagonalisation and multisection are backward stable: lambda_min is
    off by at most a small multiple of n eps |X|; 8 n eps |X| / |lambda_min| relative is allowed."""
    rng = np.random.default_rng(1000 * n + len(kind))
    t = n * (n + 1) // 2
    ctx = KernelContext()
    ctx.upload(sp.csc_matrix(np.ones((t, 1))), [n])
    ctx.identity_scaling()
    inert = P.svec(np.eye(n))
    for scale, amax in ((1.0, 1e6), (1e-100, 1e106), (1e100, 1e-90)):
        X = scale * _matrix(kind, n, rng)
        w = np.linalg.eigvalsh(X / scale)
        norm, lo = np.max(np.abs(w)), w[0]
        want = min(amax, -1.0 / (lo * scale))
        for dz, ds in ((P.svec(X), inert), (inert, P.svec(X))):
            got, st = ctx.step_length(dz, ds, amax)
            assert st == 0
            assert abs(got - want) <= 8 * n * EPS * max(1.0, norm / abs(lo)) * want, (n, kind, scale, got, want)
