"""Factor, explicit inverse and column-dot solves of the Schur complement at the edges of the 64 x 64
tiles, of the inverse's lag behind the factor (8 tile rows) and of the column dots' row groups."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("m", [1, 2, 63, 64, 65, 127, 128, 129, 130, 191, 193, 257, 320, 449, 511, 512, 513, 577, 640])
def test_factor_and_solve(m):
    """Residual of the refined solve within 4 m eps |H| |x| (a backward stable solve: a small multiple of
    eps |H| |x| per row), and the right-hand sides' columns do not mix."""
    n = 48
    t = n * (n + 1) // 2
    rng = np.random.default_rng(m)
    A = rng.standard_normal((t, m)) / np.sqrt(t)
    ctx = KernelContext()
    ctx.upload(sp.csc_matrix(A), [n])
    ctx.identity_scaling()
    H = ctx.schur()
    assert ctx.factor(0.0) == 0
    b = rng.standard_normal((m, 3))
    x = ctx.solve_many(b)
    norm = np.linalg.norm(H, 2)
    for c in range(3):
        r = np.linalg.norm(H @ x[:, c] - b[:, c])
        assert r <= 4 * m * EPS * norm * np.linalg.norm(x[:, c]), (m, c, r)
    assert np.array_equal(ctx.solve_many(b[:, 1:2])[:, 0], x[:, 1])
