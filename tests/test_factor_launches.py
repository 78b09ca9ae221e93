"""The factorisation by launches per tile row and the inverse by levels (k_potrf_diag, k_trsm_panel,
k_syrk_update, k_trtri_diag, k_trinv_level), which matrices above the dataflow launch's tile limit take,
brought down to small ones: odd and even leading dimensions, ragged last tiles, both forms."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _solve(A, orders, b, split):
    ctx = KernelContext()
    ctx.upload(A, orders)
    ctx.set_factor_form(1 if split else 0)
    ctx.identity_scaling()
    H = ctx.schur()
    assert ctx.factor(0.0) == 0
    return H, ctx.solve_many(b)


@pytest.mark.parametrize("m,split", [(m, False) for m in (1, 2, 63, 64, 65, 127, 128, 129, 130, 193, 257, 320, 513, 577)]
                         + [(m, True) for m in (1024, 1027, 1153, 1216)])
def test_factor_and_solve(m, split, monkeypatch):
    """Residual of the refined solve within 4 m eps |H| |x|, as for the dataflow launch, whose solution it
    is to the conditioning: both solve to that residual."""
    blocks = m // 1000 + 1
    t = 48 * 49 // 2 * blocks
    rng = np.random.default_rng(m)
    A = sp.csc_matrix(rng.standard_normal((t, m)) / np.sqrt(t))
    b = rng.standard_normal((m, 2))
    _, x0 = _solve(A, [48] * blocks, b, split)
    monkeypatch.setenv("SDPX_B200_DATAFLOW_TILES", "0")
    H, x = _solve(A, [48] * blocks, b, split)
    norm, inv = np.linalg.norm(H, 2), np.linalg.norm(np.linalg.inv(H), 2)
    for c in range(2):
        bound = 4 * m * EPS * norm * np.linalg.norm(x[:, c])
        assert np.linalg.norm(H @ x[:, c] - b[:, c]) <= bound
        assert np.linalg.norm(x[:, c] - x0[:, c]) <= 2 * inv * bound


def test_a_failed_pivot_is_reported(monkeypatch):
    monkeypatch.setenv("SDPX_B200_DATAFLOW_TILES", "0")
    ctx = KernelContext()
    A = sp.csc_matrix(np.eye(2080)[:, :130])
    ctx.upload(A, [64])
    ctx.identity_scaling()
    ctx.schur()
    assert ctx.factor(-2.0, dynamic=False) != 0
    assert ctx.factor(0.0, dynamic=False) == 0
