"""A residual of NaNs is not a small one: the largest magnitude of a vector with a NaN is NaN in every
reduction, so a solve whose residual overflowed to Inf - Inf reports failure as the oracle's does
(numpy's max keeps NaN too) instead of returning as converged."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200 import _lib
from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu


def _context():
    """H = 1e6 [[1, 1 - d], [1 - d, 1]] with d = 1e-9: for the right-hand side 1e300 (1, -1) the solution is
    finite, 1e303 (1, -1), and both rows of H x are Inf - Inf."""
    d = 1e-9
    a = 1e3 * np.array([[1.0, 1.0 - d], [0.0, np.sqrt(2.0 * d - d * d)], [0.0, 0.0]])
    ctx = KernelContext()
    ctx.upload(sp.csc_matrix(a), [2])
    ctx.identity_scaling()
    ctx.schur()
    assert ctx.factor(0.0, dynamic=False) == 0
    return ctx


RHS = 1e300 * np.array([1.0, -1.0])


def test_reduced_solve():
    ctx = _context()
    assert np.allclose(ctx.solve_many(RHS * 1e-290)[:, 0], [1e13, -1e13], rtol=1e-5)
    with pytest.raises(_lib.SdpxError):
        ctx.solve_many(RHS)


@pytest.mark.parametrize("graphs", ["0", "1"])
def test_kkt_solve(graphs, monkeypatch):
    monkeypatch.setenv("SDPX_B200_GRAPHS", graphs)
    ctx = _context()
    ctx.kkt_solve(RHS * 1e-290, np.zeros(3))
    with pytest.raises(_lib.SdpxError):
        ctx.kkt_solve(RHS, np.zeros(3))


def test_noalloc_solve():
    import torch

    ctx = _context()
    d = torch.from_numpy(RHS.copy()).cuda()
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    assert _lib.load().sdpxg_solve_noalloc(ctx._h, C.c_void_p(d.data_ptr()), C.c_void_p(out.data_ptr()), 1) != 0


@pytest.mark.parametrize("where", [0, 1])
def test_residual_norm(where):
    ctx = _context()
    bx, bz = np.ones(2), np.ones(3)
    (bx, bz)[where][1] = np.nan
    assert np.isnan(ctx.residual(bx, bz, np.ones(2), np.ones(3))[2])
