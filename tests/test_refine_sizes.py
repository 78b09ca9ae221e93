"""The refined KKT solve's control kernel at the sizes where its copies change (256 entries a pass, 2048 a
round of loads): the graph against the host-driven refinement, bit for bit, with several inner steps
(the factor is that of H + 1e-3 I)."""
import numpy as np
import pytest
import scipy.sparse as sp

from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1793, 2047, 2048, 2049, 4097])
def test_graph_equals_host_driven(n, monkeypatch):
    t = 2080
    blocks = (n + 1) // t + 1
    col = np.arange(n)
    A = sp.csc_matrix((np.r_[1.0 + col / n, np.full(n, 0.3)], (np.r_[col, col + 1], np.r_[col, col])),
                      shape=(t * blocks, n))
    rng = np.random.default_rng(n)
    bx, bz = rng.standard_normal(n), rng.standard_normal(t * blocks)
    outs = []
    for graphs in ("0", "1"):
        monkeypatch.setenv("SDPX_B200_GRAPHS", graphs)
        ctx = KernelContext()
        ctx.upload(A, [64] * blocks)
        ctx.identity_scaling()
        ctx.schur()
        assert ctx.factor(1e-3) == 0
        outs += [ctx.kkt_solve(bx, bz), ctx.kkt_solve(2.0 * bx, bz)]
    for (x, z), (gx, gz) in zip(outs[:2], outs[2:]):
        assert np.array_equal(x, gx) and np.array_equal(z, gz)
    x, z = outs[0]
    ex, ez, norm = ctx.residual(bx, bz, x, z)
    assert norm <= 1e-12 * max(np.max(np.abs(bx)), np.max(np.abs(bz)))
