"""Exact products at every limb count: each picks its own width of the residue kernel (words of the
mantissa) and of the CRT (digits of the prime product), at spreads that move the prime count too."""
import pytest

from oracle import exact as X

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("spread", [2, 300])
@pytest.mark.parametrize("limbs", range(1, 17))
def test_rns_gemm_at_every_width(limbs, spread, form):
    """Bitwise: the exact dot product rounded once; zeros among the entries, odd sizes."""
    from sdpx_b200.solver import KernelContext
    m, n, k = 5, 3, 9
    rng = X.Lcg(100 * limbs + spread)
    A, B = X.random_values(limbs, rng, m * k, spread), X.random_values(limbs, rng, k * n, spread)
    A[3] = A[7] = B[0] = X.Mp(limbs)
    for q in range(k):
        B[2 * k + q] = X.Mp(limbs)  # a zero column
    raw, st = KernelContext().rns_gemm(limbs, "N", "N", m, n, k, X.pack_array(A), m, X.pack_array(B), k, form=form)
    assert st == 0
    got, want = X.unpack_array(limbs, raw), X.gemm(limbs, "N", "N", m, n, k, A, m, B, k)
    assert all(g == w for g, w in zip(got, want))
