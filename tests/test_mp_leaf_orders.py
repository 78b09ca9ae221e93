"""LDL' leaves at every limb count and at the orders where their rows spread over the cluster's four
CTAs and the lane groups in another way, bitwise against the oracle."""
import sys
from pathlib import Path

import pytest

from oracle import exact as X

sys.path.insert(0, str(Path(__file__).resolve().parent / "golden"))
import make_ldl_fixtures as F  # noqa: E402

pytestmark = pytest.mark.gpu


CASES = [(limbs, n) for limbs in range(1, 9) for n in (1, 2, 3, 4, 5, 6, 33)]
CASES += [(1, 127), (4, 128), (5, 128), (6, 126)]  # whole leaves, with rows in shared memory up to 5 limbs


@pytest.mark.parametrize("limbs,n", CASES)
def test_mp_leaf_bitwise(limbs, n):
    from sdpx_b200.solver import KernelContext
    A = F.matrix(limbs, n, 20, 7 * limbs + n)
    L, dinv, st = KernelContext().mp_ldl(limbs, n, X.pack_array(A), n, None)
    assert st == 0
    want = list(A)
    wd = X.ldl_rec(limbs, want, n, 0, n)
    got = X.unpack_array(limbs, L)
    low = lambda V: F.lower_bytes(X, limbs, n, [X.Mp(limbs) if v.is_zero() else v for v in V])  # noqa: E731
    assert low(got) == low(want)
    assert all(g == w for g, w in zip(X.unpack_array(limbs, dinv), wd))
