"""Entries near the ends of MpFloat's exponent range: a dot that an entry is reduced by may lie outside the
range where every entry lies inside, and no intermediate may be cut off there."""
import random

import pytest

from oracle import exact as X
from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu

EMAX = (1 << 30) - 1


def _value(n, rng, exp):
    return X.Mp(n, False, (1 << (64 * n - 1)) | rng.getrandbits(64 * n - 1), exp)


def _power(n, e):
    return X.Mp(n, False, 1 << (64 * n - 1), e + 1)


@pytest.mark.parametrize("limbs", [1, 4, 5, 8])
def test_ldl_with_a_row_dot_below_the_range(limbs):
    """a_10 = 2^-(2^30 - 10) and a_20 = 2^-40: the dot of rows 2 and 1 lies below the range and far below
    the last bit of a_21 = 1/2, so every other entry is what it is with a_10 = 0."""
    n, one = limbs, _power(limbs, 0)
    tiny = _power(n, -EMAX + 9)
    outs = []
    for a10 in (tiny, X.Mp(n)):
        low = {(0, 0): one, (1, 0): a10, (2, 0): _power(n, -40), (1, 1): one, (2, 1): _power(n, -1), (2, 2): one}
        A = X.pack_array([low[max(i, j), min(i, j)] for j in range(3) for i in range(3)])
        L, dinv, st = KernelContext().mp_ldl(n, 3, A, 3, None)
        assert st == 0
        outs.append((X.unpack_array(n, L), X.unpack_array(n, dinv)))
    (L, dinv), (L0, dinv0) = outs
    assert L[1] == tiny and L0[1].is_zero()
    assert dinv == dinv0 and L[2] == L0[2] and L[5] == L0[5]


@pytest.mark.parametrize("limbs", [2, 4, 5])
def test_nt_scaling_of_a_block_at_the_end_of_the_range(limbs):
    """S 2^-k and Z 2^k, k a multiple of four: lambda stays and R, Rinv and G move by 2^-k/2, 2^k/2 and 2^-k,
    bit for bit, while the Cholesky's row dot of S 2^-k lies below the range."""
    n, k, rng = limbs, (1 << 30) - 1024, random.Random(limbs)
    s = [_value(n, rng, -EMAX + 3 + k + (39 if i == j else 0)) for j in range(3) for i in range(j + 1)]
    z = [_value(n, rng, 1 if i == j else -20) for j in range(3) for i in range(j + 1)]
    outs = []
    for p in (0, k):
        args = [X.pack_array([X.Mp(n, v.neg, v.mant, v.exp + q) for v in m]) for m, q in ((s, -p), (z, p))]
        lam, lis, R, Ri, G, bst, st = KernelContext().mp_nt_scale(n, [3], *args)
        assert st == 0 and list(bst) == [0]
        outs.append([X.unpack_array(n, v) for v in (lam, lis, R, Ri, G)])
    for a, b, shift in zip(*outs, (0, 0, -k // 2, k // 2, -k)):
        assert all(X.Mp(n, v.neg, v.mant, v.exp + (0 if v.is_zero() else shift)) == w for v, w in zip(a, b))
