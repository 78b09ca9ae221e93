"""The persistent INT8 GEMM when a CTA walks several tiles (more tiles than two per SM), for every tile
configuration: integers, whose products are exact, and exact MpFloat products against each other."""
import numpy as np
import pytest

from oracle import exact as X
from sdpx_b200 import _lib
from sdpx_b200.solver import KernelContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1100, 900, 140), (1281, 513, 129)])
def test_split_product_of_integers_in_every_configuration(m, n, k):
    """16 moduli x at least 33 tiles.  Sums of k products below 2^40: exact in FP64."""
    import torch
    lib = _lib.load()
    rng = np.random.default_rng(m)
    A = rng.integers(-(1 << 16), 1 << 16, size=(m, k)).astype(np.float64)
    B = rng.integers(-(1 << 16), 1 << 16, size=(k, n)).astype(np.float64)
    dA, dB = (torch.from_numpy(np.asfortranarray(x).ravel(order="F").copy()).cuda() for x in (A, B))
    try:
        for cfg in (0, 1, 2):
            assert lib.sdpx_b200_i8_config(cfg) == 0
            dC = torch.zeros(m * n, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            assert KernelContext().split_dgemm_device("N", "N", m, n, k, 1.0, dA.data_ptr(), m, dB.data_ptr(), k, 0.0,
                                                      dC.data_ptr(), m) == 0
            assert np.array_equal(dC.cpu().numpy().reshape((n, m)).T, A @ B), cfg
    finally:
        lib.sdpx_b200_i8_config(-1)


@pytest.mark.parametrize("upper", [False, True])
def test_exact_product_in_every_configuration(upper):
    """Two digits: about 20 primes x 25 or more tiles, and the FP64 form as the reference."""
    lib = _lib.load()
    limbs, m, k = 2, 520, 7
    rng = X.Lcg(3)
    A, B = (X.pack_array(X.random_values(limbs, rng, m * k, 30)) for _ in range(2))
    want, st = KernelContext().rns_gemm(limbs, "N", "N", m, m, k, A, m, B, k, upper_only=upper, form=1)
    assert st == 0
    try:
        for cfg in (0, 1, 2):
            assert lib.sdpx_b200_i8_config(cfg) == 0
            got, st = KernelContext().rns_gemm(limbs, "N", "N", m, m, k, A, m, B, k, upper_only=upper, form=0)
            assert st == 0
            assert got == want, cfg
    finally:
        lib.sdpx_b200_i8_config(-1)
