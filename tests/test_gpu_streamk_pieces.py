"""Stream-K where a tile is cut into many pieces: the warp that arrives last adds them in K order, within the
bound of any summation order, and the same bits every time."""
import numpy as np
import pytest

from conftest import gamma, rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


# 74, 74, 148, 8, 37, 3 and 2 pieces a tile, with 1 to 4 units a warp
@pytest.mark.parametrize("m,n,k", [(128, 128, 4096), (100, 67, 3000), (64, 9, 5000), (256, 256, 256), (64, 512, 1184),
                                   (300, 1000, 600), (640, 1000, 333)])
@pytest.mark.parametrize("beta", [False, True])
def test_pieces_add_up(mgx, m, n, k, beta):
    import torch
    rng = np.random.default_rng(m + n + k)
    A, B, C0 = rng_matrix(rng, (m, k)), rng_matrix(rng, (k, n)), rng_matrix(rng, (m, n))
    dA, dB = dev(A), dev(B)
    first = None
    for _ in range(3):
        dC = dev(C0)
        mgx.gemm_fp64(dA, dB, dC, ksplit=0, beta_one=beta)
        got = host(dC)
        first = got if first is None else first
        assert np.array_equal(bits(got), bits(first))
    want = A @ B + (C0 if beta else 0.0)
    bound = 2 * gamma(k + 300) * (np.abs(A) @ np.abs(B) + (np.abs(C0) if beta else 0.0))
    assert (np.abs(first - want) <= bound).all()
    assert mgx.device_status() == 0

