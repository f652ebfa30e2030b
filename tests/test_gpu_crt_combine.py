"""The CRT recombination's store paths (32-byte aligned rows, 16-byte aligned rows, odd pitches),
ragged edges of its 8- and 64-column groups, beta = 1, and outputs whose exponents leave the normal
range (subnormal and overflowing results): bit-identical to the oracle, C outside the product
untouched."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,pad", [(33, 64, 40, 0), (33, 66, 40, 0), (40, 67, 40, 0), (300, 261, 70, 3),
                                       (257, 9, 33, 3), (31, 1, 20, 0), (64, 259, 64, 1), (129, 520, 32, 0)])
@pytest.mark.parametrize("beta", [False, True])
@pytest.mark.parametrize("q", [8, 15, 16])
def test_store_paths_match_the_oracle(mgx, oracle, m, n, k, pad, beta, q):
    rng = np.random.default_rng(m + n + k + q)
    A, B = rng_matrix(rng, (m, k), "wide"), rng_matrix(rng, (k, n), "wide")
    C0 = rng_matrix(rng, (m + 1, n + pad), "wide")
    dC = dev(C0)
    mgx.gemm_ozaki_crt(dev(A), dev(B), dC[:m, :n], moduli=q, beta_one=beta)
    got = host(dC)
    ref = oracle.crt_gemm(A, B, q)
    ref = C0[:m, :n] + ref if beta else ref
    assert np.array_equal(bits(got[:m, :n]), bits(ref))
    assert np.array_equal(bits(got[m:]), bits(C0[m:])) and np.array_equal(bits(got[:, n:]), bits(C0[:, n:]))


@pytest.mark.parametrize("ea,eb", [(-540, -530), (-500, -560), (-1000, 20), (520, 510), (500, -700)])
def test_extreme_exponents_match_the_oracle(mgx, oracle, ea, eb):
    rng = np.random.default_rng(10000 + ea * 7 + eb)
    m, n, k = 70, 75, 50
    A, B = np.ldexp(rng_matrix(rng, (m, k)), ea), np.ldexp(rng_matrix(rng, (k, n)), eb)
    import torch
    dC = torch.empty((m, n), dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki_crt(dev(A), dev(B), dC, moduli=15)
    with np.errstate(all="ignore"):
        ref = oracle.crt_gemm(A, B, 15)
    assert np.array_equal(bits(host(dC)), bits(ref))
