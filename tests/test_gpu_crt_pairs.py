"""Residue products by pairs of CTAs against single CTAs: the same product as one call, whose items go to
pairs, and as calls of 256 rows, whose single tile row does not.  Scales belong to rows of A and columns of
B, so the bits agree.  Tile rows odd and even, K blocks that end inside a box, K slices, strided operands."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,q,ksplit", [(1536, 2048, 1, 15, 1), (1500, 2300, 97, 13, 1), (1281, 1990, 160, 16, 1),
                                            (1025, 1990, 33, 15, 1), (1024, 2000, 300, 15, 3), (1300, 3000, 1000, 8, 4),
                                            (1200, 1250, 2100, 12, 2)])
def test_pairs_match_single_rows(mgx, m, n, k, q, ksplit):
    import torch
    rng = np.random.default_rng(m + n + k)
    A, B = dev(rng_matrix(rng, (m, k + 3), "wide"))[:, :k], dev(rng_matrix(rng, (k, n + 5), "wide"))[:, :n]
    C = torch.full((m, n + 2), -1.0, dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki_crt(A, B, C[:, :n], moduli=q, ksplit=ksplit)
    for r in range(0, m, 256):
        D = torch.empty((min(256, m - r), n), dtype=torch.float64, device="cuda")
        mgx.gemm_ozaki_crt(A[r:r + 256], B, D, moduli=q, ksplit=ksplit)
        assert torch.equal(C[r:r + 256, :n], D), r
    assert bool((C[:, n:] == -1.0).all())
    assert mgx.device_status() == 0
