"""The slice form's row exponents where rows share a block: short rows, row counts around the rule's line
(eight rows per SM) and not a multiple of eight, rows that are not finite, and a cost that does not grow
with the number of blocks."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [148 * 8 - 1, 148 * 8, 148 * 8 + 1, 1999])
@pytest.mark.parametrize("k", [1, 8, 33, 512, 513])
def test_tall_rows_match_the_oracle(mgx, oracle, m, k):
    import torch
    rng = np.random.default_rng(m + k)
    A, B = rng_matrix(rng, (m, k), "wide"), rng_matrix(rng, (k, 9), "wide")
    A[::3] *= 2.0 ** -300
    A[1] = 0.0
    C = torch.empty((m, 9), dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki(dev(A), dev(B), C, splits=6)
    assert np.array_equal(bits(host(C)), bits(oracle.ozaki_gemm(A, B, 6)))
    assert mgx.device_status() == 0


def test_nonfinite_rows_of_a_tall_operand(mgx):
    import torch
    m, k = 2001, 70
    rng = np.random.default_rng(5)
    A, B = rng_matrix(rng, (m, k)), rng_matrix(rng, (k, 16))
    A[7, 3], A[2000, 69] = np.inf, np.nan
    C = torch.empty((m, 16), dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki(dev(A), dev(B), C, splits=8)
    got = host(C)
    assert np.isnan(got[[7, 2000]]).all() and np.isfinite(np.delete(got, [7, 2000], axis=0)).all()
    assert mgx.device_status() != 0


def test_tall_rows_cost_their_bytes(mgx):
    """Digits of 600000 x 8 against 75000 x 64, the same bytes of A and, padded to 32 columns, four times the
    digits: 4.4 times the time, 7.1 with a block for every row."""
    import torch

    def us(m, k):
        A = torch.rand((m, k), dtype=torch.float64, device="cuda")
        B = torch.rand((k, 16), dtype=torch.float64, device="cuda")
        ws = torch.empty(mgx.ozaki_workspace_size(m, 16, k, 3), dtype=torch.uint8, device="cuda")
        best = 1e30
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(10):
                mgx.ozaki_split(A, B, 3, ws)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1) / 10 * 1e3)
        return best

    tall, short = us(600000, 8), us(75000, 64)
    assert tall < 5.5 * short, (tall, short)
