"""Products whose operands are packed first (odd pitches): the packed rows are the operand's own, at row
lengths around the widths that a row's threads take, and rows that share a block cost their bytes."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


def odd_pitch(x):
    import torch
    r, c = x.shape
    buf = torch.full((r, c + 1 - c % 2), float("nan"), dtype=torch.float64, device="cuda")
    buf[:, :c].copy_(x)
    return buf[:, :c]


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 16, 17, 33, 64, 129, 511, 513, 1025, 2047, 2048, 2049, 4100])
@pytest.mark.parametrize("m,n", [(1, 3), (257, 2), (131, 67), (5, 2050)])
def test_packed_equals_aligned(mgx, m, n, k):
    import torch
    rng = np.random.default_rng(m * n + k)
    A, B = dev(rng_matrix(rng, (m, k))), dev(rng_matrix(rng, (k, n)))
    C = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    mgx.gemm_fp64(odd_pitch(A), odd_pitch(B), C)
    want = torch.zeros((m, n + n % 2), dtype=torch.float64, device="cuda")

    def even(x):
        buf = torch.zeros((x.shape[0], x.shape[1] + x.shape[1] % 2), dtype=torch.float64, device="cuda")
        buf[:, :x.shape[1]].copy_(x)
        return buf[:, :x.shape[1]]

    mgx.gemm_fp64(even(A), even(B), want[:, :n])
    assert np.array_equal(bits(host(C)), bits(host(want[:, :n].contiguous())))
    assert mgx.device_status() == 0


def test_short_rows_cost_their_bytes(mgx):
    """2,000,000 rows of 3 at an odd pitch against the same rows at an even one, which are not packed: 1.1 times
    the time, 8.4 with a block for every row."""
    import torch

    def us(pitch):
        A = torch.rand((2000000, pitch), dtype=torch.float64, device="cuda")[:, :3]
        B, C = (torch.rand((r, pitch - 2), dtype=torch.float64, device="cuda")[:, :1] for r in (3, 2000000))
        best = 1e30
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(5):
                mgx.gemm_fp64(A, B, C)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1) / 5 * 1e3)
        return best

    odd, even = us(3), us(4)
    assert odd < 3 * even, (odd, even)
