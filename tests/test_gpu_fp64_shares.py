"""The FP64 kernel's equal shares where they can go wrong: bands and units with remainders, shares
that cross bands, fewer units than SMs, shares just above the size where bands get virtual units,
and operands that are packed first (odd pitch, odd K offset, SUMMA panels that are no multiple of
32).  Bound: the any-order summation bound |C - C_ref| <= 2 gamma_K (|A||B|); C's columns and rows
beyond the product stay untouched."""
import numpy as np
import pytest

from conftest import gamma, rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,odd", [(1, 9, 33, True), (63, 7, 31, False), (65, 8, 32, False), (129, 1185, 64, False),
                                       (640, 952, 96, False), (640, 944, 96, False), (4500, 3, 40, True),
                                       (3, 4500, 40, False), (777, 1281, 130, True), (200, 2000, 65, False)])
@pytest.mark.parametrize("beta", [False, True])
def test_equal_shares_match_oracle(mgx, oracle, m, n, k, odd, beta):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A, B, C0 = rng_matrix(rng, (m, k + 1)), rng_matrix(rng, (k, n + 1)), rng_matrix(rng, (m + 1, n + 3))
    A, B = (A[:, 1:], B[:, 1:]) if odd else (np.ascontiguousarray(A[:, :k]), np.ascontiguousarray(B[:, :n]))
    if odd:  # views one column into a wider buffer: odd pitch or unaligned base
        dA, dB = dev(np.pad(A, ((0, 0), (1, 0))))[:, 1:], dev(np.pad(B, ((0, 0), (1, 0))))[:, 1:]
    else:
        dA, dB = dev(A), dev(B)
    dC = dev(C0)
    mgx.gemm_fp64(dA, dB, dC[:m, :n], beta_one=beta)
    got = host(dC)
    ref = oracle.ab_multiply(np.ascontiguousarray(A), np.ascontiguousarray(B)) + (C0[:m, :n] if beta else 0.0)
    ab = np.abs(A) @ np.abs(B) + np.abs(C0[:m, :n]) * beta
    assert np.all(np.abs(got[:m, :n] - ref) <= 2 * gamma(k + 1) * ab + 1e-300)
    assert np.array_equal(bits(got[m:]), bits(C0[m:])) and np.array_equal(bits(got[:, n:]), bits(C0[:, n:]))
    assert mgx.device_status() == 0


@pytest.mark.parametrize("M,N,K,bk,odd", [(130, 70, 200, 33, False), (389, 613, 531, 100, True), (65, 1200, 96, 96, False),
                                          (300, 300, 257, 1, False), (70, 90, 64, 32, True)])
def test_summa_panels_equal_accumulate_calls(mgx, M, N, K, bk, odd):
    """Every panel width: the running sum takes each panel with one rounding, as one accumulate
    call per panel does (bit-identical)."""
    import torch
    rng = np.random.default_rng(M + N + K + bk)
    off = 1 if odd else 0
    dA = dev(rng_matrix(rng, (M, K + off), "wide"))[:, off:]
    dB = dev(rng_matrix(rng, (K, N + off), "wide"))[:, off:]
    ref = torch.zeros((M, N), dtype=torch.float64, device="cuda")
    for k0 in range(0, K, bk):
        mgx.ab_multiply_accumulate_async(dA, dB[k0:], ref, M, N, K, k0, min(bk, K - k0), K + off, N + off, N)
    plan = mgx.SummaPlan(M, N, K, 2, 3, bk)
    C = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    plan.run(dA, dB, C)
    assert torch.equal(C.view(torch.int64), ref.view(torch.int64))
    plan.close()
    assert mgx.device_status() == 0
