"""The CRT form's scale passes at the sizes where their blocks change: row lengths around the
register-held limits, column counts around a group of 256, rows and columns that are zero, subnormal,
or not finite, and a workspace full of arbitrary bytes.  Bit-identical to the oracle (rows and columns
with a NaN or an infinity give NaN)."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


def junk_workspace(mgx, m, n, k, q, seed):
    import torch
    ws = mgx.OzakiWorkspace()
    buf = ws.get(mgx.crt_workspace_size(m, n, k, q))
    g = torch.Generator(device="cuda").manual_seed(seed)
    buf.copy_(torch.randint(0, 256, buf.shape, generator=g, device="cuda", dtype=torch.uint8))
    return ws


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (5, 300, 1024), (5, 7, 1025), (3, 257, 2048), (3, 256, 2049), (2, 255, 4097),
                                   (2, 3, 8192), (2, 513, 8193), (700, 1, 63), (1, 2000, 65)])
def test_row_and_column_lengths(mgx, oracle, m, n, k):
    import torch
    rng = np.random.default_rng(m + n + k)
    A, B = rng_matrix(rng, (m, k), "wide"), rng_matrix(rng, (k, n), "wide")
    A[0, -1], B[-1, 0] = 2.0 ** 40, -2.0 ** 41      # the maximum in the last place
    dC = torch.empty((m, n), dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki_crt(dev(A), dev(B), dC, moduli=15, workspace=junk_workspace(mgx, m, n, k, 15, 7))
    assert np.array_equal(bits(host(dC)), bits(oracle.crt_gemm(A, B, 15)))
    assert mgx.device_status() == 0


def test_zero_and_subnormal_rows_and_columns(mgx, oracle):
    import torch
    rng = np.random.default_rng(5)
    m, n, k = 40, 300, 200
    A, B = rng_matrix(rng, (m, k)), rng_matrix(rng, (k, n))
    A[3] = 0.0
    A[4] *= 1e-310        # subnormal, high words set
    A[5] = 0.0
    A[5, 17] = 5e-324     # subnormal, low words only
    A[6] = rng.integers(0, 2 ** 31, k) * 5e-324
    B[:, 2] = 0.0
    B[:, 299] *= 1e-312
    B[:, 256] = 0.0
    B[100, 256] = -5e-324
    dC = torch.empty((m, n), dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki_crt(dev(A), dev(B), dC, moduli=15, workspace=junk_workspace(mgx, m, n, k, 15, 8))
    assert np.array_equal(bits(host(dC)), bits(oracle.crt_gemm(A, B, 15)))


def test_nonfinite_rows_and_columns_give_nan(mgx, oracle):
    import torch
    rng = np.random.default_rng(6)
    m, n, k = 30, 520, 90
    A, B = rng_matrix(rng, (m, k)), rng_matrix(rng, (k, n))
    A2, B2 = A.copy(), B.copy()
    A2[7, 3], A2[9, 89], B2[0, 511], B2[50, 300] = np.nan, np.inf, -np.inf, np.nan
    dC = torch.empty((m, n), dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki_crt(dev(A2), dev(B2), dC, moduli=15, workspace=junk_workspace(mgx, m, n, k, 15, 9))
    got, ref = host(dC), oracle.crt_gemm(A, B, 15)
    bad = np.zeros((m, n), bool)
    bad[[7, 9]] = True
    bad[:, [511, 300]] = True
    assert np.all(np.isnan(got[bad])) and np.array_equal(bits(got[~bad]), bits(ref[~bad]))
    assert mgx.device_status() == 4
