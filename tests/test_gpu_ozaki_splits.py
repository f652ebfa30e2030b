"""The slice form's exponent and digit passes at the sizes where their blocks change (row lengths
around 512 and 2048, columns around groups of 64 and 256), every slice count, odd pitches, a workspace
full of arbitrary bytes, and panels of the host-buffer path that share a column group: bit-identical
to the oracle."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


def junk_workspace(mgx, nbytes, seed):
    import torch
    ws = mgx.OzakiWorkspace()
    g = torch.Generator(device="cuda").manual_seed(seed)
    buf = ws.get(nbytes)
    buf.copy_(torch.randint(0, 256, buf.shape, generator=g, device="cuda", dtype=torch.uint8))
    return ws


@pytest.mark.parametrize("m,n,k,s", [(1, 1, 1, 2), (3, 65, 512, 3), (9, 63, 513, 12), (2, 257, 2049, 8), (64, 255, 31, 9),
                                     (130, 64, 33, 5), (1, 300, 100, 10), (65, 1, 2048, 11)])
def test_every_block_shape(mgx, oracle, m, n, k, s):
    import torch
    rng = np.random.default_rng(m + n + k + s)
    A, B = rng_matrix(rng, (m, k + 1), "wide")[:, :k], rng_matrix(rng, (k, n + 1), "wide")[:, :n]
    dA, dB = dev(np.pad(A, ((0, 0), (0, 1))))[:, :k], dev(np.pad(B, ((0, 0), (0, 1))))[:, :n]
    dC = torch.empty((m, n), dtype=torch.float64, device="cuda")
    mgx.gemm_ozaki(dA, dB, dC, splits=s, workspace=junk_workspace(mgx, mgx.ozaki_workspace_size(m, n, k, s), 3))
    ref = oracle.ozaki_gemm(np.ascontiguousarray(A), np.ascontiguousarray(B), s)
    assert np.array_equal(bits(host(dC)), bits(ref))


def test_host_panels_that_share_a_column_group(mgx, oracle):
    import torch
    rng = np.random.default_rng(9)
    m, n, k = 200, 900, 96
    A, B = rng_matrix(rng, (m, k), "wide"), rng_matrix(rng, (k, n), "wide")
    hC = torch.empty((m, n), dtype=torch.float64)
    mgx.gemm_host(torch.from_numpy(A), torch.from_numpy(B), hC, form=mgx.FORM_OZAKI, splits=8, panels=8)
    torch.cuda.synchronize()
    assert np.array_equal(bits(hC.numpy()), bits(oracle.ozaki_gemm(A, B, 8)))
