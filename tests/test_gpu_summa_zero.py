"""A SUMMA plan starts from C = 0 and adds panels, so an element whose terms all underflow is +0.0,
whatever the panel width and however the plan launches its panels."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import bits, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 97])            # 16-byte and 8-byte stores of C
@pytest.mark.parametrize("panel", [7, 32, 33, 100, 128, 500])
def test_underflowed_panels_leave_no_negative_zero(mgx, n, panel):
    import torch
    m, k = 70, 128       # (a K that is padded to 32 ends in +0 terms)
    rng = np.random.default_rng(panel)
    A, B = dev(rng_matrix(rng, (m, k)) * 1e-170), dev(rng_matrix(rng, (k, n)) * 1e-170)
    C = torch.full((m, n), -1.0, dtype=torch.float64, device="cuda")
    mgx.SummaPlan(m, n, k, 2, 3, panel).run(A, B, C)
    assert not bits(host(C)).any()


def test_plain_product_keeps_the_sign_of_an_underflowed_sum(mgx):
    import torch
    A = torch.full((16, 32), -1e-170, dtype=torch.float64, device="cuda")
    B = torch.full((32, 24), 1e-170, dtype=torch.float64, device="cuda")
    C = torch.zeros((16, 24), dtype=torch.float64, device="cuda")
    mgx.gemm_fp64(A, B, C)
    assert (bits(host(C)) == np.uint64(1 << 63)).all()
