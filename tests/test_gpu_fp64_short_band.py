"""FP64 products whose last 64-row band has at most 32 rows, in every form that the kernel has: bit-identical
to the same rows of a product whose last band is whole (stream-K cuts K elsewhere: within the any-order
summation bound); rows beyond the product stay untouched."""
import numpy as np
import pytest

from conftest import gamma, rng_matrix
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 1281, 70), (17, 129, 64), (32, 3000, 33), (65, 700, 100), (80, 512, 96),
                                   (81, 2500, 65), (257, 257, 257), (336, 1201, 500), (352, 640, 1000), (1040, 1000, 90)])
@pytest.mark.parametrize("mode", ["whole", "split", "panels", "streamk"])
def test_short_last_band(mgx, m, n, k, mode):
    import torch
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    full = -(-m // 64) * 64
    A, B, C0 = rng_matrix(rng, (full, k), "wide"), rng_matrix(rng, (k, n), "wide"), rng_matrix(rng, (full, n))
    dA, dB, got, want = dev(A), dev(B), dev(C0), dev(C0)

    def run(rows, C):
        if mode == "panels":
            plan = mgx.SummaPlan(rows, n, k, 1, 1, 32)
            plan.run(dA[:rows], dB, C[:rows])
            plan.close()
        else:
            mgx.gemm_fp64(dA[:rows], dB, C[:rows], beta_one=True, ksplit={"whole": 1, "split": 3, "streamk": 0}[mode])

    run(m, got)
    run(full, want)
    assert torch.equal(got[m:].view(torch.int64), dev(C0)[m:].view(torch.int64))
    if mode == "streamk":
        bound = dev(2 * gamma(k + 1) * (np.abs(A) @ np.abs(B) + np.abs(C0)) + 1e-300)
        assert bool(((got - want).abs() <= bound)[:m].all())
    else:
        assert torch.equal(got[:m].view(torch.int64), want[:m].view(torch.int64))
    assert mgx.device_status() == 0
