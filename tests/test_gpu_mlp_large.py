"""The cost model's forward pass on either side of the batch size where it goes over to a thread per sample:
the same bits as in parts, and right against 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [131071, 131072, 131073, 300001])
def test_large_batches_equal_their_parts(mgx, batch):
    import torch
    from oracle import mlp_oracle as MO
    g = torch.Generator(device="cuda").manual_seed(batch)
    X = torch.randn((batch, 6), generator=g, device="cuda")
    P = torch.empty(mgx.mlp_param_count(), dtype=torch.float32, device="cuda")
    mgx.mlp_init(P, seed=batch)
    out = mgx.mlp_forward(X, P)
    parts = torch.cat([mgx.mlp_forward(X[i:i + 50000].contiguous(), P) for i in range(0, batch, 50000)])
    assert torch.equal(out.view(torch.int32), parts.view(torch.int32))
    # tolerance as for small batches: an FP32 sum of 64 terms of at most unit size
    tail = out[-3000:].double().cpu().numpy()
    want = MO.forward(P.cpu().numpy().astype(np.float64), X[-3000:].double().cpu().numpy())
    assert np.max(np.abs(tail - want)) < 1e-5
