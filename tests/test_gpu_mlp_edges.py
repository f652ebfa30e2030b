"""The cost model's kernels at batch sizes around a block's 16 samples and beyond one block per
sample group, against the oracle in 64 bits.  Tolerance: an FP32 dot product of 64 terms of at most
unit size is within 64 * 2^-24 * 64 / 2 of exact in the worst case and within 1e-5 in practice of
values of order one; gradients are compared relative to their largest entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 15, 16, 17, 33, 256, 9473, 20000])
def test_forward_and_gradients_match_64_bits(mgx, batch):
    import torch
    from oracle import mlp_oracle as MO
    rng = np.random.default_rng(batch)
    X = rng.normal(size=(batch, 6)).astype(np.float32)
    Y = rng.normal(size=(batch, 2)).astype(np.float32)
    P = torch.empty(mgx.mlp_param_count(), dtype=torch.float32, device="cuda")
    mgx.mlp_init(P, seed=batch)
    dX, dY, w = torch.from_numpy(X).cuda(), torch.from_numpy(Y).cuda(), torch.tensor([1.0, 0.5], device="cuda")
    out = mgx.mlp_forward(dX, P).cpu().numpy()
    assert np.max(np.abs(out - MO.forward(P.cpu().numpy().astype(np.float64), X.astype(np.float64)))) < 1e-5
    G = torch.full_like(P, float("nan"))       # overwritten, not accumulated into
    L = torch.full((1,), float("nan"), dtype=torch.float32, device="cuda")
    mgx.mlp_gradients(dX, dY, w, P, G, L)
    p = P.double().cpu().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = torch.split(p, [384, 64, 4096, 64, 128, 2])
    h = torch.tanh(torch.from_numpy(X).double() @ w1.view(64, 6).T + b1)
    o = torch.tanh(h @ w2.view(64, 64).T + b2) @ w3.view(2, 64).T + b3
    loss = ((o - torch.from_numpy(Y).double()).square() * torch.tensor([1.0, 0.5], dtype=torch.float64)).sum() / batch
    g, = torch.autograd.grad(loss, p)
    assert abs(L.item() - loss.item()) <= 1e-5 * max(1.0, loss.item())
    assert (G.double().cpu() - g).abs().max().item() <= 1e-5 * g.abs().max().item()
