"""A captured stream-K product replays: every replay finds its tiles' tickets without arrivals and writes C
anew from the inputs of that time, bit-identical to a call of its own."""
import numpy as np
import pytest

from conftest import rng_matrix
from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(64, 128, 4000), (200, 300, 2000), (777, 1282, 600), (1040, 1000, 90)])
def test_streamk_graph_replays(mgx, m, n, k):
    import torch
    rng = np.random.default_rng(m + n + k)
    A, B = dev(rng_matrix(rng, (m, k))), dev(rng_matrix(rng, (k, n)))
    C, want = (torch.zeros((m, n), dtype=torch.float64, device="cuda") for _ in range(2))
    ws = mgx.OzakiWorkspace()
    mgx.gemm_fp64(A, B, C, ksplit=0, workspace=ws)  # allocates the workspace before the capture
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        mgx.gemm_fp64(A, B, C, ksplit=0, workspace=ws)
    for _ in range(3):
        A.copy_(dev(rng_matrix(rng, (m, k))))
        graph.replay()
        mgx.gemm_fp64(A, B, want, ksplit=0)
        assert torch.equal(C.view(torch.int64), want.view(torch.int64))
    assert mgx.device_status() == 0
