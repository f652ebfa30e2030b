"""What stream-K's bookkeeping may cost, against the other FP64 schedules at the same shapes."""
import pytest

pytestmark = pytest.mark.gpu


def times(mgx, m, n, k, ksplits, reps=20):
    """Microseconds of a product for each K-slice count (0: stream-K), the best of six runs of `reps`."""
    import torch
    A, B = (torch.rand(s, dtype=torch.float64, device="cuda") for s in ((m, k + k % 2), (k, n + n % 2)))
    A, B = A[:, :k], B[:, :n]
    C, ws = torch.empty((m, n + n % 2), dtype=torch.float64, device="cuda")[:, :n], mgx.OzakiWorkspace()
    out = []
    for ksplit in ksplits:
        best = 1e30
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(reps):
                mgx.gemm_fp64(A, B, C, ksplit=ksplit, workspace=ws)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1) / reps * 1e3)
        out.append(best)
    return out


def test_uncut_tiles_cost_no_more_than_whole_k(mgx):
    """One K block, no tile cut: 0.93 times the whole-K kernel's time; 1.6 when every item asked for its piece."""
    sk, whole = times(mgx, 1102, 19749, 3, (0, 1))
    assert sk < 1.3 * whole, (sk, whole)


@pytest.mark.parametrize("m,n,k", [(128, 128, 4096), (64, 64, 65536), (300, 300, 300)])
def test_many_pieces_do_not_cost_more_than_slices(mgx, m, n, k):
    """Against eight K slices, whose sums are a kernel of their own.  With loads one by one and arrivals by
    compare-and-swap the shapes took 19, 5 and 3.6 times as long as with slices."""
    sk, slices = times(mgx, m, n, k, (0, 8))
    assert sk < 2.5 * slices + 15, (sk, slices)
