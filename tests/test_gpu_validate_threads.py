"""The constant check from short-lived threads beside other work: a thread's end does not wait for what
others have on the device, and the buffers that the threads leave serve the next ones."""
import threading
import time

import pytest

pytestmark = pytest.mark.gpu


def test_thread_end_does_not_wait_for_other_streams(mgx):
    import torch
    x = torch.full((300, 700), 8.0, dtype=torch.float64, device="cuda")
    assert mgx.validate_matrix_c(x, 300, 700, 8.0)[0]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(1_500_000_000)   # about 0.8 s of one block
        done.record()
    t0 = time.perf_counter()
    got = []
    for _ in range(3):
        t = threading.Thread(target=lambda: got.append(mgx.validate_matrix_c(x, 300, 700, 8.0)[0]))
        t.start()
        t.join()
    busy, dt = not done.query(), time.perf_counter() - t0
    torch.cuda.synchronize()
    assert got == [True] * 3
    assert busy, f"three checks took {dt:.3f} s: they waited for the other stream"


def test_buffers_are_reused_and_trimmed(mgx):
    import torch
    x = torch.full((64, 64), 2.0, dtype=torch.float64, device="cuda")
    for _ in range(3):
        threads = [threading.Thread(target=mgx.validate_matrix_c, args=(x, 64, 64, 2.0)) for _ in range(80)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        mgx.scratch_trim()
        ok, v = mgx.validate_matrix_c(x, 64, 64, 3.0)
        assert not ok and v.invalid == 64 * 64 and v.max_abs_error == 1.0
