"""The constant check's paths where they can go wrong: bases off the 16-byte grid, odd element
counts, wrong elements at both ends, non-finite elements, tolerances and expected values at their
limits.  Counts and maxima equal the oracle's exactly."""
import numpy as np
import pytest

from gpu_util import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 3, 255, 1023, 4097, 148 * 8 * 1024 * 2 + 5])
@pytest.mark.parametrize("offset", [0, 1])
def test_edges_match_the_oracle(mgx, oracle, count, offset):
    rng = np.random.default_rng(count + offset)
    C = 64.0 * (1.0 + 1e-16 * rng.integers(-9, 10, count + offset))
    C[offset] += 1e-6
    C[-1] -= 3e-6
    buf = dev(C)[offset:]
    for abs_tol, rel_tol in ((1e-9, 1e-12), (0.0, 0.0), (-1.0, 1e-14), (1e-9, 1e-3)):
        ok, v = mgx.validate_matrix_c(buf, 1, count, 64.0, abs_tol, rel_tol)
        n, ma, mr = oracle.validate_constant(C[offset:].reshape(1, count), 64.0, abs_tol, rel_tol)
        assert (v.elements, v.invalid, v.max_abs_error, v.max_rel_error) == (count, n, ma, mr) and ok == (n == 0)


@pytest.mark.parametrize("expected", [0.0, 5e-324, 1e-310, np.inf, np.nan, -128.0])
def test_limit_values_match_the_oracle(mgx, oracle, expected):
    C = np.array([[128.0, -128.0, np.inf, -np.inf, np.nan, 0.0, 1e308, 5e-324, 1.0]])
    with np.errstate(all="ignore"):
        n, ma, mr = oracle.validate_constant(C, expected, count_nonfinite=True)
    ok, v = mgx.validate_matrix_c(dev(C), 1, C.size, expected)
    assert v.invalid == n and v.max_abs_error == ma and v.max_rel_error == mr and ok == (n == 0)


def test_threads_and_streams_check_at_the_same_time(mgx):
    """Each host thread reads its own findings, whatever the others check meanwhile."""
    import threading
    import torch
    xs = [torch.full((300 + 40 * i, 700), 8.0, dtype=torch.float64, device="cuda") for i in range(6)]
    for i, x in enumerate(xs):
        x[i, :i + 1] = 9.0 + i
    torch.cuda.synchronize()
    bad = []

    def work(i):
        for _ in range(20):
            ok, v = mgx.validate_matrix_c(xs[i], xs[i].shape[0], 700, 8.0)
            if ok or v.invalid != i + 1 or v.max_abs_error != 1.0 + i or v.max_rel_error != (1.0 + i) / 8.0:
                bad.append((i, v.invalid, v.max_abs_error))

    for _ in range(2):      # the second round's threads start after the first round's have ended
        threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not bad
