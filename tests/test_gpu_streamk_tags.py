"""Stream-K in a workspace that holds what other programs leave in memory: words that look like a small tag
with arrivals are no arrivals.  In a process of its own, whose first launches would have the smallest tags."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import sys, torch
sys.path.insert(0, sys.argv[1])
import mgxbench_b200 as mgx
A = torch.rand((200, 3000), dtype=torch.float64, device="cuda")
B = torch.rand((3000, 300), dtype=torch.float64, device="cuda")
C, want = (torch.full((200, 300), -1.0, dtype=torch.float64, device="cuda") for _ in range(2))
clean = mgx.OzakiWorkspace()
clean.get(mgx.lib().mgx_fp64_streamk_workspace_size(200, 300, 3000)).zero_()
for launch in range(1, 5):
    ws = mgx.OzakiWorkspace()
    words = ws.get(mgx.lib().mgx_fp64_streamk_workspace_size(200, 300, 3000)).view(torch.int64)
    # the tag that this launch has where they count 1, 2, ..., with one to seven arrivals
    words.copy_((2 * launch - 1) * 256 + 1 + torch.arange(words.numel(), device="cuda") % 7)
    mgx.gemm_fp64(A, B, C, ksplit=0, workspace=ws)
    mgx.gemm_fp64(A, B, want, ksplit=0, workspace=clean)
    assert torch.equal(C.view(torch.int64), want.view(torch.int64)), launch
assert torch.allclose(C, A @ B) and mgx.device_status() == 0
print("ok")
"""


def test_words_of_other_programs_are_no_arrivals():
    r = subprocess.run([sys.executable, "-c", CODE, str(ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
