"""The distance transform on device buffers as the first call of a process
inside a stream capture, in every capture mode and in the tile and sweep
forms: it is captured, and the graph's replays follow the code that its
buffer then holds."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys, torch
from coldcase_gb300 import lib as L
from coldcase_gb300.workloads import uniform_code
mode, q, n, M = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]), int(sys.argv[4])
lib = L.load()
codes = [torch.from_numpy(uniform_code(q, n, M, s)).cuda() for s in (1, 2)]
code = codes[0].clone()
dist = torch.zeros(q ** n, dtype=torch.uint8, device="cuda")
want = torch.zeros_like(dist)
torch.cuda.synchronize()
graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
    L.check(lib.cov_mindist_dev(q, n, code.data_ptr(), M, dist.data_ptr(), stream.cuda_stream))
for c in (codes[0], codes[1], codes[0]):
    code.copy_(c)
    graph.replay()
    torch.cuda.synchronize()
    L.check(lib.cov_mindist_dev(q, n, c.data_ptr(), M, want.data_ptr(), None))
    torch.cuda.synchronize()
    assert torch.equal(dist, want)
print("captured")
"""


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("q,n,M", [(6, 6, 41), (8, 6, 60000)])
def test_first_call_is_captured(covlib, mode, q, n, M):
    p = subprocess.run([sys.executable, "-c", PROGRAM, mode, str(q), str(n), str(M)], cwd=REPO, capture_output=True,
                       text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip() == "captured", p.stdout + p.stderr
