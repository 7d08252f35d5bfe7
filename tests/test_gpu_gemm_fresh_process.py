"""Routes of plain GEMMs that depend on what a process has done or set before: each runs in a child of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _child(code, **env):
    res = subprocess.run([sys.executable, "-c", "import torch\n" + code], env=dict(os.environ, PYTHONPATH=ROOT, **env),
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]


@pytest.mark.parametrize("M,N,K", [(2048, 2048, 2048), (2048, 8192, 1024), (1037, 4104, 2056)])
def test_a_gemm_that_needs_no_workspace_may_be_captured_before_there_is_one(M, N, K):
    """Whole tiles need no stream-K workspace, which could not be allocated during the capture.  The kernel itself has
    been loaded by a call that rules a tail out."""
    _child(f"M, N, K = {M}, {N}, {K}\n" """
from ooverlap_b200.ops import gemm
a = torch.randn(M, K, device="cuda").bfloat16()
b = (torch.randn(N, K, device="cuda") / K ** 0.5).bfloat16()
out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
gemm(a, b, out=out, stream_k=-1, pair=1, splits=1)
torch.cuda.synchronize()
out.zero_()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    gemm(a, b, out=out)
g.replay()
torch.cuda.synchronize()
ref = a.float() @ b.float().t()
assert (out.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
""")
