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


@pytest.mark.parametrize("M,F,K", [(2048, 2048, 512), (4224, 1024, 512), (300, 8192, 1024)])
def test_the_switch_that_forbids_the_two_sm_kernel_holds_for_swiglu(M, F, K):
    """OOB_GEMM_PAIR=0 (and no weight-streaming kernel): an unsplit gate/up projection is a one-SM GEMM and the
    stand-alone activation."""
    _child(f"M, F, K = {M}, {F}, {K}\n" """
from ooverlap_b200.ops import gemm, gemm_plan_splits, gemm_swiglu, silu_mul
a = torch.randn(M, K, device="cuda").bfloat16()
b = (torch.randn(2 * F, K, device="cuda") / K ** 0.5).bfloat16()
assert gemm_plan_splits(M, 2 * F, K) == 1
got, want = gemm_swiglu(a, b), silu_mul(gemm(a, b, pair=-1, skinny=-1))
torch.cuda.synchronize()
assert torch.equal(got, want)
""", OOB_GEMM_PAIR="0", OOB_GEMM_SKINNY="0")


def test_swiglu_runs_where_no_pair_of_sms_can(monkeypatch):
    """A device (or a budget) without the two-SM kernel: the native call refuses, the op runs two kernels instead."""
    import torch
    from ooverlap_b200 import _lib
    from ooverlap_b200.ops import gemm, gemm_swiglu, silu_mul
    real = _lib.lib()

    class NoPair:
        def __getattr__(self, name):
            return getattr(real, name)

        def oob_gemm(self, comm, args, stream):
            a = getattr(args, "_obj", args)
            return _lib.ERR_UNSUPPORTED if a.epilogue == _lib.EPILOGUE_SWIGLU_TILE else real.oob_gemm(comm, args, stream)

    a = torch.randn(2048, 512, device="cuda").bfloat16()
    b = (torch.randn(4096, 512, device="cuda") / 22).bfloat16()
    want = silu_mul(gemm(a, b))
    one = gemm_swiglu(a, b, max_ctas=1)  # one CTA is no pair
    monkeypatch.setattr(_lib, "lib", lambda: NoPair())
    got = gemm_swiglu(a, b)
    wide = torch.zeros(2048, 2048 + 16, device="cuda", dtype=torch.bfloat16)
    strided = gemm_swiglu(a, b, out=wide[:, 8:2056])
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(strided, want) and strided.data_ptr() == wide[:, 8:].data_ptr()
    assert not wide[:, :8].any() and not wide[:, 2056:].any()
    assert torch.equal(one, silu_mul(gemm(a, b, max_ctas=1)))
