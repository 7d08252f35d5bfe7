"""Phase stamps of plain GEMMs (``oob_gemm_args_t.trace``): eight 64-bit words per CTA of the tiled kernels."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

START, GEMM_DONE, END = 0, 1, 4


def _launch(a, b, c, trace):
    from ooverlap_b200 import _lib
    from ooverlap_b200.ops.gemm import fill_gemm_args
    args = _lib.GemmArgs()
    args.mode = _lib.GEMM_PLAIN
    fill_gemm_args(args, a, b)
    args.C, args.ldc, args.trace = c.data_ptr(), c.stride(0), trace.data_ptr()
    _lib.check(_lib.lib().oob_gemm(None, ctypes.byref(args), torch.cuda.current_stream().cuda_stream))


def test_stamps_of_a_gemm_start_after_the_kernel_before_it():
    """The launch of a GEMM overlaps the kernel before it; its stamps must not."""
    a = torch.randn(4096, 4096, device="cuda").bfloat16()
    b = torch.randn(4352, 4096, device="cuda").bfloat16()
    c = torch.empty(4096, 4352, device="cuda", dtype=torch.bfloat16)
    traces = [torch.zeros(148, 8, dtype=torch.int64, device="cuda") for _ in range(4)]
    for t in traces:
        _launch(a, b, c, t)
    torch.cuda.synchronize()
    for before, after in zip(traces, traces[1:]):
        end, start = before[:, END], after[:, START]
        assert int((start > 0).sum()) > 1
        # The clock that is stamped advances in steps of up to 1 us.
        assert int(start[start > 0].min()) >= int(end.max()) - 1000
        assert (after[:, END] >= after[:, GEMM_DONE]).all() and (after[:, GEMM_DONE] >= after[:, START]).all()


@pytest.mark.parametrize("M,N,K", [(1, 7168, 8192), (16, 1024, 2048), (128, 1280, 8192), (200, 1280, 8192)])
def test_small_gemm_is_traced(M, N, K):
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = (torch.randn(N, K, device="cuda") / K ** 0.5).bfloat16()
    c = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    trace = torch.zeros(148 + 64, 8, dtype=torch.int64, device="cuda")
    _launch(a, b, c, trace)
    torch.cuda.synchronize()
    ref = a.float() @ b.float().t()
    assert (c.float() - ref).abs().max().item() <= 2e-2 * max(1.0, ref.abs().max().item())
    used = trace[:, START] > 0
    assert int(used.sum()) > 0 and (trace[used][:, GEMM_DONE] >= trace[used][:, START]).all()
    assert not trace[148:].any()  # one record per CTA, at most one CTA per SM
