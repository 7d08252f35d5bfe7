"""Sums over a cluster in launches back to back: turns that some threads have no unit in, columns past the weight's, one turn and several,
whole heads and tails of clusters.  A CTA may end as soon as its peers have read its part, so that a read still under way would fault."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _back_to_back(call, times=40):
    """The first result, synchronised, and those of launches that follow one another closely."""
    want = call()
    torch.cuda.synchronize()
    got = [call() for _ in range(times)]
    torch.cuda.synchronize()
    assert all(torch.equal(want, g) for g in got)
    return want


def _operands(M, N, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    return (torch.randn(M, K, device="cuda", generator=g).to(dtype),
            (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).to(dtype))


# splits 1 - 8, on CTA pairs 1 - 4; rows for one turn, a ragged last turn and a nearly empty one
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("M,N,K", [(3, 136, 2048), (25, 1000, 2048), (49, 520, 2056), (64, 1160, 4096), (127, 264, 2048), (250, 1320, 2048)])
def test_plain(M, N, K, splits, dtype):
    from ooverlap_b200.ops import gemm
    a, b = _operands(M, N, K, dtype)
    got = _back_to_back(lambda: gemm(a, b, skinny=1, splits=splits))
    exact = a.double() @ b.double().t()
    assert (got.double() - exact).norm() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * exact.norm()


@pytest.mark.parametrize("M,F,K", [(1, 520, 2048), (16, 1792, 1024), (33, 264, 4096), (42, 2304, 640), (64, 3584, 8192), (100, 1032, 2048),
                                   (128, 1280, 512), (128, 8192, 512), (16, 28672, 512), (250, 3376, 2904)])
def test_swiglu(M, F, K):
    from ooverlap_b200.ops import gemm_swiglu
    a, b = _operands(M, 2 * F, K, torch.bfloat16)
    got = _back_to_back(lambda: gemm_swiglu(a, b))
    s = a.double() @ b.double().t()
    exact = torch.nn.functional.silu(s[:, :F]) * s[:, F:]
    assert (got.double() - exact).norm() <= 2.0 ** -8 * exact.norm()


@pytest.mark.parametrize("b,heads,kv,ctx", [(1, 8, 1, 300), (2, 32, 8, 900), (5, 16, 1, 700), (3, 10, 2, 500)])
def test_attention(b, heads, kv, ctx):
    from ooverlap_b200.ops import attn_decode, attn_decode_reference
    g = torch.Generator(device="cuda").manual_seed(ctx)
    q = torch.randn(b, heads, 128, device="cuda", generator=g).bfloat16()
    kc, vc = (torch.randn(b, kv, 1024, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    got = _back_to_back(lambda: attn_decode(q, kc, vc, ctx - 1))
    want = attn_decode_reference(q, kc, vc, ctx - 1).double()
    # probabilities and result are rounded to 16 bits
    assert (got.double() - want).norm() <= 2 * 2.0 ** -8 * want.norm()
