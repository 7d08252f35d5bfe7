"""The weight-streaming GEMM asks for its first weights before the kernels in front of it are done: what it multiplies is what they
leave all the same."""
import pytest
import torch

from ooverlap_b200.ops import gemm, gemm_swiglu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 2048, 2048), (16, 1024, 1024), (16, 7168, 4096), (64, 4096, 3584), (100, 2048, 2056), (300, 2000, 1000), (5, 144, 72)])
def test_weights_written_by_the_kernel_before(M, N, K):
    torch.manual_seed(1)
    a = torch.randn(M, K, device="cuda").bfloat16()
    ws = [(torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16() for _ in range(4)]
    b, wide = torch.zeros_like(ws[0]), torch.empty(1 << 27, dtype=torch.uint8, device="cuda")
    want = [(gemm(a, w, skinny=1), gemm_swiglu(a, w)) for w in ws]
    got = []
    for w in ws:
        wide.fill_(1)  # what is in L2 is of no use
        b.copy_(w)
        got.append(gemm(a, b, skinny=1))
        b.copy_(w.flip(0))
        b.copy_(w)
        got[-1] = (got[-1], gemm_swiglu(a, b))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        replayed = []
        for w in ws:
            torch.mul(w, 1, out=b)
            replayed.append(gemm(a, b, skinny=1))
            torch.add(w, 0, out=b)
            replayed[-1] = (replayed[-1], gemm_swiglu(a, b))
    g.replay()
    torch.cuda.synchronize()
    for x, y, z in zip(want, got, replayed):
        for i in range(2):
            assert torch.equal(x[i], y[i]) and torch.equal(x[i], z[i])
