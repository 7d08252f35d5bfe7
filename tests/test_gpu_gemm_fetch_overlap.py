"""The weight-streaming GEMM fetches its first weights into L2 ahead of the wait for the kernel before.  Kernels of this library let the next one start early, so
behind one of them that writes the weights the fetch runs beside the writes: what is multiplied is what they leave all the same."""
import pytest
import torch

from ooverlap_b200.ops import gemm, gemm_swiglu, rmsnorm, silu_mul

pytestmark = pytest.mark.gpu


def _producers(N, K, turn):
    """Ways to write one of several [N, K] weights into ``b`` by a kernel of this library: a GEMM of several rounds of tiles, one of few rows of its
    weight, a norm and an activation."""
    g = torch.Generator(device="cuda").manual_seed(turn)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, y = r(N, 128).bfloat16(), (r(K, 128) * (128 * K) ** -0.5).bfloat16()
    rows, w = r(N, K).bfloat16(), torch.full((K,), K ** -0.5, device="cuda").bfloat16()
    gu = (r(N, 2 * K) * K ** -0.25).bfloat16()
    return {"gemm": lambda b: gemm(x, y, out=b), "norm": lambda b: rmsnorm(rows, w, 1e-5, out=b), "silu": lambda b: silu_mul(gu, out=b)}


# One stage and two, short and long K, two token blocks; SwiGLU of a weight that leaves L2 first, the only one with a fetch.
@pytest.mark.parametrize("M,N,K", [(1, 2048, 2048), (16, 8192, 512), (16, 4096, 4096), (64, 4096, 4096), (100, 2048, 3072), (16, 16384, 4096)])
@pytest.mark.parametrize("kind", ["gemm", "norm", "silu"])
def test_weights_written_by_a_kernel_that_lets_the_next_start(M, N, K, kind):
    torch.manual_seed(M)
    a = torch.randn(M, K, device="cuda").bfloat16()
    writes = [_producers(N, K, t)[kind] for t in range(3)]
    ops = [lambda b: gemm(a, b, skinny=1), lambda b: gemm_swiglu(a, b)]
    b, want = torch.zeros(N, K, device="cuda", dtype=torch.bfloat16), []
    for write in writes:
        write(b)
        torch.cuda.synchronize()
        want.append([op(b) for op in ops])
        torch.cuda.synchronize()
    assert not torch.equal(want[0][0], want[1][0])

    def chain():
        out = []
        for write in writes:
            out.append([])
            for i, op in enumerate(ops):
                writes[(writes.index(write) + 1 + i) % 3](b)  # other contents first, which the fetch may have asked for
                write(b)
                out[-1].append(op(b))
        return out

    got = chain() + chain()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        replayed = chain()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for x, y in zip(got + replayed, want * 3):
        for u, v in zip(x, y):
            assert torch.equal(u, v)
