"""Decode attention shared by the CTAs of a cluster, at the lengths and batch sizes where its work distribution changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,KV,L,bound,splits", [
    (1, 1, 1, 1, 0, 0), (1, 8, 1, 15, 0, 0), (1, 16, 1, 16, 0, 0), (2, 8, 1, 17, 0, 0), (1, 8, 1, 63, 0, 1), (1, 8, 1, 65, 0, 1),
    (1, 8, 1, 4096, 0, 0), (2, 24, 3, 1000, 0, 5), (40, 8, 1, 513, 0, 0), (100, 8, 1, 200, 0, 0), (150, 8, 1, 77, 0, 0),
    (300, 8, 1, 300, 0, 0), (3, 8, 2, 2000, 2000, 0), (1, 8, 1, 5, 4096, 0), (1, 4, 1, 40, 0, 7)])
def test_attention_lengths_and_clusters(B, H, KV, L, bound, splits, dtype):
    from ooverlap_b200.ops import attn_decode, attn_decode_reference
    max_len, g = 4112, torch.Generator(device="cuda").manual_seed(L * 11 + B)
    q = torch.randn(B, H, 128, device="cuda", generator=g).to(dtype)
    kc = torch.randn(B, KV, max_len, 128, device="cuda", generator=g).to(dtype)
    vc = torch.randn(B, KV, max_len, 128, device="cuda", generator=g).to(dtype)
    kc[:, :, L:] = float("nan")
    vc[:, :, L:] = float("nan")
    pos = torch.full((1,), L - 1, dtype=torch.long, device="cuda")
    out = attn_decode(q, kc, vc, pos, splits=splits, len_bound=bound)
    torch.cuda.synchronize()
    ref = attn_decode_reference(q, kc, vc, L - 1)
    # probabilities and the result are each rounded once to the 16-bit type; values are about 1, at most about 5
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert (out.float() - ref).abs().max().item() <= tol * max(1.0, ref.abs().max().item())


def test_split_calls_on_two_streams_and_in_a_graph():
    """Partial results belong to their call: neither a call on another stream nor a replayed graph touches them."""
    from ooverlap_b200.ops import attn_decode
    g = torch.Generator(device="cuda").manual_seed(9)

    def state(B):
        return (torch.randn(B, 32, 128, device="cuda", generator=g).bfloat16(),
                *(torch.randn(B, 8, 3000, 128, device="cuda", generator=g).bfloat16() for _ in range(2)))
    small, other, large = state(2), state(2), state(6)
    want = [attn_decode(*s, 2999, splits=5).clone() for s in (small, other, large)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    for _ in range(20):
        for i, s in enumerate((small, other)):
            with torch.cuda.stream(streams[i]):
                got[i].append(attn_decode(*s, 2999, splits=5))
    torch.cuda.synchronize()
    assert all(torch.equal(x, want[i]) for i in range(2) for x in got[i])
    out = torch.empty_like(want[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        attn_decode(*small, 2999, splits=5, out=out)
    assert torch.equal(attn_decode(*large, 2999, splits=5), want[2])
    guard = [torch.full((1 << 18,), 7.0, device="cuda") for _ in range(16)]  # may land where an outgrown workspace was
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert torch.equal(attn_decode(*large, 2999, splits=5), want[2])
    torch.cuda.synchronize()
    assert torch.equal(out, want[0]) and all((x == 7.0).all() for x in guard)
