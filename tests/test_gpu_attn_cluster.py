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
    ref = attn_decode_reference(q, kc, vc, L - 1).view(B, H, 128)
    # The result is rounded once.  So are the probabilities, by at most eps each and independently of one another: their
    # errors add like sqrt(sum (p v)^2), of which eight standard deviations (eps / sqrt(3)) are allowed.
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    p = torch.softmax(torch.einsum("bhd,bhld->bhl", q.float(), kc[:, :, :L].float().repeat_interleave(H // KV, 1)) / 128 ** 0.5, -1)
    spread = torch.einsum("bhl,bhld->bhd", p.square(), vc[:, :, :L].float().square().repeat_interleave(H // KV, 1)).sqrt()
    assert ((out.float().view(B, H, 128) - ref).abs() <= eps * ref.abs() + (8 * eps / 3 ** 0.5 + 1e-5) * spread + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,KV,L,bound,splits", [
    (1, 8, 1, 1, 0, 0), (1, 16, 1, 17, 0, 0), (2, 8, 2, 63, 0, 1), (1, 8, 1, 65, 4096, 0), (1, 8, 1, 2047, 0, 0), (3, 8, 1, 4097, 0, 0),
    (33, 8, 1, 515, 0, 0), (70, 8, 1, 300, 0, 0), (150, 8, 1, 129, 0, 0), (2, 24, 3, 1000, 0, 5), (1, 4, 1, 40, 0, 7), (1, 8, 8, 4112, 0, 3)])
def test_every_key_counts_once(B, H, KV, L, bound, splits, dtype):
    """Equal scores, and one key per dimension with a value of one: the result is 1 / L there and zero elsewhere, exactly."""
    from ooverlap_b200.ops import attn_decode
    max_len = 4112
    q = torch.zeros(B, H, 128, device="cuda", dtype=dtype)
    kc = torch.randn(B, KV, max_len, 128, device="cuda").to(dtype)
    kc[:, :, L:] = float("nan")
    vc = torch.zeros_like(kc)
    vc[:, :, L:] = float("nan")
    pos = torch.full((1,), L - 1, dtype=torch.long, device="cuda")
    one = torch.full((128,), 1.0 / L, device="cuda", dtype=torch.float32).to(dtype)
    for base in range(0, L, 128):
        n = min(128, L - base)
        i = torch.arange(n, device="cuda")
        vc[:, :, base + i, i] = 1
        out = attn_decode(q, kc, vc, pos, splits=splits, len_bound=bound).view(B, H, 128)
        assert (out[:, :, :n] == one[:n]).all() and (out[:, :, n:] == 0).all(), base
        vc[:, :, base + i, i] = 0


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
