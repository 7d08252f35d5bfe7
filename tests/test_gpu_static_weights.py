"""GEMMs whose weights may be loaded ahead of the kernel before them: the results of calls without the promise, the same bits each
time, and without the promise an operand that the kernel before has just written."""
import contextlib

import pytest
import torch

from ooverlap_b200.ops import attn_decode, attn_decode_reference, gemm, gemm_rope_kv_write, gemm_swiglu, rmsnorm, rope_tables, static_weights
from ooverlap_b200.ops.gemm import _scope

pytestmark = pytest.mark.gpu


def _chain(x, w, b, t, heads, kv, kc, vc, cos, sin, pos):
    """Norm -> QKV + cache write -> norm -> gate/up -> down, every GEMM right behind another kernel of this library."""
    h = rmsnorm(x, w["n"], 1e-5)
    q = gemm_rope_kv_write(h, w["qkv"], b, t, heads, kv, kc, vc, cos, sin, pos)
    y, r = rmsnorm(gemm(q, w["o"]), w["n"], 1e-5, x)
    return q, r, gemm(gemm_swiglu(y, w["gu"]), w["d"])


# one stage per CTA; several; more K than the ring holds (wide and narrow stages); two token blocks on CTA pairs
@pytest.mark.parametrize("rows,hidden,ffn", [(1, 512, 256), (16, 1024, 520), (64, 4096, 1024), (100, 4096, 1024), (250, 2048, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_weights_loaded_ahead(rows, hidden, ffn, dtype):
    torch.manual_seed(0)
    heads, kv, hd, max_len = 4, 2, 128, 64

    def w(n, k):
        return (torch.randn(n, k, device="cuda") / k ** 0.5).to(dtype)

    ws = {"n": torch.ones(hidden, device="cuda", dtype=dtype), "qkv": w((heads + 2 * kv) * hd, hidden), "o": w(hidden, heads * hd),
          "gu": w(2 * ffn, hidden), "d": w(hidden, ffn)}
    x = torch.randn(rows, hidden, device="cuda").to(dtype)
    cos, sin = rope_tables(max_len, hd, 10000.0, "cuda")
    pos = torch.full((1,), 7, dtype=torch.long, device="cuda")
    out = []
    for ahead in (False, True, True, True):
        kc = torch.zeros(rows, kv, max_len, hd, device="cuda", dtype=dtype)
        vc = torch.zeros_like(kc)
        with static_weights() if ahead else contextlib.nullcontext():
            out.append((*_chain(x, ws, rows, 1, heads, kv, kc, vc, cos, sin, pos), kc, vc))
    for again in out[2:]:
        assert all(torch.equal(a, b) for a, b in zip(out[1], again))
    # K may be split differently: sums of fp32 in another order, which now and then round to the neighbouring 16-bit value; four
    # 16-bit steps lie between x and the last result.
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(out[0], out[1]):
        assert (a.double() - b.double()).norm() <= 4 * eps * a.double().norm()


@pytest.mark.parametrize("tokens,ctx", [(3, 3), (17, 40), (33, 600)])
def test_the_promise_about_weights_says_nothing_about_the_cache(tokens, ctx):
    """A projection that appends several tokens, and attention right behind it, in one block of static weights."""
    torch.manual_seed(ctx)
    b, heads, kv, hd, max_len, hidden = 3, 8, 1, 128, 1024, 512
    x = torch.randn(b * tokens, hidden, device="cuda").bfloat16()
    w = (torch.randn((heads + 2 * kv) * hd, hidden, device="cuda") / hidden ** 0.5).bfloat16()
    cos, sin = rope_tables(max_len, hd, 10000.0, "cuda")
    first = torch.full((1,), ctx - tokens, dtype=torch.long, device="cuda")
    last = torch.full((1,), ctx - 1, dtype=torch.long, device="cuda")
    cache = torch.randn(2, b, kv, max_len, hd, device="cuda").bfloat16()
    cache[:, :, :, ctx - tokens:] = float("nan")
    kc, vc = cache.clone()
    q = gemm_rope_kv_write(x, w, b, tokens, heads, kv, kc, vc, cos, sin, first)
    newest = q.view(b, tokens, heads, hd)[:, -1].contiguous()
    want = attn_decode_reference(newest, kc, vc, ctx - 1)
    for _ in range(5):
        kc, vc = cache.clone()
        torch.cuda.synchronize()
        with static_weights():
            gemm_rope_kv_write(x, w, b, tokens, heads, kv, kc, vc, cos, sin, first)
            got = attn_decode(newest, kc, vc, last)
        assert (got.double() - want.double()).norm() < 2 * 2.0 ** -8 * want.double().norm()


@pytest.mark.parametrize("ctx", [1, 2, 16, 17, 64, 65, 200, 1000])
@pytest.mark.parametrize("b,heads,kv", [(1, 8, 1), (3, 16, 1), (40, 8, 2)])
def test_cache_read_ahead_of_the_newest_key(ctx, b, heads, kv):
    """The newest key and value come from the kernel just before; all older ones may be loaded while it runs.  Same bits."""
    torch.manual_seed(ctx)
    hd, max_len, hidden = 128, 1024, 512
    x = torch.randn(b, hidden, device="cuda").bfloat16()
    w = (torch.randn((heads + 2 * kv) * hd, hidden, device="cuda") / hidden ** 0.5).bfloat16()
    cos, sin = rope_tables(max_len, hd, 10000.0, "cuda")
    pos = torch.full((1,), ctx - 1, dtype=torch.long, device="cuda")
    cache = torch.randn(2, b, kv, max_len, hd, device="cuda").bfloat16()
    cache[:, :, :, ctx - 1:] = float("nan")  # read only once the projection has written it
    out = []
    for ahead in (False, True, True):
        kc, vc = cache.clone()
        torch.cuda.synchronize()
        with static_weights() if ahead else contextlib.nullcontext():
            q = gemm_rope_kv_write(x, w, b, 1, heads, kv, kc, vc, cos, sin, pos)
        out.append((attn_decode(q.view(b, heads, hd), kc, vc, pos, cache_ready=ahead), q))
    assert torch.equal(out[1][0], out[2][0])
    want = attn_decode_reference(out[1][1].view(b, heads, hd), kc, vc, ctx - 1)
    assert (out[1][0].double() - want.double()).norm() < 2 * 2.0 ** -8 * want.double().norm()
    if torch.equal(out[0][1], out[1][1]):
        assert torch.equal(out[0][0], out[1][0])


def test_without_the_promise_b_may_be_the_result_of_the_call_before():
    torch.manual_seed(1)
    x = torch.randn(4096, 512, device="cuda").bfloat16()
    y = (torch.randn(2048, 512, device="cuda") / 512 ** 0.5).bfloat16()
    a = torch.randn(16, 2048, device="cuda").bfloat16()
    b = torch.empty(4096, 2048, device="cuda", dtype=torch.bfloat16)
    for _ in range(5):
        b.fill_(float("nan"))
        gemm(x, y, out=b)
        got = gemm(a, b)
        want = a.double() @ b.double().t()
        assert (got.double() - want).norm() < 4e-3 * want.norm()


def test_the_promise_ends_with_its_block():
    assert not _scope.static_b
    with pytest.raises(RuntimeError):
        with static_weights():
            assert _scope.static_b
            raise RuntimeError
    assert not _scope.static_b
