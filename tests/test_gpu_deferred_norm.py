"""Projections around an RMSNorm that no kernel of its own computes: the stream, the sums of squares and what the next projection makes of
them, against the separate kernels and 64-bit sums, at the edges of tiles, splits and rows."""
import pytest
import torch

from ooverlap_b200.ops import RowSums, gemm, gemm_add_norm, gemm_rope_kv_write, gemm_swiglu, rmsnorm, rope_tables, static_weights

pytestmark = pytest.mark.gpu
EPS16 = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (2, 136, 512), (16, 8192, 1024), (17, 1000, 1032), (33, 4104, 3584), (64, 256, 8192), (65, 2048, 520),
                                   (128, 1024, 4096)])
def test_add_norm(M, N, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)

    def r(*s, f=1.0):
        return (torch.randn(*s, device="cuda", generator=g) * f).to(dtype)

    a, b, res, w = r(M, K), r(N, K, f=K ** -0.5), r(M, N + 8)[:, :N], (1 + r(N, f=0.1).float()).to(dtype)
    sums, h = gemm_add_norm(a, b, res, w, 1e-5)
    again, h2 = gemm_add_norm(a, b, res, w, 1e-5)
    assert torch.equal(h, h2) and torch.equal(sums.ssq, again.ssq) and torch.equal(sums.scaled, again.scaled)
    e = EPS16[dtype]
    # two roundings of values of the size of the product and of the sum
    assert _rel(h, a.double() @ b.double().t() + res.double()) < 2 * e
    assert torch.equal(sums.scaled, (h.float() * w.float()).to(dtype))
    want = torch.stack([h[:, i:i + 128].double().pow(2).sum(1) for i in range(0, N, 128)])
    assert ((sums.ssq.double() - want).abs() <= 128 * 2.0 ** -23 * want).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,hidden,F", [(1, 256, 64), (5, 1032, 520), (32, 8192, 3584), (100, 4096, 136), (128, 2048, 1024)])
def test_projections_behind_the_norm(M, hidden, F, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + hidden + F)

    def r(*s, f=1.0):
        return (torch.randn(*s, device="cuda", generator=g) * f).to(dtype)

    heads, kv, hd, max_len = 2, 1, 128, 32
    a, b, res, w = r(M, 512), r(hidden, 512, f=512 ** -0.5), r(M, hidden, f=3.0), (1 + r(hidden, f=0.1).float()).to(dtype)
    gu, qkv = r(2 * F, hidden, f=hidden ** -0.5), r((heads + 2 * kv) * hd, hidden, f=hidden ** -0.5)
    cos, sin = rope_tables(max_len, hd, 10000.0, "cuda")
    kc = torch.zeros(M, kv, max_len, hd, device="cuda", dtype=dtype)
    vc, kc2, vc2 = torch.zeros_like(kc), torch.zeros_like(kc), torch.zeros_like(kc)
    with static_weights():
        sums, h = gemm_add_norm(a, b, res, w, 1e-5)
        act = gemm_swiglu(sums, gu)
        q = gemm_rope_kv_write(sums, qkv, M, 1, heads, kv, kc, vc, cos, sin, 3)
    y = h.double() * torch.rsqrt(h.double().pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    s = y @ gu.double().t()
    e = EPS16[dtype]
    # one rounding of the rows of A and one of the result; the gate passes an error on with a factor of at most 1.1
    assert _rel(act, torch.nn.functional.silu(s[:, :F]) * s[:, F:]) < 4 * e
    # the same rounding in front of the product, and the rotation of both in fp32
    x = rmsnorm(h, w, 1e-5)
    q2 = gemm_rope_kv_write(x, qkv, M, 1, heads, kv, kc2, vc2, cos, sin, 3, fused=False)
    for got, want in ((q, q2), (kc, kc2), (vc, vc2)):
        assert _rel(got, want.double()) < 4 * e


def test_more_rows_are_refused():
    a, b, w = (torch.ones(s, device="cuda", dtype=torch.bfloat16) for s in ((129, 64), (64, 64), (64,)))
    with pytest.raises(ValueError):
        gemm_add_norm(a, b, torch.ones(129, 64, device="cuda", dtype=torch.bfloat16), w, 1e-5)
    sums = RowSums(a, torch.ones(1, 129, device="cuda"), 1e-5)
    with pytest.raises(RuntimeError):
        gemm_swiglu(sums, b)
