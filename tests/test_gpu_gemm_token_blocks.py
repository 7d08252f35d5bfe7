"""The weight-streaming GEMM where fewer than 128 rows are cut into blocks: the last block ragged, every epilogue that may be cut, and the
rows of a block that lie past the last one left alone.  Tolerance: one rounding to bf16 (2^-9) four times over."""
import pytest
import torch

from ooverlap_b200.ops import gemm, gemm_rope_kv_write, gemm_swiglu, rope_kv_write, rope_tables

pytestmark = pytest.mark.gpu
EPS = 4 * 2.0 ** -9


def _close(got, want):
    assert (got.float() - want).norm() <= EPS * want.norm()


@pytest.mark.parametrize("M", [33, 47, 64, 65, 81, 97, 113, 127, 128, 129, 161, 250, 333])
@pytest.mark.parametrize("N,K", [(4096, 4096), (2000, 1000), (1440, 3008), (1280, 8192), (520, 2056)])
def test_ragged_blocks(M, N, K):
    torch.manual_seed(M)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    want = a.float() @ b.float().t()
    buf = torch.full((M + 40, N), 7.0, device="cuda", dtype=torch.bfloat16)
    got = gemm(a, b, out=buf[:M])
    _close(got, want)
    assert torch.equal(got, gemm(a, b)) and bool((buf[M:] == 7.0).all())
    for s in (1, 2, 3):
        _close(gemm(a, b, skinny=1, splits=s), want)
    if N % 16 == 0:
        _close(gemm_swiglu(a, b), torch.nn.functional.silu(want[:, :N // 2]) * want[:, N // 2:])


@pytest.mark.parametrize("M,K", [(40, 4096), (70, 8192), (100, 2048), (128, 8192)])
def test_rotation_and_cache(M, K):
    H, KV, L = 8, 1, 256
    a, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn((H + 2 * KV) * 128, K, device="cuda") * K ** -0.5).bfloat16()
    cos, sin = rope_tables(L, 128, 10000.0, "cuda")
    caches = [torch.zeros(M, KV, L, 128, device="cuda", dtype=torch.bfloat16) for _ in range(4)]
    q = gemm_rope_kv_write(a, w, M, 1, H, KV, caches[0], caches[1], cos, sin, 9)
    want = rope_kv_write((a.float() @ w.float().t()).bfloat16(), M, 1, H, KV, caches[2], caches[3], cos, sin, 9)
    _close(q, want.float())
    for x, y in zip(caches[:2], caches[2:]):
        _close(x, y.float())
