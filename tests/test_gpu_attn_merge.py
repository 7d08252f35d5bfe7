"""Decode attention where its parts meet: every number of query heads a KV head may have, CTAs alone and in clusters of each size, warps and
CTAs without keys, results merged by a second kernel.  Tolerance: one rounding of the output to 16 bits (2^-9 of its size) and as much
for the 16-bit probabilities, four times over."""
import pytest
import torch

from ooverlap_b200.ops import attn_decode, attn_decode_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("G", [1, 2, 3, 5, 7, 8, 9, 12, 16])
@pytest.mark.parametrize("B,KV,L,splits", [(1, 1, 1, 0), (2, 1, 17, 0), (3, 2, 100, 0), (1, 1, 700, 0), (70, 2, 90, 0), (160, 1, 40, 0), (300, 1, 33, 0), (1, 2, 900, 3), (2, 1, 20, 4)])
def test_parts_meet(G, B, KV, L, splits, dtype):
    torch.manual_seed(G * 1000 + L)
    H = G * KV
    q = (torch.randn(B, H, 128, device="cuda") * 2).to(dtype)
    k = torch.full((B, KV, L + 40, 128), float("nan"), device="cuda", dtype=dtype)
    v = k.clone()
    k[:, :, :L] = torch.randn(B, KV, L, 128, device="cuda").to(dtype)
    v[:, :, :L] = torch.randn(B, KV, L, 128, device="cuda").to(dtype)
    got = attn_decode(q, k, v, L - 1, splits=splits)
    want = attn_decode_reference(q, k, v, L - 1)
    eps = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert torch.isfinite(got).all()
    assert (got.float() - want).norm() <= 8 * eps * want.norm()
    assert (got.float() - want).abs().max() <= 8 * eps * max(1.0, want.abs().max().item())
    assert torch.equal(got, attn_decode(q, k, v, L - 1, splits=splits))
