"""Decode attention with scores whose maximum keeps rising, by small and large steps, and falls, over many
tiles of one warp; scores far below the first, and equal ones.  Tolerance as for one rounding of the probabilities and one of the
output to 16 bits, four times over."""
import pytest
import torch

from ooverlap_b200.ops import attn_decode, attn_decode_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,KV", [(8, 1), (4, 2), (16, 1)])
@pytest.mark.parametrize("step", [0.0, 0.02, 0.3, 5.0, -0.3, -5.0])
@pytest.mark.parametrize("B,L", [(1, 120), (160, 700)])
def test_rising_and_falling_scores(B, L, H, KV, step, dtype):
    torch.manual_seed(3)
    q = torch.randn(B, H, 128, device="cuda").to(dtype)
    q[:, :, 0] = 4.0
    k = torch.randn(B, KV, L, 128, device="cuda") * 0.3
    # Scores rise by `step` (before the scale of 1 / sqrt(128), in units of the natural logarithm) every sixteen keys, up to 60 in all.
    k[..., 0] = ((torch.arange(L, device="cuda") // 16) * step).clamp(-60, 60) * 128 ** 0.5 / 4.0
    k, v = k.to(dtype), torch.randn(B, KV, L, 128, device="cuda").to(dtype)
    got, want = attn_decode(q, k, v, L - 1), attn_decode_reference(q, k, v, L - 1)
    eps = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert torch.isfinite(got).all()
    assert (got.float() - want).norm() <= 8 * eps * want.norm()
