"""Decode attention with a NaN or an infinity among values whose probability underflows to zero: 0 x NaN is NaN, whichever way the keys are
dealt out over warps, CTAs, clusters and splits."""
import pytest
import torch

from ooverlap_b200.ops import attn_decode, attn_decode_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("H", [8, 16])
@pytest.mark.parametrize("L,splits,at", [(700, 1, 3), (700, 2, 3), (700, 2, 650), (5000, 7, 2100), (20000, 40, 30), (20000, 40, 19990)])
def test_values_of_probability_zero(L, splits, at, H, bad):
    torch.manual_seed(at)
    q = torch.randn(1, H, 128, device="cuda")
    q[..., 0] = 100.0
    k = torch.randn(1, 1, L, 128, device="cuda")
    k[..., 0] = 0.0
    k[:, :, max(0, at - 600):at + 600, 0] = -100.0  # scores 880 below the others, where the values stand: exp underflows
    k[:, :, 0 if at > L // 2 else L - 1, 0] = 0.0
    v = torch.randn(1, 1, L, 128, device="cuda")
    v[:, :, at, 7::8] = bad
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    got, want = attn_decode(q, k, v, L - 1, splits=splits), attn_decode_reference(q, k, v, L - 1)
    assert bool(torch.isnan(want.view(H, 128)[:, 7::8]).all()) and int(torch.isnan(want).sum()) == H * 16
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    ok = ~torch.isnan(want)
    assert (got.float()[ok] - want[ok]).norm() <= 8 * 2.0 ** -9 * want[ok].norm()
