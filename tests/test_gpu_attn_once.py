"""Decode attention over a cache that L2 does not hold, alone and in clusters of each size: lengths on both sides of the one from which on keys and values
leave L2 first, on the host and on the device.  Tolerance as in the other attention tests: one rounding of the probabilities and one of the output to 16 bits,
four times over."""
import pytest
import torch

from ooverlap_b200.ops import attn_decode, attn_decode_reference

pytestmark = pytest.mark.gpu
LIMIT = 128 << 20


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("G", [1, 8, 16])
@pytest.mark.parametrize("B,KV,splits", [(1, 1, 1), (2, 1, 3), (9, 2, 0), (36, 1, 0), (70, 1, 0), (75, 2, 0), (300, 1, 0)])
def test_around_the_limit(B, KV, splits, G, dtype):
    torch.manual_seed(B)
    once = -(-LIMIT // (512 * B * KV))
    max_len = once + 40
    q = torch.randn(B, G * KV, 128, device="cuda").to(dtype)
    k, v = (torch.randn(B, KV, max_len, 128, device="cuda", dtype=dtype) for _ in range(2))
    for L in (once - 1, once, once + 33, 17):
        want = attn_decode_reference(q, k, v, L - 1)
        eps = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
        pos = torch.full((1,), L - 1, dtype=torch.long, device="cuda")
        got = attn_decode(q, k, v, pos, splits=splits)
        assert (got.float() - want).norm() <= 8 * eps * want.norm()
        assert torch.equal(got, attn_decode(q, k, v, pos, splits=splits))
        assert torch.equal(attn_decode(q, k, v, L - 1, splits=splits, len_bound=max_len), got)
