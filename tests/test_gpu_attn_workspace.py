"""The workspace of split decode attention as a C caller may give it: on four bytes, which is what floats need and not more."""
import ctypes

import pytest
import torch

from ooverlap_b200 import _lib
from ooverlap_b200.ops import attn_decode

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,KV,L,splits", [(8, 1, 900, 3), (16, 1, 700, 2), (3, 1, 17, 4), (8, 2, 5000, 33)])
@pytest.mark.parametrize("offset", [4, 8, 12])
def test_workspace_on_four_bytes(H, KV, L, splits, offset):
    torch.manual_seed(L)
    B = 2
    q = torch.randn(B, H, 128, device="cuda").bfloat16()
    k, v = (torch.randn(B, KV, L, 128, device="cuda").bfloat16() for _ in range(2))
    want = attn_decode(q, k, v, L - 1, splits=splits)
    need = _lib.lib().oob_attn_decode_workspace_bytes(B, H, splits)
    ws = torch.full((need + 64,), 0xA5, device="cuda", dtype=torch.uint8)
    out = torch.empty(B, H * 128, device="cuda", dtype=torch.bfloat16)
    a = _lib.AttnDecodeArgs(_lib.BF16, B, H, KV, q.data_ptr(), k.data_ptr(), v.data_ptr(), k.stride(0), L, 0, out.data_ptr(), None, L,
                            128 ** -0.5, splits, L, ws.data_ptr() + offset, 0)
    _lib.check(_lib.lib().oob_attn_decode(ctypes.byref(a), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert bool((ws[:offset] == 0xA5).all()) and bool((ws[offset + need:] == 0xA5).all())
