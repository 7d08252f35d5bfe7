"""Which forward passes of the model runner fold their norms into the projections, and that the glue around the folded ones is the
model's: kernels replaced by PyTorch functions of the same contracts, compared with the runner's PyTorch arm."""
import pytest
import torch

from ooverlap_b200.models import llama as L
from ooverlap_b200.ops import RowSums
from test_llama_glue_cpu import _attn_decode, _gemm, _gemm_rope_kv_write, _gemm_swiglu, _rmsnorm


def _normalised(x):
    """What a projection makes of a RowSums: the rows divided by their rms."""
    if not isinstance(x, RowSums):
        return x
    return x.scaled * torch.rsqrt(x.ssq.sum(0) / x.scaled.shape[1] + x.eps).unsqueeze(1)


@pytest.fixture
def folded(monkeypatch):
    """Rows of the calls of gemm_add_norm."""
    rows = []

    def add_norm(a, b, residual, weight, eps):
        rows.append(a.shape[0])
        h = residual + a @ b.t()
        ssq = torch.stack([h[:, i:i + 128].pow(2).sum(1) for i in range(0, h.shape[1], 128)])
        return RowSums(h * weight, ssq, eps), h

    for name, fn in (("gemm", _gemm), ("rmsnorm", _rmsnorm), ("attn_decode", _attn_decode), ("gemm_add_norm", add_norm),
                     ("gemm_swiglu", lambda a, b, **kw: _gemm_swiglu(_normalised(a), b)),
                     ("gemm_rope_kv_write", lambda x, *a, **kw: _gemm_rope_kv_write(_normalised(x), *a, **kw))):
        monkeypatch.setattr(L, name, fn)
    return rows


@pytest.mark.parametrize("batch,tokens", [(1, 1), (4, 16), (64, 1), (65, 1), (5, 13), (128, 1)])
def test_folded_up_to_the_rows_where_that_was_measured_faster(folded, batch, tokens):
    cfg, kw = L.TINY128, dict(max_batch=batch, max_len=24, seed=5, device=torch.device("cpu"), dtype=torch.float32)
    ours, ref = L.LlamaTP(cfg, None, backend="ours", **kw), L.LlamaTP(cfg, None, backend="nccl", **kw)
    assert not ours.deferred_norm  # not on a CPU, and not in fp32
    ours.deferred_norm = ours.fused_epilogues = True
    g = torch.Generator().manual_seed(batch)
    x = torch.randint(0, cfg.vocab, (batch, tokens), generator=g)
    pos = torch.full((1,), tokens, dtype=torch.long) if tokens == 1 else 0
    mask = torch.full((1, 1, 1, 24), float("-inf"))
    mask[..., :2] = 0
    with torch.no_grad():
        for model in (ours, ref):
            model.k_cache[:, :, :, 0] = 0.5
            model.v_cache[:, :, :, 0] = 0.25
        got, want = (m.forward(x, pos, attn_mask=mask) if tokens == 1 else m.forward(x, 0) for m in (ours, ref))
    assert torch.allclose(got, want, atol=2e-4, rtol=1e-3)
    # two projections a layer, the last layer's second one in front of the norm that the caller gets
    assert folded == [batch * tokens] * (2 * cfg.layers - 1 if batch * tokens <= 64 else 0)
