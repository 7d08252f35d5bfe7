"""What attn_decode tells its kernel about the cache: that older keys may be loaded early is the caller's promise of its own, and not
part of the one about weights."""
import importlib

import pytest
import torch

from ooverlap_b200 import _lib
from ooverlap_b200.ops import static_weights

D = importlib.import_module("ooverlap_b200.ops.decode")


class _Native:
    def oob_attn_decode_auto_splits(self, *_):
        return 1

    def oob_attn_decode(self, args, stream):
        self.ahead = args._obj.ahead
        return 0


@pytest.mark.parametrize("kw,ahead", [({}, 0), (dict(cache_ready=False), 0), (dict(cache_ready=True), 1)])
def test_the_promise_is_the_callers(monkeypatch, kw, ahead):
    native = _Native()
    monkeypatch.setattr(_lib, "lib", lambda: native)
    monkeypatch.setattr(D, "_stream", lambda: None)
    q, cache = torch.zeros(2, 8, 128, dtype=torch.bfloat16), torch.zeros(2, 1, 32, 128, dtype=torch.bfloat16)
    for scope in (False, True):
        if scope:
            with static_weights():
                D.attn_decode(q, cache, cache, 3, **kw)
        else:
            D.attn_decode(q, cache, cache, 3, **kw)
        assert native.ahead == ahead
