"""The partial results of split decode attention: calls that overlap must not share memory."""
import threading

import torch


class _Recorder:
    """Stands in for the native library; the two calls meet inside ``oob_attn_decode``, as their kernels may on two streams."""

    def __init__(self, calls):
        self.meet = threading.Barrier(calls, timeout=20)
        self.pointers = []

    def oob_attn_decode_auto_splits(self, B, KV, bound):
        return 4

    def oob_attn_decode_workspace_bytes(self, B, H, splits):
        return B * H * splits * 130 * 4

    def oob_attn_decode(self, args, stream):
        self.pointers.append(args._obj.workspace)
        self.meet.wait()
        return 0


def test_overlapping_split_calls_have_partial_results_of_their_own(monkeypatch):
    from ooverlap_b200 import _lib
    from ooverlap_b200.ops import decode
    rec = _Recorder(2)
    monkeypatch.setattr(_lib, "lib", lambda: rec)
    monkeypatch.setattr(decode, "_stream", lambda: 0)
    q = torch.zeros(2, 8, 128, dtype=torch.bfloat16)
    kc = torch.zeros(2, 1, 64, 128, dtype=torch.bfloat16)
    threads = [threading.Thread(target=decode.attn_decode, args=(q, kc, kc, 63)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    need = rec.oob_attn_decode_workspace_bytes(2, 8, 4)
    assert len(rec.pointers) == 2 and all(rec.pointers)
    assert abs(rec.pointers[0] - rec.pointers[1]) >= need


def test_a_workspace_off_four_bytes_is_refused_by_the_host():
    import ctypes

    from ooverlap_b200 import _lib
    a = _lib.AttnDecodeArgs(_lib.BF16, 1, 8, 1, 1 << 20, 1 << 20, 1 << 20, 64 * 128, 64, 0, 1 << 20, None, 64, 0.1, 2, 64, (1 << 20) + 2, 0)
    assert _lib.lib().oob_attn_decode(ctypes.byref(a), None) == _lib.ERR_INVALID
    assert "workspace" in _lib.last_error()
