"""Deferred norms: what the host refuses.  Row sums of squares that do not belong to the rows they come with are refused on the host: the kernel would scale by other rows' sums
or read past the end."""
import ctypes
import importlib

import pytest
import torch

from ooverlap_b200 import _lib
from ooverlap_b200.ops import RowSums, gemm_rope_kv_write, gemm_swiglu, rope_tables

M, K = 16, 384
SCALED = torch.zeros(M, K, dtype=torch.bfloat16)
BAD = {"a view of some rows": (SCALED[:8], torch.zeros(3, M)[:, :8]), "the sums of other rows": (SCALED, torch.zeros(3, M - 1)),
       "more rows": (SCALED[:8], torch.zeros(3, M)), "a part too few": (SCALED, torch.zeros(2, M)),
       "a part too many": (SCALED, torch.zeros(4, M)), "64 bits": (SCALED, torch.zeros(3, M, dtype=torch.float64)),
       "16 bits": (SCALED, torch.zeros(3, M, dtype=torch.bfloat16)), "transposed": (SCALED, torch.zeros(M, 3).t()),
       "one dimension": (SCALED, torch.zeros(3 * M)), "elsewhere": (SCALED, torch.zeros(3, M, device="meta"))}


@pytest.mark.parametrize("case", BAD)
def test_python_refuses_sums_of_another_form(case):
    scaled, ssq = BAD[case]
    rows = scaled.shape[0]
    with pytest.raises(ValueError, match="row sums"):
        gemm_swiglu(RowSums(scaled, ssq, 1e-5), torch.zeros(64, K, dtype=torch.bfloat16))
    cos, sin = rope_tables(32, 128, 10000.0, "cpu")
    cache = torch.zeros(rows, 1, 32, 128, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="row sums"):
        gemm_rope_kv_write(RowSums(scaled, ssq, 1e-5), torch.zeros(3 * 128, K, dtype=torch.bfloat16), rows, 1, 1, 1, cache, cache, cos, sin, 0)


@pytest.mark.parametrize("parts", [-1, 0, 1, 2, 4])
def test_native_refuses_another_number_of_parts(parts):
    g = _lib.GemmArgs()
    g.mode, g.dtype, g.M, g.N, g.K = _lib.GEMM_PLAIN, _lib.BF16, M, 64, K
    g.A, g.lda, g.B, g.ldb, g.C, g.ldc = 16, K, 16, K, 16, 64
    g.row_ssq, g.row_parts, g.row_eps = 16, parts, 1e-5
    assert _lib.lib().oob_gemm(None, ctypes.byref(g), None) == _lib.ERR_INVALID and "row sums" in _lib.last_error()


def _add_call():
    epi = _lib.AddEpilogue(residual=16, ld_residual=64, norm_weight=16, scaled_out=16, ssq=16)
    g = _lib.GemmArgs()
    g.mode, g.dtype, g.M, g.N, g.K = _lib.GEMM_PLAIN, _lib.BF16, M, 64, K
    g.A, g.lda, g.B, g.ldb, g.C, g.ldc = 16, K, 16, K, 16, 64
    g.epilogue, g.epilogue_args = _lib.EPILOGUE_ADD, ctypes.addressof(epi)
    return g, epi


def _sums_call():
    g, _ = _add_call()
    g.epilogue, g.epilogue_args = _lib.EPILOGUE_NONE, None
    g.row_ssq, g.row_parts, g.row_eps = 16, 3, 1e-5
    return g, None


@pytest.mark.parametrize("field,value", [("trace", 16), ("order", 16), ("gemv", 1), ("stream_k", 1), ("splitk_reduce", 1), ("splitk_reduce", -1),
                                         ("pair", 1), ("skinny", -1)])
@pytest.mark.parametrize("call", [_add_call, _sums_call])
def test_requests_that_the_kernel_would_drop_are_refused(call, field, value):
    g, keep = call()
    setattr(g, field, value)
    assert _lib.lib().oob_gemm(None, ctypes.byref(g), None) == _lib.ERR_UNSUPPORTED and "weight-streaming" in _lib.last_error()


@pytest.mark.parametrize("mode", [_lib.GEMM_AR, _lib.GEMM_RS_NORM, _lib.GEMM_AG])
@pytest.mark.parametrize("call", [_add_call, _sums_call])
def test_fused_modes_do_not_take_them(call, mode):
    g, keep = call()
    g.mode = mode
    assert _lib.lib().oob_gemm(None, ctypes.byref(g), None) == _lib.ERR_INVALID and "plain GEMM only" in _lib.last_error()


def test_rows_written_twice_are_refused():
    g, epi = _add_call()
    g.ldc = 56
    assert _lib.lib().oob_gemm(None, ctypes.byref(g), None) == _lib.ERR_INVALID and "ldc" in _lib.last_error()
    g.ldc, epi.ld_residual = 64, -64
    assert _lib.lib().oob_gemm(None, ctypes.byref(g), None) == _lib.ERR_INVALID and "ld_residual" in _lib.last_error()


def test_operands_of_the_norm_lie_beside_the_others(monkeypatch):
    G = importlib.import_module("ooverlap_b200.ops.gemm")
    monkeypatch.setattr(G, "_check_operands", lambda a, b: None)
    a, b, w = SCALED, torch.zeros(64, K, dtype=torch.bfloat16), torch.zeros(64, dtype=torch.bfloat16)
    res = torch.zeros(M, 64, dtype=torch.bfloat16)
    for bad in ((res.to("meta"), w), (res, w.to("meta"))):
        with pytest.raises(ValueError, match="device"):
            G.gemm_add_norm(a, b, *bad, 1e-5)
