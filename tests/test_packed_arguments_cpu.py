"""The packed form of an argument structure is the structure, byte for byte."""
import ctypes

from ooverlap_b200 import _lib


def test_packed_norm_arguments():
    values = [1, 16, 8192, 0.5, 2, 3 << 40, 4 << 40, 5 << 40, 6, 7 << 40, 8 << 40, -1, 9, 10 << 40, 11, 12, 13, 14]
    assert len(values) == len(_lib.NormArgs._fields_)
    a = _lib.NormArgs.from_buffer_copy(_lib.NORM_ARGS.pack(*values))
    assert [getattr(a, f) for f, _ in a._fields_] == values


def test_packed_model_arguments():
    for structure, pack, values in (
            (_lib.RopeArgs, _lib.ROPE_ARGS, [1, 2, 3, 4, 5, 6, 7 << 40, 8 << 40, 9 << 40, 10 << 40, 11 << 40, 12, 13, 14 << 40, 15 << 40, 16 << 40, 17]),
            (_lib.AttnDecodeArgs, _lib.ATTN_ARGS, [1, 2, 3, 4, 5 << 40, 6 << 40, 7 << 40, 8 << 40, 9, 10, 11 << 40, 12 << 40, 13, 0.25, 14, 15,
                                                   16 << 40, 1])):
        a = structure.from_buffer_copy(pack.pack(*values))
        assert [getattr(a, f) for f, _ in a._fields_] == values


def test_packed_plain_gemm_arguments():
    values = [0, 1, 16, 7168, 8192, 2 << 40, 8200, 3 << 40, 8208, 4 << 40, 7176]
    for tail, static in ((_lib.GEMM_TAIL, 0), (_lib.GEMM_TAIL_STATIC, 1)):
        a = _lib.GemmArgs.from_buffer_copy(_lib.GEMM_HEAD.pack(*values) + tail)
        names = [f for f, _ in a._fields_]
        assert [getattr(a, f) for f in names[:11]] == values
        assert names[10] == "ldc" and a.b_static == static
        assert all(not getattr(a, f) for f in names[11:] if f != "b_static")
        assert ctypes.sizeof(a) == _lib.GEMM_HEAD.size + len(tail)
