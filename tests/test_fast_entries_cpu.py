"""The native Python entries are an addition: where they cannot be built or loaded the library and the Python implementations work without them."""
import pytest
import torch

from ooverlap_b200 import _build, _lib
from ooverlap_b200.ops import gemm


@pytest.fixture
def elsewhere(monkeypatch, tmp_path):
    _lib.lib()
    monkeypatch.setattr(_build, "FAST", tmp_path / "_fast_ops.so")
    monkeypatch.setattr(_build, "FAST_STAMP", tmp_path / "fast.stamp")
    monkeypatch.setattr(_build, "OBJ", tmp_path)
    monkeypatch.setattr(_lib, "_fast", None)
    (tmp_path / _build.LIB.name).symlink_to(_build.LIB)  # found beside the module
    return tmp_path


def test_no_compiler(monkeypatch, elsewhere):
    monkeypatch.setenv("PATH", str(elsewhere))
    assert _build.is_current() and not _build.fast_is_current()
    with pytest.warns(RuntimeWarning, match="cannot be built"):
        assert _lib.fast() is _lib._no_fast
    assert _lib.fast() is _lib._no_fast  # said once
    with pytest.raises(ValueError, match="CUDA"):
        gemm(torch.zeros(2, 64, dtype=torch.bfloat16), torch.zeros(8, 64, dtype=torch.bfloat16))


def test_a_module_that_does_not_load(elsewhere):
    _build.FAST.write_bytes(b"not a library")
    _build.FAST_STAMP.write_text(_build.fast_hash())
    with pytest.warns(RuntimeWarning, match="cannot be loaded"):
        assert _lib.fast() is _lib._no_fast


def test_it_is_built_again_alone(monkeypatch, elsewhere):
    """Another PyTorch needs another module, and no other library."""
    before = _build.source_hash()
    monkeypatch.setattr(_build.importlib.metadata, "version", lambda name: "0.0")
    assert _build.source_hash() == before and _build.is_current() and not _build.fast_is_current()
    assert _lib.fast() is not _lib._no_fast and _build.fast_is_current()
    assert hasattr(_lib.fast(), "attn_decode")
