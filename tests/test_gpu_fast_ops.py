"""The native Python entries of the ops (csrc/python/fast_ops.cpp) against the Python implementations beside them: the same bits for
what they take, the same errors for what they leave alone."""
import pytest
import torch

from ooverlap_b200 import _lib
from ooverlap_b200.ops import attn_decode, gemm, gemm_rope_kv_write, gemm_swiglu, rmsnorm, rope_tables

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(dtype)


def _both(monkeypatch, call, entry, taken=True):
    """``call()`` with the native entry and without; whether the entry took it is checked too."""
    seen = []
    fast = _lib.fast()

    class Watch:
        def __getattr__(self, name):
            def f(*args):
                r = getattr(fast, name)(*args)
                seen.append((name, r is not None))
                return r
            return f

    with monkeypatch.context() as m:
        m.setattr(_lib, "fast", lambda: Watch())
        a = call()
    with monkeypatch.context() as m:
        m.setattr(_lib, "fast", lambda: _lib._no_fast)
        b = call()
    torch.cuda.synchronize()
    assert (entry, taken) in seen
    return a, b


def _same(a, b):
    a, b = (x if isinstance(x, tuple) else (x,) for x in (a, b))
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride() and not x.requires_grad and torch.equal(x, y)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,strided", [(1, 1024, 1024, False), (2, 520, 512, True), (129, 1001, 264, False), (300, 2048, 512, True), (1, 8, 8, False)])
def test_gemm_and_swiglu(monkeypatch, M, N, K, strided, dtype):
    a, b = _rand(M, 2 * K, dtype=dtype), _rand(N, K, dtype=dtype, scale=K ** -0.5)
    a = a[:, K:] if strided else a[:, :K].contiguous()
    _same(*_both(monkeypatch, lambda: gemm(a, b), "gemm"))
    p = torch.nn.Parameter(b)
    _same(*_both(monkeypatch, lambda: gemm(a, p), "gemm"))
    if N % 16 == 0:
        _same(*_both(monkeypatch, lambda: gemm_swiglu(a, b), "gemm_swiglu"))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,hidden", [(1, 8), (17, 1024), (3, 8192)])
def test_rmsnorm(monkeypatch, rows, hidden, dtype):
    x, r, w = _rand(rows, hidden, dtype=dtype), _rand(rows, hidden, dtype=dtype), _rand(hidden, dtype=dtype)
    _same(*_both(monkeypatch, lambda: rmsnorm(x, w, 1e-5, r), "rmsnorm"))
    _same(*_both(monkeypatch, lambda: rmsnorm(x, w, 1e-5), "rmsnorm"))


@pytest.mark.parametrize("B,T,on_device", [(1, 1, True), (5, 1, False), (2, 300, False)])
def test_qkv_and_attention(monkeypatch, B, T, on_device):
    H, KV, K, L = 8, 2, 512, 1024
    x, w = _rand(B * T, K), _rand((H + 2 * KV) * 128, K, scale=K ** -0.5)
    cos, sin = rope_tables(L, 128, 10000.0, "cuda")
    pos = torch.full((1,), 37, dtype=torch.long, device="cuda") if on_device else 37
    caches = [torch.zeros(B + 1, KV, L, 128, device="cuda", dtype=torch.bfloat16) for _ in range(4)]
    turn = iter((0, 2))

    def call():
        i = next(turn)
        return gemm_rope_kv_write(x, w, B, T, H, KV, caches[i], caches[i + 1], cos, sin, pos, batch0=1), caches[i], caches[i + 1]

    _same(*_both(monkeypatch, call, "gemm_rope_kv_write"))
    q = _rand(B, H, 128)
    _same(*_both(monkeypatch, lambda: attn_decode(q, caches[0], caches[1], pos, batch0=1), "attn_decode"))
    _same(*_both(monkeypatch, lambda: attn_decode(q, caches[0], caches[1], pos, batch0=1, splits=3, len_bound=64), "attn_decode"))


def test_what_is_left_to_python(monkeypatch):
    a, b, w = _rand(4, 64), _rand(64, 64), _rand(64)

    def errors(call):
        got = []
        for fast in (_lib.fast(), _lib._no_fast):
            with monkeypatch.context() as m:
                m.setattr(_lib, "fast", lambda f=fast: f)
                with pytest.raises(Exception) as e:
                    call()
            got.append((type(e.value), str(e.value)))
        assert got[0] == got[1]

    errors(lambda: gemm(a, b.half()))
    errors(lambda: gemm(a, b[:, :32]))
    errors(lambda: gemm(a.t(), b))
    errors(lambda: gemm(a.cpu(), b))
    errors(lambda: gemm(a, b.cpu()))
    errors(lambda: gemm(a[:, 4:12], b[:, 4:12]))       # off 16 bytes: refused by the library
    errors(lambda: gemm_swiglu(a, b[:40]))       # 2F = 40
    errors(lambda: rmsnorm(a.t(), w))
    errors(lambda: attn_decode(_rand(1, 3, 128), _rand(1, 2, 16, 128), _rand(1, 2, 16, 128), 3))
    errors(lambda: attn_decode(_rand(1, 2, 128), _rand(1, 2, 16, 128), _rand(1, 2, 16, 128), 16))
    errors(lambda: torch.func.vmap(lambda x: gemm(x, b))(a.view(1, 4, 64)))
    x = torch.randn(4, 64, device="cuda")
    errors(lambda: rmsnorm(x, x[0].contiguous(), 1e-5))
    # Taken by Python: a whole number for eps, a subclass, a mode that sees every call.
    _same(*_both(monkeypatch, lambda: rmsnorm(a, w, 1), "rmsnorm", taken=False))

    class Sub(torch.Tensor):
        pass

    _both(monkeypatch, lambda: gemm(a.as_subclass(Sub), b), "gemm", taken=False)
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        _same(*_both(monkeypatch, lambda: gemm(a, b), "gemm", taken=False))


def test_under_inference_mode_and_capture(monkeypatch):
    a, b = _rand(4, 512), _rand(512, 512, scale=0.05)
    want = gemm(a, b)
    with torch.inference_mode():
        got = gemm(a, b)
    assert got.is_inference() and torch.equal(got, want)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        other = gemm(a, b)
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = gemm(a, b)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(other, want)


def test_options_given_in_another_type(monkeypatch):
    """``None`` for a number of CTAs is refused as by the library's argument types, and a promise that is not a bool is still one."""
    a, b, w = _rand(4, 64), _rand(64, 64), _rand(64)
    for call in (lambda: rmsnorm(a, w, max_ctas=None), lambda: gemm_swiglu(a, b, max_ctas=None)):
        with pytest.raises(Exception):
            call()
    q, kc = _rand(1, 2, 128), _rand(1, 2, 16, 128)
    _same(*_both(monkeypatch, lambda: attn_decode(q, kc, kc, 3, cache_ready=1), "attn_decode", taken=False))
