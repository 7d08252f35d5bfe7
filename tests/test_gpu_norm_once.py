"""The streaming RMSNorm on both sides of the bytes from which on its rows leave L2 first: the same result.  Tolerance: one rounding to 16 bits, twice over."""
import pytest
import torch

from ooverlap_b200.ops import rmsnorm, rmsnorm_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hidden", [4096, 5000, 8192, 12288])
@pytest.mark.parametrize("residual", [False, True])
def test_around_the_limit(hidden, residual, dtype):
    torch.manual_seed(hidden)
    limit = -(-(160 << 20) // (2 * hidden * (4 if residual else 2)))  # rows
    x, w = torch.randn(limit, hidden, device="cuda").to(dtype), torch.randn(hidden, device="cuda").to(dtype)
    r = torch.randn(limit, hidden, device="cuda").to(dtype) if residual else None
    got = rmsnorm(x, w, 1e-5, r)
    fewer = rmsnorm(x[:-1], w, 1e-5, None if r is None else r[:-1])
    want, stream = rmsnorm_reference(x, w, 1e-5, r)
    got, fewer = (got, fewer) if residual else ((got,), (fewer,))
    for a, b in zip(got, fewer):
        assert torch.equal(a[:-1], b)
    eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert (got[0].float() - want.float()).norm() <= 2 * eps * want.float().norm()
    assert r is None or torch.equal(got[1], stream)
