"""The local residual + RMSNorm kernels at the sizes where their work distribution changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,hidden", [(1, 8), (3, 1000), (296, 4104), (297, 8), (297, 2048), (600, 2056), (1000, 8192), (2500, 1024),
                                         (300, 16384), (5, 16384), (2000, 2048), (900, 1032), (8192, 1024), (8193, 520), (8193, 1024), (9000, 1032),
                                         (310, 2056)])
@pytest.mark.parametrize("residual,max_ctas", [(True, 0), (False, 0), (True, 3)])
def test_rmsnorm_rows_and_widths(rows, hidden, residual, max_ctas, dtype):
    from ooverlap_b200.ops import rmsnorm, rmsnorm_reference
    g = torch.Generator(device="cuda").manual_seed(rows + hidden)
    x = torch.randn(rows, hidden, device="cuda", generator=g).to(dtype)
    r = torch.randn(rows, hidden, device="cuda", generator=g).to(dtype) if residual else None
    w = (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).to(dtype)
    got = rmsnorm(x, w, 1e-5, r, max_ctas=max_ctas)
    torch.cuda.synchronize()
    y_ref, r_ref = rmsnorm_reference(x, w, 1e-5, r)
    y = got[0] if residual else got
    if residual:
        assert torch.equal(got[1], r_ref)  # one fp32 addition, one rounding
    # the scale may differ in its last fp32 bits, which can move a value by one unit of the 16-bit type
    eps = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    assert ((y.float() - y_ref.float()).abs() <= eps * y_ref.float().abs() + 1e-6).all()


def test_rmsnorm_in_place():
    from ooverlap_b200.ops import rmsnorm, rmsnorm_reference
    for rows in (7, 900):
        x, r = torch.randn(rows, 1024, device="cuda").bfloat16(), torch.randn(rows, 1024, device="cuda").bfloat16()
        w = torch.ones(1024, device="cuda").bfloat16()
        y_ref, r_ref = rmsnorm_reference(x, w, 1e-5, r)
        rmsnorm(x, w, 1e-5, r, out=x, residual_out=r)
        torch.cuda.synchronize()
        assert torch.equal(r, r_ref) and ((x.float() - y_ref.float()).abs() <= 2.0 ** -7 * y_ref.float().abs() + 1e-6).all()


@pytest.mark.parametrize("rows,hidden,residual,max_ctas", [(297, 2056, True, 0), (700, 4104, False, 0), (1000, 8192, True, 0),
                                                           (300, 16384, True, 0), (2500, 3072, True, 5)])
@pytest.mark.parametrize("in_place", [False, True])
def test_rows_that_arrive_too_late_are_still_normalised(rows, hidden, residual, max_ctas, in_place):
    """A wait of the streaming kernel that runs out (here: at once) must not lose a row."""
    from ooverlap_b200 import _lib
    from ooverlap_b200.ops import rmsnorm
    x = torch.randn(rows, hidden, device="cuda").bfloat16()
    r = torch.randn_like(x) if residual else None
    w = (1 + 0.1 * torch.randn(hidden, device="cuda")).bfloat16()
    want = rmsnorm(x, w, 1e-5, r)
    want = want if residual else (want,)
    y = x if in_place else torch.full_like(x, float("nan"))
    ro = (r if in_place else torch.full_like(x, float("nan"))) if residual else None
    a = _lib.NormArgs()
    a.dtype, a.rows, a.hidden, a.eps = _lib.BF16, rows, hidden, 1e-5
    a.x_reg, a.x_off, a.weight, a.y_local, a.res_out_reg = 0, x.data_ptr(), w.data_ptr(), y.data_ptr(), -1
    a.residual = r.data_ptr() if residual else None
    a.res_out_local = ro.data_ptr() if residual else None
    _lib.check(_lib.lib().oob_test_norm_late_rows(a, max_ctas, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(y, want[0]) and (not residual or torch.equal(ro, want[1]))
