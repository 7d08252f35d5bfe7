"""The local residual + RMSNorm kernels at the sizes where their work distribution changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,hidden", [(1, 8), (3, 1000), (296, 4104), (297, 8), (297, 2048), (600, 2056), (1000, 8192), (2500, 1024),
                                         (300, 16384), (5, 16384)])
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
