"""The weight-streaming GEMM (K split inside a cluster) at the edges of its tiles, and the SwiGLU epilogue of the two-SM
kernel, against fp32 PyTorch and against the tiled kernels on the forms of operands that both accept."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}  # one rounding of the result


def _operands(M, N, K, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + M * 7 + N * 3 + K)
    return (torch.randn(M, K, device="cuda", generator=g).to(dtype),
            (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).to(dtype))


def _check(got, a, b, dtype):
    """One rounding to the output type plus K fp32 roundings of the running sum (each at most 2^-23 of the sum of
    magnitudes, whatever the order)."""
    ref = a.double() @ b.double().t()
    bound = EPS[dtype] * ref.abs() + a.shape[1] * 2.0 ** -23 * (a.double().abs() @ b.double().abs().t()) + 2.0 ** -24
    assert ((got.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 8, 8), (15, 127, 64), (16, 128, 72), (17, 129, 1096), (31, 1001, 520), (64, 1280, 8192),
                                   (127, 2048, 136), (128, 7168, 256), (129, 200, 2056), (255, 4104, 640), (256, 1000, 4096)])
@pytest.mark.parametrize("splits,pair", [(0, 0), (1, -1), (2, -1), (4, -1), (8, -1), (1, 1), (2, 1), (4, 1)])
def test_cluster_gemm_edges(shape, splits, pair, dtype):
    from ooverlap_b200.ops import gemm
    M, N, K = shape
    a, b = _operands(M, N, K, dtype)
    c = gemm(a, b, skinny=1, splits=splits, pair=pair)
    again = gemm(a, b, skinny=1, splits=splits, pair=pair)
    torch.cuda.synchronize()
    _check(c, a, b, dtype)
    assert torch.equal(c, again)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape,splits,pair", [
    ((16, 300, 520), 3, -1), ((100, 264, 1032), 5, -1), ((64, 1280, 2056), 6, -1), ((130, 200, 4096), 7, -1), ((512, 1280, 8192), 3, 1),
    ((257, 392, 520), 0, 0), ((257, 264, 520), 3, 1), ((383, 520, 264), 0, -1), ((383, 392, 1032), 2, 1), ((384, 264, 136), 1, 1),
    ((385, 264, 520), 0, 0), ((385, 1000, 520), 7, -1), ((1000, 520, 1096), 3, 1), ((1000, 264, 520), 0, 0), ((4095, 136, 264), 0, 0),
    ((4096, 392, 520), 4, -1), ((4096, 264, 520), 4, 1)])
def test_cluster_gemm_token_blocks_and_odd_splits(shape, splits, pair, dtype):
    """Two instructions per tile (257 - 384 tokens), several token blocks with a ragged last one, splits that are no power of two."""
    from ooverlap_b200.ops import gemm
    M, N, K = shape
    a, b = _operands(M, N, K, dtype)
    c = gemm(a, b, skinny=1, splits=splits, pair=pair)
    again = gemm(a, b, skinny=1, splits=splits, pair=pair)
    torch.cuda.synchronize()
    _check(c, a, b, dtype)
    assert torch.equal(c, again)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(17, 1290, 1032), (64, 1280, 2056), (200, 1000, 520), (300, 1288, 264), (1000, 640, 520)])
@pytest.mark.parametrize("splits,max_ctas", [(1, 3), (2, 4), (2, 7), (3, 6), (4, 4), (8, 8)])
def test_cluster_takes_several_tiles_one_after_the_other(shape, splits, max_ctas, dtype):
    """A budget leaves fewer clusters than tiles: shared memory, TMEM and the ring's phases are used again after the parts were
    read through distributed shared memory."""
    from ooverlap_b200.ops import gemm
    M, N, K = shape
    a, b = _operands(M, N, K, dtype)
    c = gemm(a, b, skinny=1, splits=splits, max_ctas=max_ctas)
    torch.cuda.synchronize()
    _check(c, a, b, dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(3, 520, 1032), (40, 264, 520), (200, 1000, 72)])
def test_default_route_equals_tiled_route_on_strided_operands(shape, dtype):
    from ooverlap_b200.ops import gemm
    M, N, K = shape
    wide_a, wide_b = _operands(M + 2, N + 3, K + 16, dtype, seed=5)
    a, b = wide_a[1:M + 1, 8:K + 8], wide_b[2:N + 2, 8:K + 8]
    for pad, off in ((0, 0), (8, 8), (5, 8)):  # row strides that are and are not multiples of 8 elements
        out = torch.full((M, N + pad + off), 7.0, device="cuda", dtype=dtype)
        got = gemm(a, b, out=out[:, off:off + N])
        tiled = gemm(a, b, skinny=-1, gemv=-1)
        torch.cuda.synchronize()
        _check(got, a, b, dtype)
        _check(tiled, a, b, dtype)
        assert (out[:, :off] == 7.0).all() and (out[:, off + N:] == 7.0).all()


def test_kernels_follow_one_another_without_gaps_in_order():
    """A chain of dependent launches whose set-up overlaps the kernel before: every link must see the link before it."""
    from ooverlap_b200.ops import gemm, rmsnorm, silu_mul
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(24, 512, device="cuda", generator=g).bfloat16()
    w1 = (torch.randn(1024, 512, device="cuda", generator=g) / 512 ** 0.5).bfloat16()
    w2 = (torch.randn(512, 512, device="cuda", generator=g) / 512 ** 0.5).bfloat16()
    nw = torch.ones(512, device="cuda").bfloat16()

    def chain(h, sync):
        r = h
        for _ in range(20):
            h, r = rmsnorm(gemm(silu_mul(gemm(h, w1)), w2), nw, 1e-5, r)
            if sync:
                torch.cuda.synchronize()
        return h, r

    ref = chain(x, True)
    for _ in range(3):
        got = chain(x, False)
        torch.cuda.synchronize()
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,F,K", [(1, 8, 64), (70, 72, 200), (256, 14336, 512), (257, 9480, 264), (1030, 4744, 1032), (2048, 8192, 256),
                                   (4096, 3584, 2048)])
def test_swiglu_in_the_tile_epilogue(M, F, K, dtype):
    from ooverlap_b200.ops import gemm_swiglu
    a, b = _operands(M, 2 * F, K, dtype)
    got = gemm_swiglu(a, b)
    torch.cuda.synchronize()
    gu = a.double() @ b.double().t()
    ref = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    # fp32 sums, then one rounding; the derivative of silu(g) * u is at most 1.1 |u| + |g| and the quotient and __expf add
    # a few parts in 2^22
    sum_err = K * 2.0 ** -23 * (a.double().abs() @ b.double().abs().t())
    bound = (EPS[dtype] + 2.0 ** -18) * ref.abs() + 1.1 * gu[:, F:].abs() * sum_err[:, :F] + gu[:, :F].abs() * sum_err[:, F:] + 2.0 ** -24
    assert ((got.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,F", [(64, 4096), (200, 2048), (512, 8192), (2048, 4096)])
def test_swiglu_is_one_formula_whatever_kernel_applies_it(M, F, dtype):
    """Rows of A that pick one column of B make every sum exact, so that the fused kernels see the very values that the
    stand-alone activation reads back; then the same formula gives the same bits."""
    from ooverlap_b200.ops import gemm, gemm_swiglu, silu_mul
    K = max(M, 512)
    g = torch.Generator(device="cuda").manual_seed(M + F)
    a = torch.eye(M, K, device="cuda").to(dtype)
    b = (torch.randn(2 * F, K, device="cuda", generator=g) * 3).to(dtype)
    b[:F, :4] = torch.tensor([0.0, -80.0, -1000.0, 1000.0], device="cuda", dtype=dtype)
    got, want = gemm_swiglu(a, b), silu_mul(gemm(a, b))
    torch.cuda.synchronize()
    assert torch.equal(gemm(a, b), b.t()[:M].contiguous())
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 18960, 2536), (1, 18944, 2536), (1, 19008, 2520), (2, 1152, 1032), (2, 1168, 1032), (3, 1024, 1024),
                                   (8, 38016, 4096), (9, 38016, 4096), (9, 37888, 4096), (48, 38016, 136), (49, 38016, 136),
                                   (128, 37888, 136), (128, 40000, 136)])
def test_default_route_at_the_edges_of_the_rules_for_few_rows(M, N, K, dtype):
    """One row below and above 48 M weights and 148 tiles, two rows around 1.2 M weights, more than 296 tiles of weights."""
    from ooverlap_b200.ops import gemm, gemm_swiglu
    a, b = _operands(M, N, K, dtype)
    c = gemm(a, b)
    _check(c, a, b, dtype)
    F = N // 2
    s = gemm_swiglu(a, b)
    torch.cuda.synchronize()
    gu = a.double() @ b.double().t()
    ref = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    # the two-kernel route rounds gate and up to the 16-bit type first
    tol = 4 * EPS[dtype] * ((1.1 * gu[:, F:].abs() + 1) * (gu[:, :F].abs() + 1))
    assert ((s.double() - ref).abs() <= tol).all()
