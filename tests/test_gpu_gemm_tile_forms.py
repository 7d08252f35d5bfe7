"""Forms of the tiles of the two-SM kernel: one accumulator or both at once, four or eight epilogue warps, several rounds on few pairs, edges
inside either accumulator.  The host's cut decides the form; that it decides as meant here is asserted first."""
import pytest
import torch

from test_pair_schedule_cpu import PLAIN, columns, schedule

pytestmark = pytest.mark.gpu

# M, N, K, pairs, columns of a tile, rounds of tiles
FORMS = [
    (520, 640, 2048, 2, 320, 3),      # both accumulators, N a multiple of the tile
    (512, 1440, 4096, 5, 320, 2),     # N ends in the first accumulator: the second lies wholly past it
    (1280, 1592, 4096, 5, 320, 5),    # N ends in the second; an odd number of rounds
    (768, 1728, 1032, 5, 384, 3),
    (520, 1128, 1032, 3, 384, 3),     # rows past M, K off a block
    (1000, 2016, 1032, 5, 448, 4),
    (300, 1339, 1032, 2, 448, 3),     # rows of C at any 2-byte boundary: no vector stores
    (1280, 1784, 1032, 5, 448, 4),
    (1000, 2304, 1032, 5, 512, 4),
    (1280, 2040, 1032, 5, 512, 4),
    (300, 1536, 1032, 2, 512, 3),
    (700, 1330, 1032, 6, 224, 3),     # one accumulator, eight epilogue warps
    (2304, 1024, 2048, 2, 256, 18),   # ... four: many rounds of long tiles
    (2304, 152, 3392, 1, 160, 9),
    (2200, 1443, 4096, 5, 256, 11),
    (2200, 1446, 4096, 5, 256, 11),   # rows of C on 4 bytes
    (300, 1914, 1032, 5, 384, 2),
]


def _form(M, N, K, pairs):
    items = schedule(PLAIN, M, N, K, pairs, -1)
    tiles = {}
    for item in items:
        tiles.setdefault(item[:2], []).append(item[3])
    per_pair = [sum(1 for pair, _ in tiles if pair == p) for p in range(pairs)]
    return columns(PLAIN, M, N, K, pairs, -1) * max(map(len, tiles.values())), max(per_pair)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,pairs,width,rounds", FORMS)
def test_every_form_has_the_bits_of_the_one_sm_kernel(M, N, K, pairs, width, rounds, dtype):
    """Both kernels add the K blocks of a tile in the same order in fp32."""
    from ooverlap_b200.ops import gemm
    assert _form(M, N, K, pairs) == (width, rounds)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    b = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).to(dtype)
    how = dict(splits=1, pair=1, stream_k=-1, max_ctas=2 * pairs)
    want = gemm(a, b, splits=1, pair=-1)
    exact = a.double() @ b.double().t()
    # one rounding to the output type (half a unit of the last place); the fp32 sums are far closer
    assert (want.double() - exact).norm() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * exact.norm()
    for _ in range(2):
        assert torch.equal(gemm(a, b, **how), want)
    wide = torch.full((M, N + 24), 7.0, device="cuda", dtype=dtype)
    gemm(a, b, out=wide[:, :N], **how)
    assert torch.equal(wide[:, :N], want) and (wide[:, N:] == 7.0).all()


@pytest.mark.parametrize("N", [1026, 1027, 1030, 1279])
def test_a_tail_writes_rows_off_a_vector(N):
    """The pair that owns a tile of the tail adds the parts and writes; against 64 bits and bit by bit between calls."""
    from ooverlap_b200.ops import gemm
    M, K, pairs = 700, 4096, 7
    assert any(item[6] >= 0 for item in schedule(PLAIN, M, N, K, pairs, 1))
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    b = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    exact = a.double() @ b.double().t()
    outs = []
    for _ in range(2):
        wide = torch.full((M, N + 24), 7.0, device="cuda", dtype=torch.bfloat16)
        gemm(a, b, out=wide[:, :N], splits=1, pair=1, stream_k=1, max_ctas=2 * pairs)
        assert (wide[:, N:] == 7.0).all()
        outs.append(wide[:, :N])
    # one rounding to the output type
    assert torch.equal(*outs) and (outs[0].double() - exact).norm() <= 2.0 ** -8 * exact.norm()
