"""Decoding of a tile-order record: as stamped, and with the tiles of a pair in that pair's sequence."""
import torch

from ooverlap_b200.ops import tile_order


def _record(stamps):
    """stamps: {unit: (nanoseconds, pair, index)}"""
    rec = torch.zeros(max(stamps) + 2, 2, dtype=torch.int64)
    for unit, (t, pair, index) in stamps.items():
        rec[unit, 0], rec[unit, 1] = t, pair << 32 | index
    return rec


# pair 0: CTA 0 stores its half of its second tile before CTA 1 has stored the first, and of the third before both
STAMPS = {0: (1000, 0, 0), 1: (5000, 0, 0), 4: (3000, 0, 1), 5: (7000, 0, 1), 8: (4500, 0, 2), 9: (9000, 0, 2),
          2: (2000, 1, 0), 3: (2500, 1, 0), 6: (6000, 1, 1), 7: (6500, 1, 1)}


def test_as_stamped():
    rec = tile_order(_record(STAMPS), in_sequence=False)
    assert [r["unit"] for r in rec] == [0, 2, 3, 4, 8, 1, 6, 7, 5, 9]
    assert [r["t_us"] for r in rec] == [0.0, 1.0, 1.5, 2.0, 3.5, 4.0, 5.0, 5.5, 6.0, 8.0]
    assert rec[4] == dict(unit=8, t_us=3.5, pair=0, index=2)


def test_in_sequence():
    rec = tile_order(_record(STAMPS))
    assert sorted(r["unit"] for r in rec) == sorted(STAMPS)
    for pair in (0, 1):
        index = [r["index"] for r in rec if r["pair"] == pair]
        assert index == sorted(index)
    when = {r["unit"]: r["t_us"] for r in rec}
    assert when == {0: 0.0, 1: 4.0, 4: 4.0, 5: 6.0, 8: 6.0, 9: 8.0, 2: 1.0, 3: 1.5, 6: 5.0, 7: 5.5}
    assert [r["t_us"] for r in rec] == sorted(when.values())


def test_nothing_recorded():
    assert tile_order(torch.zeros(4, 2, dtype=torch.int64)) == []
