"""Work schedule of the two-SM GEMM (whole tiles round robin, of 256 columns or fewer, or a stream-K tail), enumerated on the host through the
test hook ``oob_test_pair_schedule`` (the kernel runs the same code on the device).

Checked for many shapes and pair counts: every (tile, K block) is computed exactly once; a pair parks at most one
partial accumulator; the number of parts the kernel expects for a tile is the number of pairs that
really contribute; the fused modes' tile orders are permutations of the tile grid."""
import ctypes

import pytest

from ooverlap_b200 import _lib

PLAIN, AR, RS, AG = range(4)


def schedule(mode, M, N, K, pairs, stream_k, world=1, rank=0):
    lib = _lib.lib()
    cap = 9 * (4 * ((M + 255) // 256) * ((N + 255) // 256) + 8 * pairs + 64)
    buf = (ctypes.c_int * cap)()
    n = lib.oob_test_pair_schedule(mode, M, N, K, pairs, stream_k, world, rank, buf, cap)
    assert n >= 0
    return [tuple(buf[i * 9:(i + 1) * 9]) for i in range(n)]


def columns(mode, M, N, K, pairs, stream_k):
    return _lib.lib().oob_test_pair_tile_columns(mode, M, N, K, pairs, stream_k)


SHAPES = [(512, 8192, 8192), (2048, 8192, 8192), (8192, 8192, 8192), (4096, 3584, 8192), (4096, 8192, 3584),
          (300, 520, 1024), (256, 256, 64), (1024, 1024, 4096), (2304, 768, 2048), (128 * 9, 256 * 5, 8192),
          (250, 8192, 3584), (1037, 4104, 2056), (2048, 2048, 2048), (129, 40, 72)]


@pytest.mark.parametrize("pairs", [74, 70, 66, 7, 3, 2, 1])
@pytest.mark.parametrize("stream_k", [0, 1, -1])
def test_every_k_block_of_every_tile_is_computed_once(pairs, stream_k):
    for M, N, K in SHAPES:
        items = schedule(PLAIN, M, N, K, pairs, stream_k)
        width = columns(PLAIN, M, N, K, pairs, stream_k)
        assert width % 32 == 0 and 128 <= width <= 256 and (width == 256 or stream_k <= 0)
        tm, tn, nkb = (M + 255) // 256, (N + width - 1) // width, (K + 63) // 64
        cover = {}
        slots = set()
        per_pair = {}
        for p, seq, mb, nb, kb0, kb1, slot, parts, first in items:
            assert 0 <= mb < tm and 0 <= nb < tn and 0 <= kb0 < kb1 <= nkb
            key = (mb, nb)
            cover.setdefault(key, []).append((kb0, kb1, p, slot, parts, first))
            per_pair.setdefault(p, []).append((seq, kb0, kb1, slot))
            if slot >= 0:
                assert slot not in slots, "a workspace slot is written by one item only"
                assert slot == p and kb0 > 0
                slots.add(slot)
                assert kb1 - kb0 < nkb
            elif slot == -2:  # the part that starts a tile: its pair owns the tile and parks nothing
                assert kb0 == 0 and kb1 < nkb
            else:
                assert kb0 == 0 and kb1 == nkb
        assert len(cover) == tm * tn, (M, N, K, pairs, stream_k)
        for key, parts_list in cover.items():
            parts_list.sort()
            pos = 0
            for kb0, kb1, p, slot, parts, first in parts_list:
                assert kb0 == pos
                pos = kb1
            assert pos == nkb
            if len(parts_list) > 1:
                # what the summing warp assumes: consecutive pairs starting at `first`, head part first
                contributors = [p for _, _, p, _, _, _ in parts_list]
                assert all(x[4] == len(parts_list) for x in parts_list)
                assert all(x[5] == contributors[0] for x in parts_list)
                assert contributors == list(range(contributors[0], contributors[0] + len(parts_list)))
        # a pair's partial items: at most one that does not start a tile and one that does, whole tiles come first
        for p, lst in per_pair.items():
            assert len([x for x in lst if x[3] >= 0]) <= 1 and len([x for x in lst if x[3] == -2]) <= 1
            # the parked part comes before the owned part in the pair's order (the owner of a tile never waits for a
            # pair that is itself waiting: parked parts are computed right after the whole tiles)
            kinds = [x[3] for x in lst if x[3] != -1 or True]
            if any(k >= 0 for k in kinds) and -2 in kinds:
                assert min(i for i, k in enumerate(kinds) if k >= 0) < kinds.index(-2)
            whole_before = [i for i, k in enumerate(kinds) if k == -1]
            parked = [i for i, k in enumerate(kinds) if k >= 0]
            if parked and whole_before:
                # whole tiles dealt round robin come first; at most one whole tile lies inside the tail range
                assert len([i for i in whole_before if i > parked[0]]) <= 1


def test_stream_k_balances_the_last_wave():
    """With a tail, the K blocks per pair differ by at most one tile's worth of rounding; without it, by a whole tile."""
    for M, N, K in [(512, 8192, 8192), (2048, 8192, 8192), (4096, 3584, 8192)]:
        nkb = K // 64
        for pairs in (74, 70):
            load = {}
            for p, seq, mb, nb, kb0, kb1, slot, parts, first in schedule(PLAIN, M, N, K, pairs, 1):
                load[p] = load.get(p, 0) + kb1 - kb0
            assert len(load) == pairs and max(load.values()) - min(load.values()) <= 1, (M, N, K, pairs)
            load = {}
            for p, seq, mb, nb, kb0, kb1, slot, parts, first in schedule(PLAIN, M, N, K, pairs, -1):
                load[p] = load.get(p, 0) + kb1 - kb0
            width = columns(PLAIN, M, N, K, pairs, -1)
            tiles = ((M + 255) // 256) * ((N + width - 1) // width)
            if tiles % pairs:
                assert max(load.values()) - min(load.get(p, 0) for p in range(pairs)) == nkb


def _tail(mode, M, N, K, pairs=74):
    return any(item[6] >= 0 for item in schedule(mode, M, N, K, pairs, 0))


def test_auto_rule_picks_a_tail_only_where_it_pays():
    # 8192^3 on 74 pairs wastes 1.2 % of the last wave: whole tiles only
    assert not _tail(PLAIN, 8192, 8192, 8192) and columns(PLAIN, 8192, 8192, 8192, 74, 0) == 256
    # less than a wave of tiles with operands beyond L2: a tail measured slower, narrower tiles fill the wave
    assert not _tail(PLAIN, 512, 8192, 8192) and columns(PLAIN, 512, 8192, 8192, 74, 0) == 224
    # a quarter of the last wave idle and no narrower width that fills it: tail
    assert _tail(PLAIN, 4096, 3584, 8192)
    # few tiles, shallow K: parking and adding accumulators costs more than the idle pairs
    assert not _tail(PLAIN, 512, 2048, 2048) and columns(PLAIN, 512, 2048, 2048, 74, 0) == 128
    # K of a tensor-parallel shard is never cut
    assert not _tail(PLAIN, 2048, 8192, 512)


def tile_columns(M, N, K, pairs=74):
    """Columns of a tile: both accumulators where a pair takes two neighbouring ones in one item."""
    items = schedule(PLAIN, M, N, K, pairs, 0)
    assert not any(item[6] >= 0 for item in items)
    joined = max(sum(1 for i in items if i[:2] == first[:2]) for first in items[:2])
    return joined * columns(PLAIN, M, N, K, pairs, 0)


def test_the_widths_that_were_measured_faster():
    # rows that start off a 128-byte line, but on a sector, cost a tenth more and not half: no wide tile to spare a round
    assert tile_columns(3983, 1648, 1808) == 192 and tile_columns(3769, 1424, 3040) == 160
    # off a sector they cost more than half: one round of wide tiles
    assert tile_columns(1037, 4104, 2056) == 320
    # many rounds: the power cap, not the last round, decides
    assert tile_columns(8192, 14336, 8192) == 256 and tile_columns(4096, 28672, 8192) == 256
    assert tile_columns(8192, 8192, 4096) == 256 and tile_columns(8192, 8192, 6144) == 256
    assert tile_columns(8192, 8192, 7168) == 512 and tile_columns(16384, 8192, 8192) == 512
    # ... unless the wide tiles leave more of a round idle
    assert tile_columns(4096, 14336, 8192) == 256


def test_all_gather_keeps_whole_columns_and_the_tail():
    # the chunk flags of an all-gather count 256-column tiles: a tail is the only way to fill the last wave
    assert _tail(AG, 4096, 3584, 8192) and _tail(AG, 2048, 8192, 8192)
    assert all(columns(mode, M, N, K, 70, 0) == 256 for mode in (AR, RS, AG) for M, N, K in SHAPES)


@pytest.mark.parametrize("world", [2, 4, 8])
def test_fused_orders_are_permutations(world):
    for mode in (AR, RS, AG):
        for M, N, K in [(256 * world * 2, 768, 256), (4096, 8192, 3584), (128 * world, 512, 128)]:
            for rank in (0, world - 1):
                items = schedule(mode, M, N, K, 5, -1, world, rank)
                tm, tn = (M + 255) // 256, (N + 255) // 256
                seen = {(mb, nb) for _, _, mb, nb, *_ in items}
                assert len(items) == tm * tn and len(seen) == tm * tn
    # reduce-scatter: consecutive row blocks of the order belong to consecutive owners (when rows split evenly)
    items = sorted(schedule(RS, 4096, 8192, 3584, 64, -1, 8, 0), key=lambda x: x[1])
    owners = [mb * 256 // 512 for _, _, mb, nb, *_ in items if nb == 0]
    assert owners[:8] == list(range(8))
    # all-gather: a rank starts with its own rows
    items = sorted(schedule(AG, 4096, 3584, 8192, 64, -1, 8, 3), key=lambda x: x[1])
    assert items[0][2] * 256 // 512 == 3
