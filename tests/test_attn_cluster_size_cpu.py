"""How many CTAs share the keys of one (sequence, KV head) in decode attention: the host knows a bound of the length only."""
import pytest

from ooverlap_b200 import _lib


def size(items, bound):
    return _lib.lib().oob_test_attn_cluster_size(items, bound)


@pytest.mark.parametrize("bound", [64, 128, 512, 2048, 4096, 8192])
@pytest.mark.parametrize("items", [150, 256, 296, 300, 512, 600, 2048])
def test_a_batch_that_fills_the_gpu_gets_one_cta_each(items, bound):
    """More CTAs gain at most a few per cent on a full cache and cost several times the time on a short context."""
    assert size(items, bound) == 1


def test_few_long_sequences_share_their_keys():
    assert size(1, 32768) == 8 and size(2, 2048) == 8 and size(16, 8192) == 8
    assert size(37, 32768) == 4 and size(74, 8192) >= 2


@pytest.mark.parametrize("items", [1, 7, 16, 100])
def test_every_warp_of_a_cluster_has_two_tiles_at_least(items):
    for bound in (1, 16, 127, 128, 255, 256, 511, 512, 1023, 1024, 4096):
        s = size(items, bound)
        assert s in (1, 2, 4, 8) and (s == 1 or bound >= s * 2 * 4 * 16)


def test_bad_arguments():
    assert size(0, 64) == -1 and size(1, 0) == -1
