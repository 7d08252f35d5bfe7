"""How many CTAs share the keys of one (sequence, KV head) in decode attention: the host knows a bound of the length only."""
import pytest

from ooverlap_b200 import _lib


def size(items, bound, slots=(296, 264, 256)):
    return _lib.lib().oob_test_attn_cluster_size(items, bound, *slots)


@pytest.mark.parametrize("bound", [64, 128, 512, 2048, 4096, 8192, 32768])
@pytest.mark.parametrize("items", [149, 150, 256, 296, 300, 512, 600, 2048])
def test_a_batch_that_fills_the_gpu_gets_one_cta_each(items, bound):
    """More CTAs gain at most a few per cent on a full cache and cost several times the time on a short context."""
    assert size(items, bound) == 1


def test_few_long_sequences_share_their_keys():
    assert size(1, 32768) == 8 and size(2, 2048) == 8 and size(32, 8192) == 8
    # clusters that do not all run at once would take a second round
    assert size(33, 8192) == 4 and size(64, 2048) == 4 and size(72, 8192) == 2


def test_the_clusters_that_fit_the_device_count():
    assert size(32, 16384) == 8 and size(32, 16384, (296, 264, 240)) == 4
    assert size(64, 8192, (296, 240, 192)) == 2
    assert size(1, 32768, (296, 264, 0)) == 4 and size(1, 32768, (0, 0, 0)) == 1  # a size that does not fit at all


@pytest.mark.parametrize("items", [1, 7, 16, 100])
def test_every_warp_of_a_cluster_has_a_tile_and_short_bounds_get_one_cta(items):
    for bound in (1, 16, 127, 128, 255, 256, 511, 512, 1023, 1024, 4096):
        s = size(items, bound)
        assert s in (1, 2, 4, 8) and (s == 1 or bound >= s * 4 * 16)
        assert s == 1 or bound > 128


def test_bad_arguments():
    assert size(0, 64) == -1 and size(1, 0) == -1
