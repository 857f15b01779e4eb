"""The bounds that a row-major launch takes from its arguments (csrc/sched.cuh ``row_tile_bound``, ``pieces_bound``): pieces
and CTAs of a cluster that a row tile's keys are shared out among hang on them."""
import pytest

from pth_flash_attn_b200 import capi

WIDE = (1 << 31) - 1


def _touched(window, causal, bq, first):
    """KV tiles of a row tile whose first token is at position `first` of an endless context."""
    last = first + bq - 1
    lo, hi = max(0, first - window + 1), last if causal else last + window - 1
    return hi // 128 - lo // 128 + 1


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("bq", [1, 8, 64, 256])
@pytest.mark.parametrize("window", [1, 2, 127, 128, 129, 1000, 4096])
def test_a_window_bounds_what_a_row_tile_touches(window, bq, causal):
    most = max(_touched(window, causal, bq, first) for first in range(2 * window, 2 * window + 128))
    tiles, _ = capi.load_library().row_bounds(block_table_row_stride=1 << 20, block_size=16, bq=bq, num_splits=1000,
                                              window=window, causal=causal)
    assert most <= tiles <= most + 2


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("window", [0, WIDE, WIDE - 1, WIDE // 2 + 1])
@pytest.mark.parametrize("stride, block_size, tiles", [(8192, 16, 1024), (100, 816, 638), (1, 16, 1)])
def test_a_window_beyond_every_context_leaves_the_block_table(stride, block_size, tiles, window, causal):
    got = capi.load_library().row_bounds(block_table_row_stride=stride, block_size=block_size, bq=128, num_splits=37,
                                         window=window, causal=causal)
    assert got == (tiles, max(1, min((tiles + 2) // 4, 37)))


def test_a_stride_that_says_nothing():
    assert capi.load_library().row_bounds(block_table_row_stride=0, block_size=16, bq=128, num_splits=37) == (WIDE, 37)
