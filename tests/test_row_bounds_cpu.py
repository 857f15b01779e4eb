"""The bounds that a row-major launch takes from its arguments (csrc/sched.cuh ``row_tile_bound``, ``pieces_bound``): pieces
and CTAs of a cluster that a row tile's keys are shared out among hang on them."""
import re
from pathlib import Path

import numpy as np
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


@pytest.mark.parametrize("seed", range(20))
def test_pieces_that_a_request_alone_rules_out(seed):
    """No launch cuts a request into more pieces than its own tiles allow, so a CTA behind them leaves without the launch's work."""
    rng = np.random.default_rng(seed)
    R, G, Hkv, bq = int(rng.integers(1, 50)), int(rng.choice([1, 4, 8])), int(rng.choice([1, 2, 8])), int(rng.choice([8, 64]))
    qlens = rng.integers(1, 3 * bq, size=R).tolist()
    lens = [int(q + rng.integers(0, int(rng.choice([100, 3000, 60000])))) for q in qlens]
    window, causal, S = int(rng.choice([0, 900])), bool(rng.integers(0, 2)), int(rng.choice([3, 37, 400]))
    items = capi.load_library().schedule(np.concatenate([[0], np.cumsum(qlens)]), lens, group=G, num_kv_heads=Hkv, bq=bq,
                                         num_splits=S, num_ctas=148, window=window, causal=causal)
    for r, (q, n) in enumerate(zip(qlens, lens)):
        mine = items[items[:, 1] == r]
        lo = max(0, n - q - window + 1) if window else 0
        end = n if causal or not window else min(n, n - 1 + window)
        tiles = -(-end // 128) - lo // 128
        assert mine[:, 5].max() <= max(1, min((tiles + 2) // 4, S))


def test_a_piece_is_ruled_out_before_the_work_of_the_launch_is_summed_up():
    code = (Path(capi.__file__).parent / "csrc" / "umma_rows.cuh").read_text()
    body = code[code.index("RowsItem rows_item("):]
    assert body.index("req_splits(kv_tiles, kItemTilesMin,") < body.index("if (split >= most) return it;") < body.index("work()")
    for name in ("umma_rows_kernel.cu", "umma_rows2_kernel.cu", "umma_rows256_kernel.cu"):
        kernel = (Path(capi.__file__).parent / "csrc" / name).read_text()
        calls = re.findall(r"rows_item<kClusters>\(([^;]*);", kernel)
        assert len(calls) == 2 and all("[&] {" in c for c in calls)
