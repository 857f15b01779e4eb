"""The schedule that deals a launch out in ranges, checked on the host (csrc/sched.cuh ``range_sched``)."""
import numpy as np
import pytest

from pth_flash_attn_b200 import capi

KV_TILE = 128


def _tiles(seq_len, q_len, row_tile, bq, window):
    """First and end KV tile that the rows of a row tile see together (causal)."""
    first, last = row_tile * bq, min(q_len, row_tile * bq + bq) - 1
    lo = max(0, seq_len - q_len + first - window + 1) if window else 0
    end = seq_len - q_len + last + 1
    return (lo // KV_TILE, -(-end // KV_TILE)) if end > lo else (lo // KV_TILE, lo // KV_TILE)


def _check(items, qlens, lens, *, Hkv, bq, S, ctas, window=0):
    """Every row tile and KV head once, its pieces in order and none too many."""
    by_key = {}
    for cta, r, rt, kvh, split, splits, tb, te in items.tolist():
        by_key.setdefault((r, rt, kvh), []).append((split, splits, tb, te))
    assert set(by_key) == {(r, rt, h) for r, q in enumerate(qlens) for rt in range(-(-q // bq)) for h in range(Hkv)}
    for (r, rt, _), pieces in by_key.items():
        pieces.sort()
        splits = pieces[0][1]
        assert splits <= S and [p[0] for p in pieces] == list(range(splits)), pieces
        t0, t1 = _tiles(lens[r], qlens[r], rt, bq, window)
        assert pieces[0][2] == t0 and pieces[-1][3] == t1
        assert all(a[3] == b[2] for a, b in zip(pieces, pieces[1:]))


@pytest.mark.parametrize("seed", range(40))
def test_random_launches_are_covered_exactly_once(seed):
    rng = np.random.default_rng(seed)
    R, Hkv = int(rng.integers(1, 70)), int(rng.choice([1, 2, 3, 5, 8, 16]))
    bq, ctas = int(rng.choice([1, 2, 4])), int(rng.choice([7, 148, 148, 160]))
    qlens = rng.integers(0, bq + 1 if seed % 2 else 3 * bq + 1, size=R).tolist()
    lens = [int(q + rng.integers(1, int(rng.choice([300, 9000, 70000])))) for q in qlens]
    window = int(rng.choice([0, 0, 3000]))
    S = int(rng.choice([2, 5, 37, 296]))
    items = capi.load_library().schedule(np.concatenate([[0], np.cumsum(qlens)]), lens, group=4, num_kv_heads=Hkv, bq=bq,
                                         num_splits=S, num_ctas=ctas, window=window, ranges=True)
    if len(items):
        _check(items, qlens, lens, Hkv=Hkv, bq=bq, S=S, ctas=ctas, window=window)


@pytest.mark.parametrize("seed", range(40))
def test_random_launches_that_are_dealt_out(seed):
    """Launches drawn until one is dealt out in ranges (about every second is): one row tile a request and several."""
    rng = np.random.default_rng(1000 + seed)
    for _ in range(40):
        R, Hkv = int(rng.integers(1, 70)), int(rng.choice([1, 2, 3, 5, 8, 16]))
        bq, ctas = int(rng.choice([1, 2, 4])), int(rng.choice([7, 148, 148, 160]))
        qlens = rng.integers(0, bq + 1 if seed % 2 else 3 * bq + 1, size=R).tolist()
        lens = [int(q + rng.integers(1, int(rng.choice([300, 9000, 70000])))) for q in qlens]
        window, S = int(rng.choice([0, 0, 3000])), int(rng.choice([2, 5, 37, 296]))
        items = capi.load_library().schedule(np.concatenate([[0], np.cumsum(qlens)]), lens, group=4, num_kv_heads=Hkv, bq=bq,
                                             num_splits=S, num_ctas=ctas, window=window, ranges=True)
        if len(items):
            break
    assert len(items)
    _check(items, qlens, lens, Hkv=Hkv, bq=bq, S=S, ctas=ctas, window=window)


@pytest.mark.parametrize("lens, Hkv, S, least", [
    ([8192] * 64, 2, 37, 0.95),                                 # two heads: 256 equal pieces would take two rounds of 148
    ([8192] * 64, 8, 5, 0.98),
    ([131072], 8, 37, 0.97),
    (list(range(4096, 131072, 2700)), 8, 8, 0.98),
    ([37 * k % 988 + 1 for k in range(200)], 8, 5, 0.90),       # a few tiles per request: a CTA has 40
])
def test_ctas_get_equal_loads(lens, Hkv, S, least):
    items = capi.load_library().schedule(np.arange(len(lens) + 1), lens, group=4, num_kv_heads=Hkv, bq=1, num_splits=S,
                                         num_ctas=148, ranges=True)
    load = np.bincount(items[:, 0], weights=items[:, 7] - items[:, 6], minlength=148)
    assert load.mean() >= least * load.max()
    _check(items, [1] * len(lens), lens, Hkv=Hkv, bq=1, S=S, ctas=148)


def test_launches_that_keep_equal_pieces():
    lib = capi.load_library()

    def items(lens, S, Hkv=8, qlens=None):
        qlens = qlens or [1] * len(lens)
        return lib.schedule(np.concatenate([[0], np.cumsum(qlens)]), lens, group=4, num_kv_heads=Hkv, bq=1, num_splits=S,
                            num_ctas=148, ranges=True)
    assert len(items([8192] * 64, 1)) == 0                      # no workspace for pieces
    assert len(items([131072], 8)) == 0                         # 20 pieces do not fit 8
    assert len(items([900] * 8, 37)) == 0                       # not enough work
    assert len(items([8192] * 64 + [0], 5)) == 0                # a request without keys has no tiles to find it by
    assert len(items([8192] * 64 + [0], 5, qlens=[1] * 64 + [0])) > 0   # (padding without queries is nothing at all)
