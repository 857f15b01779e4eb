"""Row-major kernels with few row tiles and no workspace: CTAs of a cluster share a row tile's keys and merge their rows
through distributed shared memory.  Lengths around the number of tiles that decides how many take part, rows that some
of the pieces do not see, every output type, and rows made NaN or without finite scores by their inputs."""
import numpy as np
import pytest
import torch

from oracle import paged_int8_attention as orc
from pth_flash_attn_b200 import capi
from tests.gpu_util import run_case
from tests.helpers import check_lse, check_out

pytestmark = pytest.mark.gpu


def _run(qlens, priors, D, G, Hkv, seed, out_dtype=torch.bfloat16, window=0, edit=None):
    rng = np.random.default_rng(seed)
    c = orc.make_paged_cache([a + b for a, b in zip(qlens, priors)], Hkv, D, 16, seed=seed)
    q = orc.round_to_bf16(rng.standard_normal((sum(qlens), Hkv * G, D), dtype=np.float32))
    if edit is not None:
        edit(q)
    qsl = np.concatenate([[0], np.cumsum(qlens)]).astype(np.int64)
    kw = dict(window=window) if window else {}
    with np.errstate(all="ignore"):
        ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5, **kw)
    res = run_case(c, q, qsl, D ** -0.5, bq=(128 if D == 256 else 256 if D == 64 else 128) // G, num_splits=1,
                   kernel=capi.KERNEL_UMMA_ROWS, out_dtype=out_dtype, q_dtype=torch.bfloat16, **kw)
    assert capi.load_library().device_status() == 0
    assert res["tail_intact"]
    return res, ref


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("prior", [0, 100, 400, 511, 900, 1025, 1930, 2048, 5000])
def test_lengths(D, prior):
    res, ref = _run([37], [prior], D, 4, 1, seed=D + prior)
    check_out(res["out"], ref.out, what=f"D{D} prior {prior}")
    check_lse(res["lse"], ref.lse, what=f"D{D} prior {prior}")


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("requests, prior, ctas", [(1, 400, 1), (1, 900, 4), (1, 1930, 8), (1, 5000, 16), (160, 5000, 1)])
def test_how_many_ctas_share_a_row_tile(D, requests, prior, ctas):
    """From 8 tiles on a power of two with two tiles each, on SMs that the launch leaves idle (none beside 160 requests)."""
    res, ref = _run([37] + [1] * (requests - 1), [prior] + [5] * (requests - 1), D, 4, 1, seed=D + ctas)
    assert capi.load_library().lib.pthb200_test_row_cluster() == ctas
    check_out(res["out"], ref.out, what=f"D{D} prior {prior}")


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("D, G, Hkv, qlens, priors", [
    (128, 8, 1, [300], [0]), (128, 1, 2, [600], [700]), (128, 5, 2, [1, 130, 0, 40], [3000, 0, 500, 1290]),
    (64, 4, 2, [400, 7], [0, 4000]), (256, 6, 2, [120, 22], [1000, 0]), (256, 1, 1, [400], [0])])
def test_rows_that_some_pieces_do_not_see(D, G, Hkv, qlens, priors, out_dtype):
    res, ref = _run(qlens, priors, D, G, Hkv, seed=D + G, out_dtype=out_dtype)
    check_out(res["out"], ref.out, what=f"D{D} {qlens}")
    check_lse(res["lse"], ref.lse, what=f"D{D} {qlens}")


@pytest.mark.parametrize("window", [100, 513, 1500])
def test_window(window):
    res, ref = _run([200, 16], [2500, 1000], 128, 4, 1, seed=window, window=window)
    check_out(res["out"], ref.out, what=f"window {window}")


@pytest.mark.parametrize("D", [64, 128, 256])
def test_rows_that_are_nan(D):
    def edit(q):
        q[5, 1] = np.nan
        q[20, 2, 3] = np.inf
    alone, _ = _run([40], [3000], D, 4, 1, seed=D, edit=edit)
    many, _ = _run([40] * 160, [3000] + [5] * 159, D, 4, 1, seed=D, edit=edit)  # row tiles for every SM: no clusters
    want = np.zeros((40, 4), dtype=bool)
    want[5, 1] = want[20, 2] = True
    for res in (alone, many):
        nan = np.isnan(res["out"][:40])
        assert (nan.all(-1) == want).all() and (nan.any(-1) == want).all()
        assert (np.isneginf(res["lse"][:40]) == want).all()


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("lens", [[30, 9, 40, 120], [1500, 9, 700, 2000]])
def test_bound_on_pieces_above_what_the_lengths_allow(D, lens):
    """Pieces that a row of the block table is too short for get no CTA; they read as holding no keys all the same."""
    qlens, rng = [30, 9, 0, 25], np.random.default_rng(D)
    c = orc.make_paged_cache(lens, 2, D, 16, seed=D)
    q = orc.round_to_bf16(rng.standard_normal((sum(qlens), 8, D), dtype=np.float32))
    qsl = np.concatenate([[0], np.cumsum(qlens)]).astype(np.int64)
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    res = run_case(c, q, qsl, D ** -0.5, bq=16, num_splits=24, kernel=capi.KERNEL_UMMA_ROWS)
    assert capi.load_library().device_status() == 0
    check_out(res["out"], ref.out, what=f"D{D} {lens}")
    check_lse(res["lse"], ref.lse, what=f"D{D} {lens}")
    most = (-(-max(lens) // 128) + 2) // 4
    assert np.isneginf(res["ws_lse"][max(1, most):]).all()


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("lens", [[30, 9, 40, 120], [1500, 9, 700, 2000], [9000, 20, 30, 40]])
def test_pieces_that_find_nothing(D, lens):
    """A block table as wide as the longest context an engine allows: every piece of the bound gets a CTA, few find keys."""
    qlens, rng = [30, 9, 0, 25], np.random.default_rng(D + 1)
    c = orc.make_paged_cache(lens, 2, D, 16, seed=D + 1)
    q = orc.round_to_bf16(rng.standard_normal((sum(qlens), 8, D), dtype=np.float32))
    qsl = np.concatenate([[0], np.cumsum(qlens)]).astype(np.int64)
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    c.block_table = np.pad(c.block_table, ((0, 0), (0, 8192 - c.block_table.shape[1])))
    res = run_case(c, q, qsl, D ** -0.5, bq=16, num_splits=24, kernel=capi.KERNEL_UMMA_ROWS)
    assert capi.load_library().device_status() == 0
    check_out(res["out"], ref.out, what=f"D{D} {lens}")
    check_lse(res["lse"], ref.lse, what=f"D{D} {lens}")
    tiles = sum(-(-n // 128) * -(-4 * t // (128 if D == 256 else 256)) for n, t in zip(lens, qlens))
    used = int((~np.isneginf(res["ws_lse"])).any(axis=(1, 2)).sum())
    assert 1 <= used <= max(1, -(-max(lens) // 128) // 4 + 1) and (tiles < 16 or used > 1)
