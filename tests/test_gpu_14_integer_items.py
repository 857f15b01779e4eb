"""Integer kernel: items of every row count in one launch, and launches dealt out in ranges.

One instance serves row tiles of 1 to 16 rows with loops of its own for 4, 8 and 16, and the two softmax groups
write alternate rows of an item; a launch with enough KV tiles is cut into equal runs of the tile sequence
(csrc/sched.cuh), here with cuts next to the ends of row tiles, in requests of a tile or two and in launches
whose KV heads do not divide the number of SMs.
"""
import numpy as np
import pytest
import torch

from oracle import paged_int8_attention as orc
from pth_flash_attn_b200 import capi, host
from tests.gpu_util import run_case
from tests.helpers import check_lse, check_out

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [1, 3])
@pytest.mark.parametrize("D, G, bq, qlens", [
    (128, 4, 4, [1, 2, 3, 4, 1, 4]), (128, 1, 16, [1, 4, 5, 8, 9, 16, 15]), (128, 5, 3, [3, 1, 2, 3]),
    (64, 4, 4, [4, 1, 2, 3]), (64, 8, 2, [2, 1, 1]), (256, 4, 4, [1, 4, 3, 2]), (256, 6, 2, [2, 1]), (128, 8, 4, [4, 1, 3, 2])])
def test_row_counts_in_one_launch(D, G, bq, qlens, S):
    lens = [q + 61 * (17 * r % 13) for r, q in enumerate(qlens)]
    c = orc.make_paged_cache(lens, 2, D, 16, seed=D + G)
    q = orc.round_to_bf16(np.random.default_rng(G).standard_normal((sum(qlens), 2 * G, D), dtype=np.float32))
    qsl = np.concatenate([[0], np.cumsum(qlens)]).astype(np.int64)
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    res = run_case(c, q, qsl, D ** -0.5, bq=bq, num_splits=S, kernel=capi.KERNEL_UMMA)
    assert capi.load_library().device_status() == 0
    check_out(res["out"], ref.out, what=f"D{D} G{G} S{S}")
    check_lse(res["lse"], ref.lse, what=f"D{D} G{G} S{S}")
    assert res["tail_intact"]


def _device_cache(lens, Hkv, D, hnd, gen):
    """Random cells in 16-slot pages, one request after the other; the op's views and the dense fp64 K and V."""
    pages = [-(-n // 16) for n in lens]
    cell, blocks = 2 * D + 8, sum(pages)
    shape = (blocks, Hkv, 16) if hnd else (blocks, 16, Hkv)
    storage = torch.randint(0, 256, (*shape, cell), generator=gen, device="cuda", dtype=torch.uint8)
    words = storage.view(torch.float32)
    for at in (D // 4, D // 2 + 1):
        words[..., at] = torch.rand(shape, generator=gen, device="cuda") * 0.02 + 0.001
    cells = storage.view(torch.int8)
    if hnd:
        cells, words = cells.transpose(1, 2), words.transpose(1, 2)
    k, v, ks, vs = cells[..., :D], cells[..., D + 4:2 * D + 4], words[..., D // 4], words[..., D // 2 + 1]
    table = torch.zeros((len(lens), max(pages)), dtype=torch.int32, device="cuda")
    first = 0
    for r, n in enumerate(pages):
        table[r, :n] = torch.arange(first, first + n, device="cuda", dtype=torch.int32)
        first += n
    dense = []
    for r, n in enumerate(lens):
        b = table[r, :pages[r]].long()
        flat = [t[b].reshape(-1, Hkv, *t.shape[3:])[:n].double() for t in (k, ks, v, vs)]
        dense.append((flat[0] * flat[1][..., None], flat[2] * flat[3][..., None]))
    return storage, host.CacheViews.from_tensors(k, v, ks, vs), table, dense


@pytest.mark.parametrize("Hkv, D, G, qlen, hnd, S, lens", [
    (8, 128, 4, 1, False, 37, [20000, 130, 33000, 127, 24000, 1, 4100, 256]),
    (8, 128, 2, 4, True, 37, [90000, 5, 128, 129, 6000]),
    (3, 64, 4, 1, True, 90, [70000, 64, 1, 90000, 300, 60000]),
    (2, 256, 6, 1, True, 40, [8192] * 41),
    (1, 128, 8, 1, False, 296, [300000, 128, 400000, 3]),
    (16, 128, 1, 2, False, 9, [300 + 40 * r for r in range(100)]),
])
def test_ranges(Hkv, D, G, qlen, hnd, S, lens):
    gen = torch.Generator(device="cuda").manual_seed(Hkv + D)
    lens = [max(n, qlen) for n in lens]
    qsl = np.arange(len(lens) + 1) * qlen
    planned = capi.load_library().schedule(qsl, lens, group=G, num_kv_heads=Hkv, bq=qlen, num_splits=S, num_ctas=148, ranges=True)
    assert len(planned) > 0 and planned[:, 5].max() > 1
    storage, views, table, dense = _device_cache(lens, Hkv, D, hnd, gen)
    T, Hq = qlen * len(lens), Hkv * G
    q = torch.randn((T, Hq, D), generator=gen, device="cuda").to(torch.bfloat16)
    out = torch.full_like(q, float("nan"))
    lse = torch.full((T, Hq), float("nan"), device="cuda")
    ws_o = torch.full((S, T, Hq, D), float("nan"), device="cuda")
    ws_lse = torch.full((S, T, Hq), float("nan"), device="cuda")
    host.attention_forward(q, out, views, table, torch.tensor(lens, dtype=torch.int32, device="cuda"),
                           torch.tensor(qsl, dtype=torch.int32, device="cuda"), bq=qlen, num_splits=S, softmax_scale=D ** -0.5,
                           ws_o=ws_o, ws_lse=ws_lse, lse_out=lse, kernel=capi.KERNEL_UMMA)
    torch.cuda.synchronize()
    assert capi.load_library().device_status() == 0
    for r, (k, v) in enumerate(dense):
        n, rows = lens[r], slice(r * qlen, (r + 1) * qlen)
        s = torch.einsum("tgrd,ngd->tgrn", q[rows].double().view(qlen, Hkv, G, D), k) * D ** -0.5
        pos = torch.arange(n, device="cuda")
        s = s.masked_fill(pos > torch.arange(n - qlen, n, device="cuda")[:, None, None, None], float("-inf"))
        ref = torch.einsum("tgrn,ngd->tgrd", s.softmax(-1), v).reshape(qlen, Hq, D)
        check_out(out[rows].float().cpu().numpy(), ref.cpu().numpy(), what=f"request {r}")
        check_lse(lse[rows].cpu().numpy(), s.logsumexp(-1).reshape(qlen, Hq).cpu().numpy(), what=f"request {r}")


@pytest.mark.parametrize("Hkv, G, bq, S, window, kernel, qlens, lens", [
    (8, 4, 4, 37, 0, "UMMA", [10, 3, 4, 1, 9], [20000, 130, 33000, 127, 9000]),           # two or three row tiles a request
    (2, 4, 2, 60, 0, "UMMA", [7, 1, 8], [60000, 900, 50000]),
    (8, 2, 4, 37, 3000, "UMMA", [20, 3, 16, 17], [20000, 130, 33000, 4000]),              # row tiles of different first tiles
    (2, 4, 2, 20, 900, "UMMA", [40, 64, 33] * 3, [9000, 200, 4000] * 3),
    (8, 4, 16, 37, 0, "AUTO", [1, 200, 1, 4, 70, 2], [40000, 2000, 300, 20000, 90, 9000]),    # the short requests of a pair launch
    (2, 4, 16, 60, 0, "AUTO", [100, 1, 1, 3], [1500, 90000, 4000, 50000]),
])
def test_ranges_of_several_row_tiles_and_of_pair_launches(Hkv, G, bq, S, window, kernel, qlens, lens):
    D, qsl = 128, np.concatenate([[0], np.cumsum(qlens)])
    pair = dict(bq=16 // G, row_class=1, class_rows=16) if kernel == "AUTO" else dict(bq=bq)
    planned = capi.load_library().schedule(qsl, lens, group=G, num_kv_heads=Hkv, num_splits=S, num_ctas=148, window=window,
                                           ranges=True, **pair)
    assert len(planned) > 0 and planned[:, 5].max() > 1
    if kernel == "UMMA":
        assert planned[:, 2].max() > 0
    gen = torch.Generator(device="cuda").manual_seed(Hkv + G + window)
    storage, views, table, dense = _device_cache(lens, Hkv, D, False, gen)
    T, Hq = sum(qlens), Hkv * G
    q = torch.randn((T, Hq, D), generator=gen, device="cuda").to(torch.bfloat16)
    out = torch.full_like(q, float("nan"))
    lse = torch.full((T, Hq), float("nan"), device="cuda")
    ws_o = torch.full((S, T, Hq, D), float("nan"), device="cuda")
    ws_lse = torch.full((S, T, Hq), float("nan"), device="cuda")
    host.attention_forward(q, out, views, table, torch.tensor(lens, dtype=torch.int32, device="cuda"),
                           torch.tensor(qsl, dtype=torch.int32, device="cuda"), bq=bq, num_splits=S, softmax_scale=D ** -0.5,
                           ws_o=ws_o, ws_lse=ws_lse, lse_out=lse, window=window, kernel=getattr(capi, f"KERNEL_{kernel}"))
    torch.cuda.synchronize()
    assert capi.load_library().device_status() == 0
    for r, (k, v) in enumerate(dense):
        n, rows = lens[r], slice(int(qsl[r]), int(qsl[r + 1]))
        pos, at = torch.arange(n, device="cuda"), torch.arange(n - qlens[r], n, device="cuda")[:, None]
        hidden = (pos > at) | (pos <= at - window if window else pos < 0)
        for h in range(Hkv):
            s = torch.einsum("trd,nd->trn", q[rows, h * G:(h + 1) * G].double(), k[:, h]) * D ** -0.5
            s = s.masked_fill(hidden[:, None], float("-inf"))
            ref = torch.einsum("trn,nd->trd", s.softmax(-1), v[:, h])
            check_out(out[rows, h * G:(h + 1) * G].float().cpu().numpy(), ref.cpu().numpy(), what=f"request {r} head {h}")
            check_lse(lse[rows, h * G:(h + 1) * G].cpu().numpy(), s.logsumexp(-1).cpu().numpy(), what=f"request {r} head {h}")


@pytest.mark.parametrize("D, G, bq", [(128, 2, 2), (128, 2, 4), (64, 4, 4), (256, 1, 4)])
@pytest.mark.parametrize("S", [1, 2])
def test_rows_without_keys_beside_an_infinite_scale(D, G, bq, S):
    """More query tokens than keys: the first see none and are zero, whatever the cells hold that the others see."""
    c = orc.make_paged_cache([bq - 1, 300], 1, D, 16, seed=D)
    c.v_scale[c.block_table[0, 0], 0] = np.inf                # (what the writer makes of a row with an infinity)
    q = orc.round_to_bf16(np.random.default_rng(D).standard_normal((bq + 1, G, D), dtype=np.float32))
    res = run_case(c, q, [0, bq, bq + 1], D ** -0.5, bq=bq, num_splits=S, kernel=capi.KERNEL_UMMA)
    assert capi.load_library().device_status() == 0
    assert (res["out"][0] == 0).all() and np.isneginf(res["lse"][0]).all()
    assert not np.isfinite(res["out"][1:bq]).any() and np.isfinite(res["out"][bq]).all()
