"""The combine at the edges of its launch rules: split counts around 8, 32 and 64, rows that do not fill a warp's four,
rows with one live split or none, and garbage in the others."""
import numpy as np
import pytest
import torch

from oracle import paged_int8_attention as orc
from pth_flash_attn_b200 import host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("S", [2, 7, 8, 9, 31, 32, 33, 64, 65, 129, 513])
def test_split_counts(S, D, out_dtype):
    T, Hq, used = 5, 3, 4                                    # the last token is padding
    rng = np.random.default_rng(S * D)
    o = rng.standard_normal((S, T, Hq, D)).astype(np.float32)
    lse = rng.uniform(-20, 20, (S, T, Hq)).astype(np.float32)
    live = rng.random((S, T, Hq)) < min(1.0, 6 / S)          # a few pieces of the bound
    live[:, 0, 0] = False                                     # a row without keys
    live[:, 0, 1] = False
    live[S - 1, 0, 1] = True                                  # one piece, the last
    live[:, 1, :] = True                                      # every split
    lse[~live] = -np.inf
    o[~live] = np.nan
    want, want_l2 = orc.combine_partials(np.where(live[..., None], o, 0), lse)
    out = torch.full((T, Hq, D), 7.0, dtype=out_dtype, device="cuda")
    lse_out = torch.full((T, Hq), 7.0, device="cuda")
    qsl = torch.tensor([0, 1, used], dtype=torch.int32, device="cuda")
    host.combine_partials(torch.from_numpy(o).cuda(), torch.from_numpy(lse).cuda(), out, qsl, lse_out=lse_out)
    got, got_lse = out.float().cpu().numpy(), lse_out.cpu().numpy()
    assert (got[used:] == 7.0).all() and (got_lse[used:] == 7.0).all()
    # weights and their sum are exact to a few 2^-22 (exp2f, one rounding per addition); bf16 rounds by 2^-9 of a value
    tol = 1e-5 if out_dtype == torch.float32 else 2 ** -8
    np.testing.assert_allclose(got[:used], want[:used], rtol=tol, atol=1e-5)
    empty = np.isneginf(want_l2[:used])
    assert np.array_equal(np.isneginf(got_lse[:used]), empty) and empty[0, 0]
    np.testing.assert_allclose(got_lse[:used][~empty], want_l2[:used][~empty] * np.log(2), rtol=1e-5, atol=1e-5)
