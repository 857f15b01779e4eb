"""Row-major kernels: the row tile of a CTA at every way of finding it (one warp, 32 requests at a time, or a shared copy
of query_start_loc beyond 96), and rows that go through shared memory on their way in and out: part-filled warps,
float32 results, strided queries."""
import numpy as np
import pytest
import torch

from oracle import paged_int8_attention as orc
from pth_flash_attn_b200 import capi
from tests.gpu_util import run_case
from tests.helpers import check_lse, check_out

pytestmark = pytest.mark.gpu


def _run(qlens, D, G, S, seed, out_dtype=torch.bfloat16, q_dtype=torch.bfloat16):
    rng = np.random.default_rng(seed)
    lens = [int(q + rng.integers(0, 150)) if q else 0 for q in qlens]
    c = orc.make_paged_cache(lens, 2, D, 16, seed=seed)
    q = rng.standard_normal((sum(qlens), 2 * G, D), dtype=np.float32)
    q = orc.round_to_bf16(q) if q_dtype == torch.bfloat16 else q.astype(np.float16).astype(np.float32)
    qsl = np.concatenate([[0], np.cumsum(qlens)]).astype(np.int64)
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    res = run_case(c, q, qsl, D ** -0.5, bq=64 // G, num_splits=S, kernel=capi.KERNEL_UMMA_ROWS, out_dtype=out_dtype, q_dtype=q_dtype)
    assert capi.load_library().device_status() == 0
    check_out(res["out"], ref.out, what=f"{len(qlens)} requests D{D} S{S}")
    check_lse(res["lse"], ref.lse, what=f"{len(qlens)} requests D{D} S{S}")
    assert res["tail_intact"]


@pytest.mark.parametrize("S", [1, 3])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("R", [1, 31, 32, 33, 64, 65, 96, 97, 130])
def test_request_counts(R, D, S):
    rng = np.random.default_rng(R + D)
    qlens = rng.integers(0, 12, size=R).tolist()
    qlens[R // 2] = 70                      # a request of several row tiles among short and empty ones
    _run(qlens, D, 4, S, seed=R + D + S)


@pytest.mark.parametrize("out_dtype, q_dtype", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("D, G, qlens", [
    (128, 4, [64, 65, 1, 127]), (128, 4, [200]), (128, 5, [52, 103, 51]), (64, 4, [64, 33]), (64, 7, [37, 100]),
    (256, 4, [33, 8, 31]), (256, 6, [21, 22, 43]), (128, 1, [256, 300, 129]), (128, 16, [17, 16, 8])])
def test_row_counts_and_types(D, G, qlens, out_dtype, q_dtype):
    _run(qlens, D, G, 1, seed=D + G, out_dtype=out_dtype, q_dtype=q_dtype)
