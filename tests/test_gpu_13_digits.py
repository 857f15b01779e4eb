"""GPU test of the integer kernel's fixed-point probabilities at the top of their range: equal keys
under equal value scales all get the largest digits there are, and a row count decides which instance
(and which of its row groups of four) computes them."""
import numpy as np
import pytest
import torch

from oracle import paged_int8_attention as orc
from pth_flash_attn_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 700])
@pytest.mark.parametrize("D,qlen,G", [(128, 1, 3), (128, 1, 4), (128, 1, 5), (128, 2, 4), (128, 3, 4), (128, 4, 4),
                                      (128, 1, 32), (128, 1, 40), (64, 1, 1), (64, 4, 4), (64, 1, 33), (256, 1, 6),
                                      (256, 4, 4), (256, 1, 17)])
def test_equal_keys_reach_the_largest_digit(D, qlen, G, n):
    from tests.gpu_util import run_case

    n = max(n, qlen)
    rng = np.random.default_rng(D + G)
    k = np.broadcast_to(rng.standard_normal((1, 2, D), dtype=np.float32), (n, 2, D)).copy()
    v = rng.standard_normal((n, 2, D), dtype=np.float32)
    v[:, :, 0] = 4.0 * 1.015625   # every value scale is the same, and so is dim 0
    c = orc.make_paged_cache([n], 2, D, 16, sources=[(k, v)], seed=1)
    q = orc.round_to_bf16(rng.standard_normal((qlen, 2 * G, D), dtype=np.float32))
    qsl = np.array([0, qlen])
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5, causal=False)
    res = run_case(c, q, qsl, D ** -0.5, bq=qlen, kernel=capi.KERNEL_UMMA, causal=False, out_dtype=torch.float32)
    assert capi.load_library().device_status() == 0
    out, want = res["out"].reshape(qlen, 2 * G, D), ref.out.reshape(qlen, 2 * G, D)
    # two digits (tall row tiles, 256 dims): half a unit of 2^-14; three: of 2^-21; both with the fp32 sums' rounding
    digits = 3 if qlen * G <= 16 and D < 256 else 2
    np.testing.assert_allclose(out, want, rtol=0, atol=4.1 * (2.0 ** (-7 * digits) + 2.0 ** -18))
