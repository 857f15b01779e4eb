"""GPU parity of the row-major kernels' fp16 operands: queries in both types at the edges of row and
key tiles, and the scalings that keep fp16's range out of the results (the power of two of bf16
queries, the weighted probabilities)."""
import numpy as np
import pytest
import torch

from oracle import paged_int8_attention as orc
from pth_flash_attn_b200 import capi
from tests.helpers import check_lse, check_out

pytestmark = pytest.mark.gpu

# (head size, query tokens at G = 4): the one-tile kernel, the two-row-tile kernel at both of its
# head sizes, the 256-dim kernel
SHAPES = [(128, 16), (128, 70), (64, 70), (256, 40)]


def _run(c, q, qsl, D, bq, **kw):
    from tests.gpu_util import run_case

    res = run_case(c, q, qsl, D ** -0.5, bq=bq, kernel=capi.KERNEL_UMMA_ROWS, **kw)
    assert capi.load_library().device_status() == 0
    return res


@pytest.mark.parametrize("q_dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("qlen", [5, 31, 32, 33, 63, 64, 65])   # around 128 and 256 rows at G = 4
@pytest.mark.parametrize("D", [64, 128, 256])
def test_row_and_key_tile_edges(D, qlen, q_dtype):
    lens = [max(n, qlen) for n in (qlen, qlen + 1, 63 + qlen, 128, 129 + qlen)]
    c = orc.make_paged_cache(lens, 2, D, 16, seed=40 + qlen, layout="NHD" if qlen % 2 else "HND")
    rng = np.random.default_rng(qlen)
    q = orc.round_to_bf16(rng.standard_normal((qlen * len(lens), 8, D), dtype=np.float32))
    q = orc.round_to_bf16(q.astype(np.float16).astype(np.float32))   # exact in both types
    qsl = np.arange(len(lens) + 1) * qlen
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    res = _run(c, q, qsl, D, 16, q_dtype=q_dtype, out_dtype=torch.float32)
    # P and the MMA operands are fp16: every term is off by at most 2^-11 of itself, |out| <= max |v| < 8
    check_out(res["out"], ref.out, max_tol=8 * 2.0 ** -11, mean_tol=2.0 ** -11, what=f"D{D} q{qlen}")
    check_lse(res["lse"], ref.lse)
    assert res["tail_intact"]


@pytest.mark.parametrize("D,qlen", SHAPES)
def test_a_row_of_infinities_leaves_the_other_rows_alone(D, qlen):
    c = orc.make_paged_cache([300], 2, D, 16, seed=9)
    rng = np.random.default_rng(10)
    q = orc.round_to_bf16(rng.standard_normal((qlen, 8, D), dtype=np.float32))
    qsl = np.array([0, qlen])
    clean = _run(c, q, qsl, D, 16, out_dtype=torch.float32)
    q[3, 2] = np.inf
    q[4, 5, ::2] = np.nan
    dirty = _run(c, q, qsl, D, 16, out_dtype=torch.float32)
    others = np.ones((qlen, 8), dtype=bool)
    others[3, 2] = others[4, 5] = False
    out = lambda r: r["out"].reshape(qlen, 8, D)[others]  # noqa: E731
    assert np.array_equal(out(dirty), out(clean))
    assert np.array_equal(dirty["lse"][others], clean["lse"][others])
    assert not np.isfinite(dirty["out"].reshape(qlen, 8, D)[3, 2]).any()


@pytest.mark.parametrize("D,qlen", SHAPES)
def test_a_huge_finite_row_leaves_the_other_rows_alone(D, qlen):
    """The power of two of bf16 queries is the row's own: beside a row near the type's largest value and one near
    its smallest, the ordinary rows keep every bit."""
    c = orc.make_paged_cache([300], 2, D, 16, seed=9)
    rng = np.random.default_rng(10)
    q = orc.round_to_bf16(rng.standard_normal((qlen, 8, D), dtype=np.float32))
    qsl = np.array([0, qlen])
    clean = _run(c, q, qsl, D, 16, out_dtype=torch.float32)
    q[3, 2] = np.where(rng.random(D) < 0.5, 3e38, -3e38)
    q[4, 5] *= np.float32(2.0 ** -120)
    dirty = _run(c, q, qsl, D, 16, out_dtype=torch.float32)
    others = np.ones((qlen, 8), dtype=bool)
    others[3, 2] = others[4, 5] = False
    out = lambda r: r["out"].reshape(qlen, 8, D)  # noqa: E731
    assert np.array_equal(out(dirty)[others], out(clean)[others])
    assert np.array_equal(dirty["lse"][others], clean["lse"][others])
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    others[4, 5] = True   # (a row of tiny queries weighs its keys alike)
    check_out(out(dirty)[others], ref.out.reshape(qlen, 8, D)[others], max_tol=8 * 2.0 ** -11, mean_tol=2.0 ** -11)
    check_lse(dirty["lse"][others], ref.lse.reshape(qlen, 8)[others])


@pytest.mark.parametrize("D,qlen", SHAPES)
def test_every_row_with_a_power_of_two_of_its_own(D, qlen):
    """Rows on both sides of the limits between which the common power serves (largest value in [2^-4, 2^8)), mixed
    in every warp, against the oracle: the scaling is exact, so only the scores' own rounding may show."""
    c = orc.make_paged_cache([200], 2, D, 16, seed=17)
    rng = np.random.default_rng(18)
    q = orc.round_to_bf16(rng.standard_normal((qlen, 8, D), dtype=np.float32))
    q /= np.abs(q).max(axis=-1, keepdims=True)          # largest magnitude of every row: one
    top = np.exp2(rng.integers(-6, 9, (qlen, 8, 1)).astype(np.float32)) * rng.choice([1.0, 0.99609375], (qlen, 8, 1))
    q = orc.round_to_bf16((q * top).astype(np.float32))
    qsl = np.array([0, qlen])
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    res = _run(c, q, qsl, D, 16, out_dtype=torch.float32)
    # scores reach 2^8 * 4 * sqrt(D) / ln 2 < 2^15 and are held to 2^-24 of that: P within 2^-9, |out| < 8
    check_out(res["out"], ref.out, max_tol=8 * 2.0 ** -8, mean_tol=2.0 ** -10)


@pytest.mark.parametrize("exponent", [-90, 100])
@pytest.mark.parametrize("D,qlen", SHAPES)
def test_bf16_queries_beyond_the_range_of_fp16(D, qlen, exponent):
    """Queries far outside fp16's range, their keys scaled the other way: the power of two is exact,
    so nothing but the scores' own rounding may show."""
    c = orc.make_paged_cache([200], 2, D, 16, seed=11)
    c.k_scale[...] = np.ldexp(c.k_scale, -exponent).astype(np.float32)
    rng = np.random.default_rng(12)
    q = orc.round_to_bf16(np.ldexp(rng.standard_normal((qlen, 8, D), dtype=np.float32), exponent))
    qsl = np.array([0, qlen])
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    res = _run(c, q, qsl, D, 16, out_dtype=torch.float32)
    check_out(res["out"], ref.out, max_tol=8 * 2.0 ** -11, mean_tol=2.0 ** -11)
    check_lse(res["lse"], ref.lse)


@pytest.mark.parametrize("q_dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,qlen", SHAPES)
def test_small_probabilities_beside_a_large_one(D, qlen, q_dtype):
    """One key takes nearly all the mass and has V = 0 in the odd dims; the 2^15 others, each 2^-25.5 of
    it, are all of the odd outputs.  fp16 holds P to 2^-32 of the reference."""
    n, gap = 1 << 15, 25.5
    k = np.zeros((n, 1, D), dtype=np.float32)
    k[5] = gap / (2.0 * np.log2(np.e) * D ** 0.5)   # queries are all 2
    v = np.ones((n, 1, D), dtype=np.float32)
    v[5, 0, 1::2] = 0.0
    c = orc.make_paged_cache([n], 1, D, 64, sources=[(k, v)], seed=13)
    q = np.full((qlen, 4, D), 2.0, dtype=np.float32)
    qsl = np.array([0, qlen])
    rows = [0, qlen - 1]
    ref = orc.ref_attention_paged(q[rows], c, np.array([0, 2]), D ** -0.5, causal=False)
    res = _run(c, q, qsl, D, 16, q_dtype=q_dtype, out_dtype=torch.float32, causal=False)
    got = res["out"].reshape(qlen, 4, D)[rows]
    assert ref.out.reshape(2, 4, D)[:, :, 1::2].min() > 6e-4
    # half a step of P for every key, and 2^-10 of the value for the fp32 scores' last digits
    np.testing.assert_allclose(got, ref.out.reshape(2, 4, D), rtol=2.0 ** -10, atol=n * 2.0 ** -32)
    check_lse(res["lse"][rows], ref.lse.reshape(2, 4))


@pytest.mark.parametrize("q_dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D,qlen", SHAPES)
def test_small_probabilities_keep_eight_bits(D, qlen, q_dtype):
    """The same with no allowance for P's steps: at 2^-25.5 of the reference P is 2^-14.5 and a step 2^-24, so the
    outputs are within half of bf16's step of 2^-8 (2^-10.5 of P, 2^-10 of the scores' last digits)."""
    n, gap = 1 << 15, 25.5
    k = np.zeros((n, 1, D), dtype=np.float32)
    k[5] = gap / (2.0 * np.log2(np.e) * D ** 0.5)   # queries are all 2
    v = np.ones((n, 1, D), dtype=np.float32)
    v[5, 0, 1::2] = 0.0
    c = orc.make_paged_cache([n], 1, D, 64, sources=[(k, v)], seed=13)
    q = np.full((qlen, 4, D), 2.0, dtype=np.float32)
    ref = orc.ref_attention_paged(q[:1], c, np.array([0, 1]), D ** -0.5, causal=False)
    res = _run(c, q, np.array([0, qlen]), D, 16, q_dtype=q_dtype, out_dtype=torch.float32, causal=False)
    got, want = res["out"].reshape(qlen, 4, D)[:, :, 1::2], ref.out.reshape(1, 4, D)[:, :, 1::2]
    np.testing.assert_allclose(got, np.broadcast_to(want, got.shape), rtol=2.0 ** -9)


@pytest.mark.parametrize("D,qlen", SHAPES)
def test_values_of_scale_zero_and_of_very_different_scales(D, qlen):
    c = orc.make_paged_cache([500], 2, D, 16, seed=14)
    rng = np.random.default_rng(15)
    c.v_scale[...] = (c.v_scale * np.exp2(rng.integers(-30, 1, c.v_scale.shape))).astype(np.float32)
    c.v_scale[rng.random(c.v_scale.shape) < 0.3] = 0.0
    q = orc.round_to_bf16(rng.standard_normal((qlen, 8, D), dtype=np.float32))
    qsl = np.array([0, qlen])
    ref = orc.ref_attention_paged(q, c, qsl, D ** -0.5)
    res = _run(c, q, qsl, D, 16, out_dtype=torch.float32)
    check_out(res["out"], ref.out, max_tol=8 * 2.0 ** -11, mean_tol=2.0 ** -11)
    check_lse(res["lse"], ref.lse)
