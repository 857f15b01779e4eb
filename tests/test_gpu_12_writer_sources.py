"""GPU test of the cache writer's load paths: sources on and off 8-byte boundaries, cell counts around
what a warp and a CTA take, NaN and infinities; bytes equal the oracle's."""
import numpy as np
import pytest
import torch

from oracle import paged_int8_attention as orc
from pth_flash_attn_b200 import host
from tests.test_gpu_7_writer import _empty_cache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 4])     # elements off the tensor's start
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("T,Hkv,D", [(1, 1, 64), (3, 1, 128), (33, 1, 128), (11, 3, 64), (17, 2, 256), (64, 8, 128)])
def test_bytes_whatever_the_alignment_of_the_source(T, Hkv, D, dtype, offset):
    from tests.gpu_util import cache_to_device

    c = _empty_cache(-(-T // 16) + 1, Hkv, D, 16, "NHD", seed=T)
    rng = np.random.default_rng(T + D + offset)
    flat = torch.zeros(2, T * Hkv * D + 8, dtype=dtype)
    src = flat[:, offset:offset + T * Hkv * D].view(2, T, Hkv, D)
    src.copy_(torch.from_numpy(rng.standard_normal((2, T, Hkv, D), dtype=np.float32) * 2))
    slots = rng.permutation(c.num_blocks * 16)[:T].astype(np.int64)
    if T > 2:
        slots[T // 2] = -1
    want = c.storage.copy()
    exp = orc.PagedInt8Cache(**{**c.__dict__, "storage": want})
    live = slots >= 0
    b, s = slots[live] // 16, slots[live] % 16
    for i, (cache, scale) in enumerate(((exp.k_cache, exp.k_scale), (exp.v_cache, exp.v_scale))):
        q, sc = orc.quantize_rows(src[i].float().numpy())
        cache[b, s], scale[b, s] = q[live], sc[live]
    storage, views, _, _ = cache_to_device(c)
    dev = flat.cuda()[:, offset:offset + T * Hkv * D].view(2, T, Hkv, D)
    host.write_kv(dev[0], dev[1], views, torch.from_numpy(slots).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(storage.cpu().numpy(), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_a_nan_is_the_lowest_value_and_leaves_its_row_alone(dtype):
    """fmaxf passes a NaN by, so the scale is that of the other elements; the NaN itself clamps to -128."""
    from tests.gpu_util import cache_to_device

    c = _empty_cache(1, 1, 128, 16, "NHD", seed=3)
    x = torch.randn(1, 1, 128, generator=torch.Generator().manual_seed(4)).to(dtype)
    y = x.clone()
    y[0, 0, 7] = float("nan")
    x[0, 0, 7] = 0.0
    kq, ks = orc.quantize_rows(x.float().numpy())
    storage, views, _, _ = cache_to_device(c)
    host.write_kv(y.cuda(), x.cuda(), views, torch.zeros(1, dtype=torch.int64, device="cuda"))
    torch.cuda.synchronize()
    back = orc.PagedInt8Cache(**{**c.__dict__, "storage": storage.cpu().numpy()})
    kq = kq.copy()
    kq[0, 0, 7] = -128
    assert np.array_equal(back.k_cache[0, 0], kq[0]) and back.k_scale[0, 0, 0] == ks[0, 0]
