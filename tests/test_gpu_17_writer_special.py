"""Cache writer: infinities, NaNs and every other 16-bit pattern, against the arithmetic restated in torch."""
import pytest
import torch

from pth_flash_attn_b200 import host

pytestmark = pytest.mark.gpu


def _quantised(x):
    """absmax without NaNs, scale, round half away from zero, clamp (a NaN becomes -128), in fp32 step by step."""
    x = x.float()
    amax = torch.where(x.isnan(), torch.zeros_like(x), x.abs()).amax(-1)
    scale = torch.fmax(amax / torch.full_like(amax, 127.0), torch.full_like(amax, 1e-6))  # (by a number: torch multiplies by 1 / 127)
    v = x * (torch.ones_like(scale) / scale)[..., None]
    v = v + torch.copysign(torch.full_like(v, 0.5), v)
    v = torch.fmin(torch.fmax(v, torch.full_like(v, -128.0)), torch.full_like(v, 127.0))
    return v.trunc().to(torch.int8), scale


@pytest.mark.parametrize("offset", [0, 1])          # rows on 8-byte boundaries, or two bytes off
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128, 256])
def test_every_pattern(D, dtype, offset):
    T, Hkv, page = 37, 3, 16
    gen = torch.Generator(device="cuda").manual_seed(D)
    bits = torch.randint(0, 1 << 16, (2, T, Hkv, D), generator=gen, device="cuda", dtype=torch.int32)
    special = 0x7F80 if dtype == torch.bfloat16 else 0x7C00
    finite = torch.where((bits & special) == special, bits & 0x03FF, bits)
    rows = torch.arange(T, device="cuda")[None, :, None, None]
    bits = torch.where(rows % 3 == 0, bits, finite)                    # rows of everything, and finite ones
    bits[:, 1] = 0                                                     # zeros
    bits[:, 2, :, ::2], bits[:, 2, :, 1::2] = special, 0x8000 | special  # infinities
    bits[:, 4, :, 5] = special | 1                                     # a NaN among finite values
    raw = torch.zeros(2 * T * Hkv * D + 8, dtype=torch.int16, device="cuda")
    src = raw[offset:offset + bits.numel()].view(2, T, Hkv, D)
    src.copy_(torch.where(bits >= 1 << 15, bits - (1 << 16), bits).to(torch.int16))
    src = src.view(dtype)
    cell = 2 * D + 8
    storage = torch.zeros((-(-T // page), page, Hkv, cell), dtype=torch.uint8, device="cuda")
    c, w = storage.view(torch.int8), storage.view(torch.float32)
    views = (c[..., :D], c[..., D + 4:2 * D + 4], w[..., D // 4], w[..., D // 2 + 1])
    host.write_kv(src[0], src[1], host.CacheViews.from_tensors(*views), torch.arange(T, device="cuda"))
    for got, got_scale, x in ((views[0], views[2], src[0]), (views[1], views[3], src[1])):
        want, scale = _quantised(x)
        assert torch.equal(got.reshape(-1, Hkv, D)[:T], want)
        assert torch.equal(got_scale.reshape(-1, Hkv)[:T], scale)
