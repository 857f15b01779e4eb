"""The cache writer's argument block is packed by position: every named field of the structure gets its own value."""
import types

import pytest
import torch

from pth_flash_attn_b200 import capi, host


class _Lib:
    def write_kv(self, args, stream=None):
        self.args, self.stream = args, stream
        return capi.OK


def _tensor(ptr, strides, tokens, dtype=torch.bfloat16):
    """What ``write_kv`` asks of a tensor, on a device this machine need not have."""
    return types.SimpleNamespace(element_size=lambda: dtype.itemsize, stride=lambda: strides, dtype=dtype, shape=(tokens, 3, 64),
                                 device=types.SimpleNamespace(type="cuda", index=0), data_ptr=lambda: ptr)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_every_field_of_the_write_arguments_gets_its_own_value(monkeypatch, dtype):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(cuda_stream=77))
    streams = {name: tuple(1000 * (i + 1) + j for j in range(4)) for i, name in enumerate(("k", "v", "ks", "vs"))}
    cache = host.CacheViews(**streams, num_blocks=11, block_size=12, num_kv_heads=13, head_size=14)
    lib = _Lib()
    host.write_kv(_tensor(101, (201, 202, 1), 15, dtype), _tensor(102, (203, 204, 1), 15, dtype), cache,
                  _tensor(103, (1,), 15), lib=lib)
    es = dtype.itemsize
    want = dict(abi_version=capi.ABI_VERSION, key=101, value=102, src_dtype=host._DTYPE_CODE[dtype], key_stride_token=201 * es,
                key_stride_head=202 * es, value_stride_token=203 * es, value_stride_head=204 * es, num_blocks=11, block_size=12,
                num_kv_heads=13, head_size=14, num_tokens=15, slot_mapping=103)
    for field, value in want.items():
        assert getattr(lib.args, field) == value, field
    for field, name in (("k_cache", "k"), ("v_cache", "v"), ("k_scale", "ks"), ("v_scale", "vs")):
        s = getattr(lib.args, field)
        assert (s.data, s.stride_block, s.stride_slot, s.stride_head) == streams[name], field
    named = set(want) | {"struct_bytes", "k_cache", "v_cache", "k_scale", "v_scale"}
    assert named == {f for f, _ in capi.PthB200WriteArgs._fields_}
    assert lib.stream == 77
