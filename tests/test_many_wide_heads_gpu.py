"""Fused decode attention where blocks of a wide head outnumber the SMs (four warps a block, stages of 64 keys)."""
import math

import pytest
import torch

from test_kernels_gpu import _fused_decode_case, attention_reference, close, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_dim,block_size,lengths,window,splits", [
    (24, 24, 128, 64, [1, 16, 63, 64, 65, 128, 129, 700], 0, 1),          # pieces that end at a stage's edge
    (32, 8, 128, 16, [300] * 9 + [65, 2, 1000] * 4, 0, 1),                # four query heads a key head
    (24, 24, 128, 64, [700, 64, 129, 33], 0, 2),                          # two blocks a context
    (24, 24, 128, 64, [400, 90, 61, 1, 64, 65, 200], 50, 1),              # a window
    (38, 38, 80, 16, [130, 64, 5, 257], 0, 1),                            # rows that are padded, not swizzled
    (80, 80, 192, 32, [150, 64], 0, 1),
])
def test_more_blocks_than_sms(heads, kv_heads, head_dim, block_size, lengths, window, splits):
    dtype, n, scale = torch.bfloat16, len(lengths), 0.5 / math.sqrt(head_dim)
    assert n * kv_heads * splits > torch.cuda.get_device_properties(0).multi_processor_count
    k = lib(dtype, head_dim)
    setup, qkv, table, _ = _fused_decode_case(dtype, lengths, heads, kv_heads, head_dim, block_size, seed=heads + head_dim)
    out = torch.full((n, heads * head_dim), float("nan"), device="cuda").to(dtype)
    k.attention_decode_fused(qkv, table, setup["k_cache"], setup["v_cache"], setup["table"],
                             torch.tensor(lengths, dtype=torch.int32, device="cuda"), out, heads, kv_heads, head_dim,
                             block_size, scale, window, splits, True)
    close(out, attention_reference(setup, dtype, heads, kv_heads, scale, window).view(n, -1), dtype)
