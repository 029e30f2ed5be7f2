"""Fused decode attention where blocks of a wide head outnumber the SMs (four warps a block, stages of 64 keys), and where few blocks share
a long context (sixteen pieces)."""
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


@pytest.mark.parametrize("heads,kv_heads,head_dim,block_size,lengths,window", [
    (32, 4, 64, 64, [8100], 0), (32, 4, 64, 16, [4096], 0), (8, 2, 64, 64, [4100, 1, 300], 0),    # pieces without keys, a piece of one
    (20, 1, 128, 64, [9000, 64], 4097), (1, 1, 80, 32, [5000], 0), (8, 1, 192, 64, [4500], 0),
    (8, 2, 128, 64, [40000], 0)])               # above: a window, more than 16 heads a key head; more blocks than a block keeps of the table
def test_a_long_context_in_sixteen_pieces(heads, kv_heads, head_dim, block_size, lengths, window):
    dtype, n, scale = torch.bfloat16, len(lengths), 0.5 / math.sqrt(head_dim)
    k = lib(dtype, head_dim)
    setup, qkv, table, _ = _fused_decode_case(dtype, lengths, heads, kv_heads, head_dim, block_size, seed=heads + head_dim)
    out = torch.full((n, heads * head_dim), float("nan"), device="cuda").to(dtype)
    k.attention_decode_fused(qkv, table, setup["k_cache"], setup["v_cache"], setup["table"],
                             torch.tensor(lengths, dtype=torch.int32, device="cuda"), out, heads, kv_heads, head_dim,
                             block_size, scale, window, 8, True)
    close(out, attention_reference(setup, dtype, heads, kv_heads, scale, window).view(n, -1), dtype)


@pytest.mark.parametrize("heads,kv_heads,lengths,window,reach,splits", [(160, 160, [130], 0, 200, 1), (160, 160, [700], 90, 90, 1),
                                                                       (24, 24, [700, 1, 64, 333] * 2, 0, 400, 1), (40, 2, [520, 77], 0, 600, 8)])
def test_bias_by_distance(heads, kv_heads, lengths, window, reach, splits):
    """Against the split kernel, which reads the bias score by score: pieces whose distances end beyond the table."""
    dtype, n, head_dim, scale = torch.bfloat16, len(lengths), 128, 0.04
    k = lib(dtype, head_dim)
    setup, qkv, table, _ = _fused_decode_case(dtype, lengths, heads, kv_heads, head_dim, 64, seed=heads)
    bias = torch.rand(heads, reach, device="cuda") * 4
    ctx = torch.tensor(lengths, dtype=torch.int32, device="cuda")
    out, other = (torch.full((n, heads * head_dim), float("nan"), device="cuda").to(dtype) for _ in range(2))
    k.attention_decode_fused(qkv, table, setup["k_cache"], setup["v_cache"], setup["table"], ctx, out, heads, kv_heads, head_dim, 64, scale,
                             window, splits, True, bias=bias)
    k.attention_decode(setup["q"].view(n, -1), setup["k_cache"], setup["v_cache"], setup["table"], ctx, other, heads, kv_heads, head_dim, 64,
                       scale, window, 1, bias=bias)
    close(out, other, dtype)


@pytest.mark.parametrize("head_dim,length", [(64, 4097), (64, 4200), (128, 4097)])
def test_a_nan_is_not_lost_among_sixteen_pieces(head_dim, length):
    """The newest key alone makes its warp's scores of a piece, and it is NaN: so is the result."""
    dtype, heads, kv_heads, block_size = torch.bfloat16, 8, 2, 64
    k = lib(dtype, head_dim)
    setup, qkv, table, _ = _fused_decode_case(dtype, [length], heads, kv_heads, head_dim, block_size, seed=1)
    qkv[0, heads * head_dim:(heads + 1) * head_dim] = math.nan                    # the key of the first key head
    out = torch.zeros(1, heads, head_dim, device="cuda").to(dtype)
    k.attention_decode_fused(qkv, table, setup["k_cache"], setup["v_cache"], setup["table"], torch.tensor([length], dtype=torch.int32, device="cuda"),
                             out.view(1, -1), heads, kv_heads, head_dim, block_size, 0.1, 0, 8, True)
    assert out[0, :heads // 2].isnan().all() and out[0, heads // 2:].isfinite().all()
