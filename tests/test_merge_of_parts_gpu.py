"""The merge of a context's parts behind split decode attention: counts around what a thread takes by itself, what is asked for at once and
what the weights of a round hold, parts without keys, head sizes above and below a block's threads, a sink, a gate."""
import ctypes
import math

import pytest
import torch

from test_kernels_gpu import attention_reference, close, lib, paged_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 8, 9, 16, 17, 64, 256, 257, 513])
@pytest.mark.parametrize("head_dim", [48, 64, 128, 208, 256])
def test_parts(splits, head_dim):
    dtype, heads, kv_heads, block, lengths, scale = torch.bfloat16, 8, 2, 16, [1000, 1, 130], 0.5 / math.sqrt(head_dim)
    k = lib(dtype, head_dim)
    setup = paged_setup(dtype, lengths, [1] * 3, heads, kv_heads, head_dim, block, seed=head_dim)
    q, ctx = setup["q"].view(3, -1), torch.tensor(lengths, dtype=torch.int32, device="cuda")
    out = torch.full((3, heads * head_dim), float("nan"), device="cuda").to(dtype)
    scratch_o = torch.full((3 * heads * splits * head_dim,), float("nan"), device="cuda")
    scratch_ml = torch.full((3 * heads * splits * 2 + 1,), float("nan"), device="cuda")[1:]      # (rows of 4 bytes' alignment)
    run = lambda **more: k.attention_decode(q, setup["k_cache"], setup["v_cache"], setup["table"], ctx, out, heads, kv_heads, head_dim, block,
                                            scale, 0, splits, scratch_o, scratch_ml, **more)
    run()
    want = attention_reference(setup, dtype, heads, kv_heads, scale)
    close(out, want.view(3, -1), dtype)
    if 24 * splits * (head_dim + 2) <= 9 << 17:                                     # (what the entry without scratch of the caller's holds)
        other, p = torch.full_like(out, float("nan")), lambda tensor: ctypes.c_void_p(tensor.data_ptr())
        assert k.lib.skv_attention_decode_no_alloc(p(q), p(setup["k_cache"]), p(setup["v_cache"]), p(setup["table"]), setup["table"].shape[1],
                                                   p(ctx), p(other), 3, heads, kv_heads, head_dim, block, ctypes.c_float(scale), 0, splits,
                                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert torch.equal(out, other)
    sink, gate = torch.randn(heads, device="cuda"), torch.randn(3, heads, device="cuda")
    run(sink=sink, gate=gate, gate_stride=heads)
    scores = [scale * torch.einsum("hd,khd->hk", setup["q"][s].double().cpu(), setup["keys"][s].to(dtype).double().repeat_interleave(heads // kv_heads, 1))
              for s in range(3)]
    kept = torch.stack([1 / (1 + (sink.double().cpu() - torch.logsumexp(x, -1)).exp()) for x in scores])
    close(out, (want.double().cpu() * (kept * torch.sigmoid(gate.double().cpu()))[..., None]).float().to(want.device).view(3, -1), dtype)
