"""The 32-bit projection and attention kernels against float64, at the sizes where a tile, a part of K or a part of the
keys ends."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def lib(head_dim=64):
    from stratakv_b200.ops import kernels_for
    return kernels_for(torch.float32, head_dim, verbose=False)


def at_offset(tensor, offset):
    """The same numbers ``offset`` floats into a larger buffer (no multiple of 16 bytes)."""
    flat = torch.empty(tensor.numel() + offset, device="cuda")
    view = flat[offset:].view(tensor.shape)
    view.copy_(tensor)
    return view


# few tokens: 1, 2, 4, 8, 16 a block, K in two or four parts, rows beyond the last group of 16; K no multiple of 4 and
# operands off 16 bytes take single loads.  More: tiles of 32, 64 and 128 rows, alone and with K shared by 2, 4, 8 blocks.
@pytest.mark.parametrize("M,N,K,offset", [
    (1, 16, 4, 0), (1, 2560, 2048, 0), (2, 40, 7, 0), (3, 11264, 2048, 0), (3, 2048, 5632, 0), (4, 33, 260, 0), (5, 48, 129, 0),
    (8, 12000, 512, 0), (9, 64, 1030, 0), (16, 2048, 516, 0), (16, 48, 512, 1), (17, 2048, 2048, 0), (17, 16, 3, 0), (32, 208, 1000, 0),
    (33, 144, 4100, 0), (64, 130, 4099, 0), (64, 2048, 2048, 3), (65, 384, 520, 0), (129, 2000, 1024, 0), (192, 256, 300, 0),
    (321, 129, 260, 0), (639, 2048, 5632, 0), (700, 160, 17, 0)])
def test_float_projection(M, N, K, offset):
    from stratakv_b200 import ops
    k = lib()
    a, w = at_offset(torch.randn(M, K, device="cuda"), offset), at_offset(torch.randn(N, K, device="cuda") / math.sqrt(K), offset)
    ref, bound = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # a sum of K products in float in any order errs by a few units of 2^-24 of the sum of their magnitudes
    allowed = 2e-6 * (bound + 1e-3)
    out = torch.full((M, N), float("nan"), device="cuda")
    k.linear(a, w, out, ops.MODE_STORE)
    assert ((out.double() - ref).abs() <= allowed).all()
    total = torch.randn(M, N, device="cuda")
    before = total.double()
    k.linear(a, w, total, ops.MODE_ADD_F32)
    assert ((total.double() - before - ref).abs() <= allowed + 2.0 ** -23 * total.double().abs()).all()
    if N % 16 == 0:
        gated = torch.full((M, N // 2), float("nan"), device="cuda")
        k.linear(a, w, gated, ops.MODE_GATED, "silu")
        gate = ref.view(M, N // 16, 2, 8)[:, :, 0].reshape(M, N // 2)
        up = ref.view(M, N // 16, 2, 8)[:, :, 1].reshape(M, N // 2)
        slack = allowed.view(M, N // 16, 2, 8).amax(dim=(2, 3)).repeat_interleave(8, dim=1)
        value = torch.nn.functional.silu(gate) * up
        assert ((gated.double() - value).abs() <= slack * (1.2 * up.abs() + gate.abs() + 1) + 1e-6 * value.abs()).all()


# eight, four and one warp a (token, head); contexts that end at a chunk's and a part's edge; a window
@pytest.mark.parametrize("lengths,heads,kv_heads", [((1,), 4, 2), ((31, 32, 33), 8, 2), ((255, 256, 257, 600), 8, 8), ((300,) * 40, 32, 4),
                                                    ((70,) * 200, 32, 4)])
@pytest.mark.parametrize("window", [0, 40])
def test_float_attention_over_parts_of_the_keys(lengths, heads, kv_heads, window):
    d, block = 64, 16
    k = lib(d)
    width = -(-max(lengths) // block)
    table = torch.randperm(len(lengths) * width, device="cuda").to(torch.int32).view(len(lengths), width)
    keys, values = (torch.randn(len(lengths) * width, kv_heads, block, d, device="cuda") for _ in range(2))
    q = torch.randn(len(lengths), heads, d, device="cuda") * 2
    positions = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device="cuda")
    seqs = torch.arange(len(lengths), dtype=torch.int32, device="cuda")
    out = torch.full_like(q, float("nan"))
    k.attention(q, keys, values, table, positions, seqs, out, heads, kv_heads, d, block, d ** -0.5, window)
    for i, n in list(enumerate(lengths))[:: max(1, len(lengths) // 5)]:
        gather = lambda cache: cache[table[i].long()].permute(1, 0, 2, 3).reshape(kv_heads, -1, d)[:, max(0, n - window) if window else 0:n].double()
        K, V = (gather(c).repeat_interleave(heads // kv_heads, dim=0) for c in (keys, values))
        scores = torch.einsum("hd,hjd->hj", q[i].double(), K) * d ** -0.5
        ref = torch.einsum("hj,hjd->hd", torch.softmax(scores, dim=-1), V)
        # scores of up to about 10 carry 64 roundings of 2^-24 each, which the softmax turns into relative errors
        assert (out[i].double() - ref).abs().max() <= 2e-5


def test_float_attention_over_a_part_that_weighs_nothing():
    """Keys whose scores are all -infinity, a whole part of them: they take no share, as in a walk over all keys in turn."""
    d, block, n, heads = 64, 16, 300, 4
    keys, values = (torch.randn(19, 1, block, d, device="cuda") for _ in range(2))
    keys[4:6] = -math.inf                                                  # keys 64 to 95: the third part's first
    q, i32 = torch.rand(1, heads, d, device="cuda") + 0.1, lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    out = torch.full_like(q, float("nan"))
    lib(d).attention(q, keys, values, i32([list(range(19))]), i32([n - 1]), i32([0]), out, heads, 1, d, block, d ** -0.5, 0)
    scores = q[0].double() @ keys.view(-1, d)[:n].double().T * d ** -0.5
    assert (scores[:, 64:96] == -math.inf).all()
    assert (out[0].double() - torch.softmax(scores, -1) @ values.view(-1, d)[:n].double()).abs().max() <= 2e-5
