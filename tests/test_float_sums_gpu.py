"""Float sums that tensor cores make err no more than the chain of float multiply-adds that they stand for."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def lib():
    from stratakv_b200.ops import kernels_for
    return kernels_for(torch.bfloat16, 64, verbose=False)


def chain(x, w):
    """[..., m, k] and [..., n, k] -> [..., m, n] in float32, one multiply-add after the other."""
    total = torch.zeros(*x.shape[:-1], w.shape[-2], device=x.device)
    for k in range(x.shape[-1]):
        total = (total.double() + x[..., :, None, k].double() * w[..., None, :, k].double()).float()
    return total


def error(got, want):
    return float((got.double() - want).norm() / want.norm())


# (a sum of one sign is what drifts where it is cut off instead of rounded)
@pytest.mark.parametrize("heads,in_dim,out_dim", [(32, 64, 64), (8, 256, 64), (2, 512, 96), (3, 2048, 40)])
@pytest.mark.parametrize("n", [8, 100])
@pytest.mark.parametrize("x_float", [False, True])
@pytest.mark.parametrize("one_sign", [False, True])
def test_headwise_projection(heads, in_dim, out_dim, n, x_float, one_sign):
    x, w = torch.randn(n, heads * in_dim, device="cuda"), (torch.randn(heads, out_dim, in_dim, device="cuda") / math.sqrt(in_dim)).bfloat16()
    x = x if x_float else x.bfloat16()
    if one_sign:
        x, w = x.abs(), w.abs()
    out = torch.empty(n, heads * out_dim, device="cuda")
    lib().headwise_linear(x, w, out, heads)
    by_head = x.view(n, heads, in_dim).transpose(0, 1)
    want = by_head.double() @ w.double().transpose(1, 2)
    assert error(out.view(n, heads, out_dim).transpose(0, 1), want) <= error(chain(by_head, w), want)


def test_headwise_projection_of_the_largest_floats():
    """Beyond the largest bfloat16, short of the largest float: rounded to nearest, the first of its three parts was infinite."""
    x, w = torch.ones(2, 64, device="cuda"), torch.ones(1, 8, 64, device="cuda").bfloat16()
    x[1, 3], x[0, 5] = 3.4e38, -3.4e38
    out = torch.empty(2, 8, device="cuda")
    lib().headwise_linear(x, w, out, 1)
    assert torch.equal(out, x.sum(-1, keepdim=True).expand(2, 8))


# scores of rows that differ, and (queries of zero) means of values of one sign, whose sums are the longest
@pytest.mark.parametrize("heads,dim,vdim,length,splits", [(32, 272, 256, 780, 2), (32, 288, 256, 8000, 2), (20, 320, 64, 3000, 3)])
@pytest.mark.parametrize("means", [False, True])
def test_attention_over_one_cached_row(heads, dim, vdim, length, splits, means):
    """The parts before the merge (the merged output is rounded to bfloat16)."""
    block, n = 64, 2
    width = -(-length // block)
    q = torch.randn(n, heads * dim, device="cuda").bfloat16() * (0 if means else 1)
    cache = torch.randn(n * width, 1, block, dim, device="cuda").bfloat16()
    cache = cache.abs() if means else cache
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    out = torch.empty(n, heads * vdim, device="cuda").bfloat16()
    scratch_o, scratch_ml = (torch.empty(n * heads * splits * size, device="cuda") for size in (vdim, 2))
    lib().attention_general(q, cache, cache, torch.arange(n * width, device="cuda").int().view(n, width), i32([length - 1] * n), i32(range(n)), out,
                            heads, 1, dim, vdim, block, dim ** -0.5, value_stride=dim, splits=splits, scratch_o=scratch_o, scratch_ml=scratch_ml)
    rows = cache.view(n, width * block, dim)[:, :length]
    parts, (top, total) = scratch_o.view(n, heads, splits, vdim).double(), scratch_ml.view(n, heads, splits, 2).double().unbind(-1)
    weight = torch.exp(top - top.amax(-1, keepdim=True))
    got = (weight[..., None] * parts).sum(2) / (weight * total).sum(-1, keepdim=True)
    scores = q.double().view(n, heads, dim) @ rows.double().transpose(1, 2) * dim ** -0.5
    want = torch.softmax(scores, -1) @ rows.double()[..., :vdim]
    # the same in float32, one multiply-add after the other in each part
    tiles = -(-length // 64)
    each = -(-tiles // splits) * 64
    mine = chain(q.view(n, heads, dim), rows) * torch.tensor(dim ** -0.5, device="cuda")
    p = torch.exp(mine - mine.amax(-1, keepdim=True))
    plain = sum(chain(p[..., i:i + each], rows[:, i:i + each, :vdim].transpose(1, 2)).double() for i in range(0, length, each))
    plain = plain / sum(chain(p[..., i:i + each], torch.ones(n, 1, min(each, length - i), device="cuda")).double() for i in range(0, length, each))
    assert error(got, want) <= error(plain, want)


def warp_sum(x, w):
    """``chain`` as a warp makes it: a lane takes four neighbouring numbers of every 128, then the lanes are added in pairs."""
    lanes = lambda z: z.view(*z.shape[:-1], -1, 32, 4).transpose(-3, -2).flatten(-2).transpose(-3, -2)
    parts = torch.stack([chain(a, b) for a, b in zip(lanes(x).unbind(-3), lanes(w).unbind(-3))])
    while len(parts) > 1:
        parts = parts[:len(parts) // 2] + parts[len(parts) // 2:]
    return parts[0]


# few tokens (a cluster of 16 tokens) and many (of 32)
@pytest.mark.parametrize("dim,hidden", [(64, 2048), (32, 4096)])
@pytest.mark.parametrize("n", [8, 300])
def test_token_input(dim, hidden, n):
    x, ids = 3 * torch.randn(n, hidden, device="cuda"), torch.randint(0, 50, (n,), device="cuda").int()
    table, gate = torch.randn(50, dim, device="cuda").bfloat16(), (torch.randn(dim, hidden, device="cuda") / math.sqrt(hidden)).bfloat16()
    proj, norm = torch.randn(dim, hidden, device="cuda").bfloat16(), 1 + 0.1 * torch.randn(hidden, device="cuda")
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")
    unit = lambda y: y * torch.rsqrt((y * y).mean(-1, keepdim=True) + 1e-5)
    want = unit((gelu(x.double() @ gate.double().T) * table[ids.long()].double()) @ proj.double()) * norm.double()
    plain = x + unit(chain(gelu(warp_sum(x, gate.float())) * table[ids.long()].float(), proj.T)) * norm
    got = x.clone()
    lib().token_side(got, ids, table, 0, dim, gate, proj, norm, 1e-5)
    before = x.double()
    assert error(got.double() - before, want) <= error(plain.double() - before, want)


# nine to sixteen tokens, weights on both sides of 48 MB
@pytest.mark.parametrize("M,N,K", [(9, 32000, 2048), (16, 6144, 4096), (12, 4096, 4096)])
def test_projection_of_up_to_sixteen_tokens(M, N, K):
    from stratakv_b200 import ops
    a, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
    out, want = torch.empty(M, N, device="cuda"), a.double() @ w.double().T
    lib().linear(a, w, out, ops.MODE_STORE_F32)
    assert error(out, want) <= error(chain(a, w), want)


@pytest.mark.parametrize("rank,channels", [(64, 2048), (256, 512), (480, 512)])
@pytest.mark.parametrize("n", [4, 100])
def test_decay_per_channel(rank, channels, n):
    lora, w2, w0 = torch.randn(n, rank, device="cuda"), (torch.randn(rank, channels, device="cuda") / math.sqrt(rank)).bfloat16(), torch.randn(channels, device="cuda") - 2
    out = torch.empty(n, channels, device="cuda")
    lib().time_mix_decay(lora, rank, w2, w0, out)
    want = torch.exp(-torch.exp(torch.tanh(lora.double()) @ w2.double() + w0.double()))
    plain = torch.exp(-torch.exp(chain(torch.tanh(lora), w2.T) + w0))
    assert error(out, want) <= error(plain, want)


# (a softmax of large scores: the error of a sum is the relative error of its weight)
@pytest.mark.parametrize("experts,hidden", [(8, 2048), (64, 4096)])
def test_router(experts, hidden, n=2000):
    h, w = torch.randn(n, hidden, device="cuda").bfloat16(), (8 * torch.randn(experts, hidden, device="cuda") / math.sqrt(hidden)).bfloat16()
    chosen, weights = torch.empty(n, 4, dtype=torch.int32, device="cuda"), torch.empty(n, 4, device="cuda")
    lib().route_tokens(h, w, None, 4, 1.0, False, chosen, weights, softmax=True)
    want = torch.softmax(h.double() @ w.double().T, -1).gather(1, chosen.long())
    plain = torch.softmax(warp_sum(h.float(), w.float()).double(), -1).gather(1, chosen.long())
    # (besides the sums' errors the kernel's weights have those of an exponential, a sum and a division: four units of 2^-24)
    assert error(weights / want, torch.ones_like(want)) <= math.hypot(error(plain / want, torch.ones_like(want)), 4 * 2.0 ** -24)


# sequences of several chunks: what the state gives and what the chunk's own tokens give are sums of their own
@pytest.mark.parametrize("heads,dim", [(8, 64), (4, 128)])
def test_retention_of_prompts(heads, dim):
    """Against the recurrence in float32, a multiply-add a product."""
    from stratakv_b200.ops import kernels_for
    k, length = kernels_for(torch.float32, 64, verbose=False), 500
    fused = torch.randn(length, 4 * heads * dim, device="cuda")
    decay = 1 - 2.0 ** -(5.0 + torch.arange(heads, device="cuda") % 4)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    state, out = torch.zeros(1, 2 * heads * dim * dim, device="cuda"), torch.empty(length, heads * dim, device="cuda")
    scratch = torch.empty(k.retention_scratch(1, length, heads, dim, dim), device="cuda")
    k.retention(fused.clone(), None, 0, decay, 1e-5, out, state, (i32(range(length)), i32([0] * length), i32([0, length]), i32([0])), heads, dim, dim,
                length, scratch)
    q, key, v, gate = fused.double().view(length, 4, heads, dim).unbind(1)

    def run(round_it):
        S, rows, scaled = torch.zeros(heads, dim, dim, device="cuda").double(), [], round_it(key * dim ** -0.5)
        for t in range(length):
            S = round_it(decay.double()[:, None, None] * S + round_it(scaled[t, :, :, None] * v[t, :, None, :]))
            o = torch.zeros(heads, dim, device="cuda").double()
            for d in range(dim):
                o = round_it(o + q[t, :, d, None] * S[:, d])
            rows.append(o)
        o = torch.stack(rows)
        return o * torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-5) * torch.nn.functional.silu(gate)

    want = run(lambda z: z)
    assert error(out.view(length, heads, dim), want) <= error(run(lambda z: z.float().double()), want)
