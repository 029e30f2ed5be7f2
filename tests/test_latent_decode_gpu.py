"""The tensor-core forms of the per-head projection and of attention over one cached row for all heads, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def lib():
    from stratakv_b200.ops import kernels_for
    return kernels_for(torch.bfloat16, 64, verbose=False)


# inner sizes of one load, part of a step, several steps; outputs that end inside a tile of 8 and inside a warp's tiles; token
# counts at the edges of 16 and where the wide form takes over; odd distances between heads, padded rows
@pytest.mark.parametrize("heads,in_dim,out_dim", [(1, 8, 5), (3, 40, 16), (5, 64, 65), (4, 256, 64), (2, 72, 256), (2, 20, 24)])
@pytest.mark.parametrize("n", [1, 16, 17, 64, 65, 200])
@pytest.mark.parametrize("x_float,out_float", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("layout", ["tight", "padded", "apart"])
def test_headwise_projection(heads, in_dim, out_dim, n, x_float, out_float, layout):
    k = lib()
    x = torch.randn(n, heads * in_dim + 8, device="cuda").to(torch.float32 if x_float else torch.bfloat16)
    w = (torch.randn(heads, out_dim, in_dim, device="cuda") / math.sqrt(in_dim)).bfloat16()
    stride = out_dim + 3 if layout == "apart" else out_dim
    width = (heads - 1) * stride + out_dim + (5 if layout == "padded" else 0)
    out = torch.full((n, width), 7.0, device="cuda", dtype=torch.float32 if out_float else torch.bfloat16)
    k.headwise_linear(x[:, :heads * in_dim], w, out, heads, zero_pad=layout == "padded", out_head_stride=stride if layout == "apart" else 0)
    ref = torch.einsum("thi,hoi->tho", x[:, :heads * in_dim].double().view(n, heads, in_dim), w.double())
    bound = torch.einsum("thi,hoi->tho", x[:, :heads * in_dim].double().abs().view(n, heads, in_dim), w.double().abs())
    for h in range(heads):
        got = out[:, h * stride:h * stride + out_dim].double()
        # float sums of exact products: a few 2^-24 of the magnitudes' sum (a float input rounded to bfloat16 would be off by 2^-9)
        assert ((got - ref[:, h]).abs() <= 5e-7 * bound[:, h] + 1e-9 + (0 if out_float else 2.0 ** -8) * ref[:, h].abs()).all()
        if layout == "apart" and h + 1 < heads:
            assert (out[:, h * stride + out_dim:(h + 1) * stride] == 7.0).all()
    if layout == "padded":
        assert (out[:, heads * out_dim:] == 0).all()


def test_headwise_projection_keeps_an_infinity():
    k = lib()
    x, w = torch.ones(2, 64, device="cuda"), torch.ones(1, 8, 64, device="cuda").bfloat16()
    x[1, 3] = float("inf")
    out = torch.empty(2, 8, device="cuda")
    k.headwise_linear(x, w, out, 1)
    assert (out[0] == 64).all() and torch.isinf(out[1]).all()


# rows with and without a part that is no value, one and several groups of 32 heads (the last not full), contexts that end at a
# tile's and a part's edge, blocks smaller than a tile, more parts than tiles
@pytest.mark.parametrize("heads,dim,vdim", [(32, 272, 256), (24, 288, 256), (3, 48, 32), (40, 320, 208), (16, 64, 64)])
@pytest.mark.parametrize("lengths", [(1,), (63, 64, 65), (128, 129, 700), (2000, 3)])
@pytest.mark.parametrize("block,splits", [(16, 2), (64, 7), (64, 40)])
def test_attention_over_one_cached_row(heads, dim, vdim, lengths, block, splits):
    k = lib()
    n, width = len(lengths), -(-max(lengths) // block)
    q = torch.randn(n, heads * dim, device="cuda").bfloat16()
    cache = torch.full((n * width + 1, 1, block, dim), float("nan"), device="cuda").bfloat16()
    table = torch.randperm(n * width, device="cuda").int().view(n, width)
    kept = []
    for i, length in enumerate(lengths):                    # (what lies beyond a sequence's end is not a number)
        rows = torch.randn(length, dim, device="cuda").bfloat16()
        kept.append(rows)
        for j in range(0, length, block):
            cache[table[i, j // block].long(), 0, :len(rows[j:j + block])] = rows[j:j + block]
    positions = torch.tensor([length - 1 for length in lengths], dtype=torch.int32, device="cuda")
    seqs = torch.arange(n, dtype=torch.int32, device="cuda")
    gate, sink = torch.randn(n, heads + 3, device="cuda"), torch.randn(heads, device="cuda")
    out = torch.full((n, heads * vdim), float("nan"), device="cuda").bfloat16()
    scratch_o, scratch_ml = (torch.full((n * heads * splits * size,), float("nan"), device="cuda") for size in (vdim, 2))
    k.attention_general(q, cache, cache, table, positions, seqs, out, heads, 1, dim, vdim, block, dim ** -0.5, gate=gate, gate_stride=heads + 3,
                        sink=sink, value_stride=dim, splits=splits, scratch_o=scratch_o, scratch_ml=scratch_ml)
    for i, rows in enumerate(kept):
        scores = q[i].double().view(heads, dim) @ rows.double().T * dim ** -0.5
        whole = torch.softmax(torch.cat([scores, sink.double()[:, None]], dim=1), dim=1)[:, :-1]
        ref = whole @ rows.double()[:, :vdim] * torch.sigmoid(gate[i, :heads].double())[:, None]
        # float throughout (a probability rounded to bfloat16 would show as 1e-3 in the partial sums), then one rounding
        assert ((out[i].double().view(heads, vdim) - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-5).all()
        merged = scratch_o.view(n, heads, splits, vdim)[i].double()
        ml = scratch_ml.view(n, heads, splits, 2)[i].double()
        live = ml[..., 0] > -math.inf
        weight = torch.where(live, torch.exp(ml[..., 0] - ml[..., 0].max(dim=1, keepdim=True).values), 0.0)
        total = (weight[..., None] * torch.where(live[..., None], merged, 0.0)).sum(1) / (weight * torch.where(live, ml[..., 1], 0.0)).sum(1)[:, None]
        assert (total - torch.softmax(scores, dim=1) @ rows.double()[:, :vdim]).abs().max() <= 1e-5


# every size in quads, tokens few (a token's queries in slices) and many, and sizes that are not
@pytest.mark.parametrize("heads,dim,rope,latent,rotated", [(32, 96, 32, 256, 32), (2, 8, 12, 1028, 8), (9, 4, 8, 4, 0), (4, 48, 16, 64, 12), (3, 5, 6, 10, 4)])
@pytest.mark.parametrize("n", [1, 7, 320])
@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_latent_finish(heads, dim, rope, latent, rotated, n, whole, dtype):
    from stratakv_b200.ops import kernels_for
    k, q_head, block_size = kernels_for(dtype, 64, verbose=False), dim + rope, 16
    at = -(-heads * q_head // 4) * 4
    fused = torch.randn(n, -(-(at + latent + rope) // 4) * 4 + 4, device="cuda")
    positions = (torch.arange(n, device="cuda") * 7 % 48).int()
    table = torch.randperm(n * 3, device="cuda").int().view(n, 3)
    rotation = torch.randn(48, rotated // 2, 2, device="cuda") if rotated else None
    gamma = torch.rand(latent, device="cuda") + 0.5
    nan = lambda *shape: torch.full(shape, float("nan"), device="cuda").to(dtype)
    plain, folded, together, cache = nan(n, heads * dim), nan(n, heads * (latent + rope)), nan(n, heads * q_head), nan(n * 3, 1, block_size, latent + rope)
    for write in (True, False):
        k.latent_finish(fused, None if whole else plain, None if whole else folded, cache, positions, torch.arange(n, device="cuda").int(), table, heads, dim,
                        rope, latent, block_size, rotation, rotated, at, gamma, 1e-5, write, q_whole=together if whole else None)
        kept = cache.clone() if write else kept

    def turn(x):
        if not rotated:
            return x
        c, s = rotation.double()[positions.long()].unbind(-1)
        while c.dim() < x.dim():
            c, s = c[:, None], s[:, None]
        u, v = x[..., :rotated // 2], x[..., rotated // 2:rotated]
        return torch.cat([u * c - v * s, v * c + u * s, x[..., rotated:]], -1)

    rows = fused.double()
    queries = rows[:, :heads * q_head].view(n, heads, q_head)
    queries = torch.cat([queries[..., :dim], turn(queries[..., dim:])], -1)
    vector = rows[:, at:at + latent]
    vector = vector * torch.rsqrt((vector * vector).mean(-1, keepdim=True) + 1e-5) * gamma.double()
    want = torch.cat([vector, turn(rows[:, at + latent:at + latent + rope])], -1)
    error = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-6                 # one rounding, or a few of float
    near = lambda got, ref: ((got.double() - ref).abs() <= error * ref.abs() + 4e-6).all()
    if whole:
        assert near(together.view(n, heads, q_head), queries)
    else:
        assert near(plain.view(n, heads, dim), queries[..., :dim])
        assert near(folded.view(n, heads, -1)[..., latent:], queries[..., dim:]) and torch.isnan(folded.view(n, heads, -1)[..., :latent]).all()
    blocks = table[torch.arange(n, device="cuda"), (positions // block_size).long()].long()
    assert near(cache[blocks, 0, (positions % block_size).long()], want)
    assert int((~torch.isnan(cache)).sum()) == n * (latent + rope) and torch.equal(cache.nan_to_num(), kept.nan_to_num())


def test_attention_over_one_cached_row_whose_scores_begin_at_minus_infinity():
    """The first tile of the second part: its rows take no share."""
    heads, dim, vdim, block, n = 4, 48, 32, 64, 256
    cache, q = torch.randn(4, 1, block, dim, device="cuda").bfloat16(), (torch.rand(1, heads * dim, device="cuda") + 0.1).bfloat16()
    cache[2, :, :, vdim:] = -math.inf
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    out, scratch_o, scratch_ml = torch.empty(1, heads * vdim, device="cuda").bfloat16(), torch.empty(heads * 2 * vdim, device="cuda"), torch.empty(heads * 4, device="cuda")
    lib().attention_general(q, cache, cache, i32([list(range(4))]), i32([n - 1]), i32([0]), out, heads, 1, dim, vdim, block, dim ** -0.5,
                            value_stride=dim, splits=2, scratch_o=scratch_o, scratch_ml=scratch_ml)
    rows = cache.view(n, dim).double()
    scores = q.double().view(heads, dim) @ rows.T * dim ** -0.5
    assert (scores[:, 128:192] == -math.inf).all()
    want = torch.softmax(scores, -1) @ rows[:, :vdim]
    assert ((out.double().view(heads, vdim) - want).abs() <= 2.0 ** -8 * want.abs() + 2e-5).all()
