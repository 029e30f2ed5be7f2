"""Prompt attention on tensor cores where the blocks of a cluster share a query tile's keys (few query tiles over long contexts), against
float64: pieces without keys beside long ones, windows, and the optional terms, whose merge is another."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# (new tokens, context after) of the sequences: clusters of two and of four, contexts shorter than the pieces are many; windows that end inside tiles,
# of two pieces and of four (whole pieces that a row does not see)
@pytest.mark.parametrize("sequences", [[(100, 3100)], [(40, 1100), (33, 33)], [(200, 5000), (130, 130), (1, 64)]])
@pytest.mark.parametrize("heads,kv_heads,dim", [(2, 1, 64), (20, 4, 64), (2, 2, 128), (20, 4, 128)])
@pytest.mark.parametrize("extras", ["plain", "window 1001", "window 2101", "sink cap gate", "bias gate per number"])
def test_keys_shared_by_a_cluster(sequences, heads, kv_heads, dim, extras):
    from stratakv_b200.ops import kernels_for
    k, block = kernels_for(torch.bfloat16, dim, verbose=False), 64
    g = torch.Generator(device="cuda").manual_seed(7)
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    width = -(-max(c for _, c in sequences) // block)
    n, blocks = sum(q for q, _ in sequences), len(sequences) * width
    keys, values = (normal(blocks, kv_heads, block, dim).bfloat16() for _ in "kv")
    table = torch.randperm(blocks, generator=g, device="cuda").int().view(len(sequences), width)
    cu_q = torch.tensor([0] + [sum(q for q, _ in sequences[:i + 1]) for i in range(len(sequences))], dtype=torch.int32, device="cuda")
    after = torch.tensor([c for _, c in sequences], dtype=torch.int32, device="cuda")
    q, out = normal(n, heads * dim).bfloat16(), torch.full((n, heads * dim), float("nan"), device="cuda").bfloat16()
    scale, window = 1.3 / math.sqrt(dim), int(extras.split()[1]) if extras.startswith("window") else 0
    tiles = len(sequences) * -(-max(t for t, _ in sequences) // 128)
    splits = k.lib.skv_attention_prefill_tc_splits(tiles, heads, width, block, window, torch.cuda.get_device_properties(0).multi_processor_count)
    assert splits > 1 and (splits == 4 or tiles * heads > 74 or min(width * block, window + 128 if window else math.inf) < 2048)
    more, sink, gate, bias, cap = {}, None, None, None, 0.0
    if extras == "sink cap gate":
        sink, gate, cap = normal(heads), normal(n, heads), 20.0
        more = dict(sink=sink, gate=gate, gate_stride=heads, softcap=cap)
    elif extras == "bias gate per number":
        gate, bias = normal(n, heads * dim), normal(heads, 1).abs() * torch.log1p(0.3 * torch.arange(5000, device="cuda"))
        more = dict(gate=gate, gate_stride=heads * dim, gate_per_element=True, bias=(bias * math.log2(math.e)).contiguous())
    k.attention_prefill_tc(q, keys, values, table, cu_q, after, out, max(t for t, _ in sequences), heads, kv_heads, dim, block, scale, window, **more)
    for s, (new, ctx) in enumerate(sequences):
        rows = slice(int(cu_q[s]), int(cu_q[s + 1]))
        dense = lambda cache: cache[table[s].long()].transpose(1, 2).reshape(-1, kv_heads, dim)[:ctx].double().repeat_interleave(heads // kv_heads, 1)
        scores = scale * torch.einsum("qhd,khd->hqk", q[rows].double().view(new, heads, dim), dense(keys))
        distance = torch.arange(ctx - new, ctx, device="cuda")[:, None] - torch.arange(ctx, device="cuda")
        if cap:
            scores = cap * torch.tanh(scores / cap)
        if bias is not None:
            scores = scores - bias.double()[:, distance.clamp(min=0)]
        scores = scores.masked_fill((distance < 0) | (distance >= (window or ctx)), -math.inf)
        if sink is not None:
            scores = torch.cat([scores, sink.double()[:, None, None].expand(heads, new, 1)], -1)
        shares = torch.softmax(scores, -1)[..., :ctx]
        want, size = (torch.einsum("hqk,khd->qhd", shares, v) for v in (dense(values), dense(values).abs()))
        if gate is not None:
            opened = torch.sigmoid(gate[rows].double()).view(new, heads, -1)
            want, size = want * opened, size * opened
        # every probability is rounded to bfloat16 once (by up to 2^-8 of it), and so is the result; scores err by float sums of order one
        assert ((out[rows].double().view_as(want) - want).abs() <= 2.0 ** -8 * (want.abs() + size) * 1.01 + 1e-5).all()
    assert int(k.error_flag) == 0


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("fault", ["key", "query with a sink", "value beyond reach"])
def test_what_is_not_finite_is_not_lost_in_a_merge(dim, fault):
    """Four pieces a query tile.  A NaN key is the only one that its own row sees of its piece (the pieces of the first two tiles are
    single tiles of 64 keys); a NaN query makes all pieces' scores NaN; a value of infinity is reached with weights that vanish."""
    from stratakv_b200.ops import kernels_for
    k, block, n, heads, kv_heads = kernels_for(torch.bfloat16, dim, verbose=False), 64, 2100, 2, 1
    blocks = -(-n // block)
    g = torch.Generator(device="cuda").manual_seed(9)
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda").bfloat16()
    keys, values, q = normal(blocks, kv_heads, block, dim), normal(blocks, kv_heads, block, dim), normal(n, heads * dim)
    table = torch.arange(blocks, dtype=torch.int32, device="cuda")[None]
    cu_q, after = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, n], [n]))
    sink = None
    if fault == "key":
        first = 192
        keys[first // block, 0, first % block] = math.nan
        bad = slice(first, n)
    elif fault == "query with a sink":
        first, sink = 300, torch.zeros(heads, device="cuda")
        q[first] = math.nan
        bad = slice(first, first + 1)
    else:
        first = 0                                            # (0 x infinity spoils the rows ahead of it in its tile as well)
        q.fill_(1.0)
        keys.fill_(1.0)
        keys[0].fill_(-1.0)                                  # the first piece's weights are 2^-180 and less beyond its own tile
        values[0, 0, first] = math.inf
        bad = slice(first, n)
    out = torch.zeros(n, heads * dim, device="cuda").bfloat16()
    k.attention_prefill_tc(q, keys, values, table, cu_q, after, out, n, heads, kv_heads, dim, block, 1.0, sink=sink)
    wrong = torch.ones(n, dtype=torch.bool, device="cuda")
    wrong[bad] = False
    assert not out[bad].isfinite().all(-1).any() and out[wrong].isfinite().all()
