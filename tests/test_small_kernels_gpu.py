"""Row kernels in their wide forms against float64: the norm of few rows, the embedding, the per-channel
decay on tensor cores."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def lib(dtype=torch.bfloat16):
    from stratakv_b200.ops import kernels_for
    return kernels_for(dtype, 64, verbose=False)


# widths of one quad, of part of a block, of several quads a thread, of all a block holds and one beyond; rows below and above the
# count where a warp takes a row; parts of a row; chosen rows; a width that is no multiple of 4
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width,groups", [(4, 1), (130, 1), (500, 2), (2048, 1), (3076, 1), (4096, 2), (8192, 1), (8196, 1)])
@pytest.mark.parametrize("n,chosen", [(1, False), (7, True), (1030, False)])
def test_rmsnorm_forms(dtype, width, groups, n, chosen):
    k = lib(dtype)
    x, gamma = 3 * torch.randn(n, width, device="cuda"), 1 + 0.1 * torch.randn(width, device="cuda")
    rows = torch.randint(0, n, (2 * n,), device="cuda").int() if chosen else None
    out = torch.full((2 * n if chosen else n, width), float("nan"), device="cuda").to(dtype)
    k.rmsnorm(x, gamma, 1e-5, out, rows, groups=groups)
    source = x.double()[rows.long()] if chosen else x.double()
    parts = source.view(len(out), groups, -1)
    ref = (parts * torch.rsqrt((parts * parts).mean(-1, keepdim=True) + 1e-5)).view(len(out), width) * gamma.double()
    assert ((out.double() - ref).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2e-6) * ref.abs() + 1e-6).all()


@pytest.mark.parametrize("hidden", [4, 260, 2048, 2052, 8192, 30])
def test_embedding_with_a_folded_norm(hidden):
    from types import SimpleNamespace
    from stratakv_b200.residual import ResidualStats
    k = lib()
    ids = torch.tensor([3, 0, 12, 99, -1], dtype=torch.int32, device="cuda")
    table, gamma = torch.randn(13, hidden, device="cuda").bfloat16(), 1 + 0.1 * torch.randn(hidden, device="cuda")
    nan = lambda *shape: torch.full(shape, float("nan"), device="cuda")
    stats = ResidualStats(nan(5, hidden).bfloat16(), nan(5), nan(5, -(-hidden // 16) + 4), torch.zeros(1, device="cuda", dtype=torch.int32))
    stats.expect(SimpleNamespace(gamma=gamma, spec=SimpleNamespace(eps=1e-5)))
    out, flag = nan(5, hidden), torch.zeros(1, dtype=torch.int32, device="cuda")
    k.embed(table, ids, out, flag, stats=stats)
    ref = torch.cat([table[ids[:3].long()].float(), torch.zeros(2, hidden, device="cuda")])
    assert torch.equal(out, ref) and int(flag) == 1
    assert torch.equal(stats.scaled, (ref * gamma).bfloat16())
    torch.testing.assert_close(stats.partials[:, :1].double().sum(-1), (ref.double() ** 2).sum(-1), rtol=1e-5, atol=1e-9)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 40])
@pytest.mark.parametrize("rank,channels", [(16, 64), (64, 576), (128, 2048), (24, 64), (64, 100)])
def test_decay_per_channel(n, rank, channels):
    k = lib()
    lora, w2t, w0 = torch.randn(n, rank + 8, device="cuda"), (torch.randn(rank, channels, device="cuda") / math.sqrt(rank)).bfloat16(), torch.randn(channels, device="cuda") - 2
    out = torch.full((n, channels), float("nan"), device="cuda")
    k.time_mix_decay(lora, rank, w2t, w0, out)
    z = torch.tanh(lora[:, :rank].double()) @ w2t.double() + w0.double()
    # float throughout: exp(-exp(z)) has a slope of at most 0.37 in z, whose sum errs by a few 2^-24 of its terms
    assert (out.double() - torch.exp(-torch.exp(z))).abs().max() <= 1.5e-6


# widths of one quad, of a block's first round and beyond it, and no multiple of 4
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hidden", [4, 516, 2052, 4096, 30])
@pytest.mark.parametrize("pairs,places", [(True, True), (True, False), (False, True)])
def test_embedding_sum(dtype, hidden, pairs, places):
    k = lib(dtype)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    ids, positions = i32([3, 0, 12, 5, 13, 7]), i32([0, 1, 2, 9, 0, 20])            # three sequences; an id and a place too far
    seq, cu, slots = i32([0, 0, 0, 1, 2, 2]), i32([0, 3, 4, 6]), i32([2, 0, 1])
    table, pair, place = (torch.randn(rows, hidden, device="cuda").to(dtype) for rows in (13, 8, 15))
    last = i32([6, 4, 0, 0, 0, 0])
    out, flag = torch.full((6, hidden), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    k.embed_sum(table, ids, out, positions, seq, cu, slots, flag, pair_table=pair if pairs else None, last_ids=last if pairs else None, mul_prev=5,
                mul_cur=3, position_table=place if places else None, position_scale=0.5)
    previous = [None, 3, 0, 6, None, None]                                          # position 9 reads the entry of even places
    for t, (id, position) in enumerate(zip(ids.tolist(), positions.tolist())):
        want = table[id].float() if id < 13 else torch.zeros(hidden, device="cuda")
        if pairs and id < 13:
            before = 13 if t == 5 else previous[t]
            want = want + pair[7 if position == 0 else (before * 5 + id * 3) % 7].float()
        if places and position < 15:
            want = want + place[position].float() * 0.5
        torch.testing.assert_close(out[t], want, rtol=1e-6, atol=1e-6)
    assert int(flag) == (9 if places else 1)
    assert not pairs or last.tolist() == [6, 5, 7, 0, 12, 0]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hidden", [4, 2048, 2052, 4096, 4100, 30])
@pytest.mark.parametrize("count", [1, 2, 8])
def test_streams_of_wide_rows(dtype, hidden, count):
    k, n = lib(dtype), 5
    streams, branch = torch.randn(count, n, hidden, device="cuda"), torch.randn(n, hidden, device="cuda")
    mix, write, read = torch.randn(count, count, device="cuda") / count, torch.randn(count, device="cuda"), torch.randn(count, device="cuda")
    gamma = 1 + 0.1 * torch.randn(hidden, device="cuda")
    want = torch.einsum("st,snw->tnw", mix.double(), streams.double()) + write.double()[:, None, None] * branch.double()
    u = torch.einsum("s,snw->nw", read.double(), want)
    normed = (u * torch.rsqrt((u * u).mean(-1, keepdim=True) + 1e-5)) * gamma.double()
    out, total = torch.full((n, hidden), float("nan"), device="cuda").to(dtype), torch.full((n, hidden), float("nan"), device="cuda")
    k.stream_mix(streams, count, branch=branch, mix=mix.reshape(-1), write=write, read=read, gamma=gamma, eps=1e-5, normed_out=out, sum_out=total)
    # float sums of at most nine products of order one, twice over
    assert (streams.double() - want).abs().max() <= 2e-6 * (1 + want.abs().max())
    assert (total.double() - want.sum(0)).abs().max() <= 4e-6 * (1 + want.abs().max())
    assert ((out.double() - normed).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * normed.abs() + 1e-5 * (1 + normed.abs().max())).all()


# lengths below, at and beyond four tokens and a staged set of sixteen; a state to go on from and none; steps of few sequences (a
# head's columns in slices) and of many; a state that does not lie on 16 bytes (the form of other head sizes)
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("lengths,heads", [([1], 2), ([35], 3), ([16, 1, 4, 33, 2, 17], 2), ([5] * 40, 8)])
@pytest.mark.parametrize("offset", [0, 4, 2])
def test_time_mix_scan(dim, lengths, heads, offset):
    k = lib()
    n, inner, hidden, seqs = sum(lengths), heads * dim, 24, len(lengths)
    starts = [0 if s % 2 == 0 else 3 + s for s in range(seqs)]
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    cu = [0]
    for length in lengths:
        cu.append(cu[-1] + length)
    slots = list(range(seqs, 0, -1))
    meta = (i32([p + i for p, length in zip(starts, lengths) for i in range(length)]), i32([s for s, length in enumerate(lengths) for _ in range(length)]),
            i32(cu), i32(slots))
    rows = torch.randn(4, n, inner, device="cuda")
    r, key, value = rows[0], rows[1] / 8, rows[2]
    decay, bonus = torch.rand(n, inner, device="cuda"), torch.rand(inner, device="cuda")
    floats = k.time_mix_state_floats(hidden, heads, dim)
    state = torch.randn(seqs + 1, 4 + -(-floats // 4) * 4, device="cuda")
    before, half = state.double(), heads * dim * dim
    out, h = torch.full((n, inner), float("nan"), device="cuda"), torch.randn(n, hidden, device="cuda").bfloat16()
    k.time_mix_scan(r, key, value, decay, bonus, out, h, seqs, heads, dim, meta, state, offset)
    per_head = lambda t: t.double().view(-1, heads, dim)
    for s in range(seqs):
        p0, last = starts[s], starts[s] + lengths[s] - 1
        S = torch.zeros(heads, dim, dim, device="cuda", dtype=torch.float64)
        if p0 > 0:
            S = before[slots[s], offset + ((p0 - 1) & 1) * half:][:half].view(heads, dim, dim).clone()
        size = torch.ones_like(S)
        for t in range(cu[s], cu[s + 1]):
            rt, kt, vt, wt = (per_head(a[t])[0] for a in (r, key, value, decay))
            kv = kt[:, :, None] * vt[:, None, :]
            want = torch.einsum("hi,hij->hj", rt, S + bonus.double().view(heads, dim, 1) * kv)
            mass = torch.einsum("hi,hij->hj", rt.abs(), S.abs() + kv.abs())
            S = wt[:, :, None] * S + kv
            # float sums of dim products, each with a few roundings behind it
            assert ((per_head(out[t])[0] - want).abs() <= 1e-6 * mass + 1e-6).all()
        got = state[slots[s], offset + (last & 1) * half:][:half].double().view(heads, dim, dim)
        assert ((got - S).abs() <= 2e-6 * (1 + S.abs())).all()
        kept = state[slots[s], offset + 2 * half + (last & 1) * hidden:][:hidden]
        assert torch.equal(kept, h[cu[s + 1] - 1].float())


# segments inside a row, of one quad, of a block's first round and beyond it, of more than a block holds, and off 16 bytes
@pytest.mark.parametrize("segments", [[(4, 4, True), (8, 516, False)], [(0, 2052, False), (2052, 256, True)], [(0, 4096, True)], [(0, 4100, False), (4100, 8, False)],
                                      [(2, 256, True)], [(0, 30, False), (32, 64, True)]])
@pytest.mark.parametrize("n", [1, 9])
def test_norm_of_segments(n, segments):
    k = lib()
    rows = torch.randn(n, max(o + w for o, w, _ in segments) + 4 & ~3, device="cuda")
    want, given = rows.double(), []
    for offset, width, biased in segments:
        bias, weight = torch.randn(width, device="cuda") if biased else None, torch.randn(width, device="cuda")
        x = want[:, offset:offset + width] + (bias.double() if biased else 0.0)
        want[:, offset:offset + width] = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * weight.double()
        given.append((offset, width, bias, weight))
    k.projection_norm(rows, 1e-5, given)
    assert ((rows.double() - want).abs() <= 2e-6 * want.abs() + 1e-6).all()


def packed(lengths, starts, slots):
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    cu = [0]
    for length in lengths:
        cu.append(cu[-1] + length)
    return cu[-1], (i32([p + i for p, length in zip(starts, lengths) for i in range(length)]), i32([s for s, length in enumerate(lengths) for _ in range(length)]),
                    i32(cu), i32(slots))


STEPS = [([1, 1, 1], [0, 2, 9]), ([5, 1, 2, 70], [0, 1, 3, 0]), ([700, 3, 600, 1, 2], [0, 0, 5, 2, 1])]      # the last: eight tokens a thread


# the forms of four channels a thread against the general ones, which a state (or row) off 16 bytes takes; the sums have one order
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,kv_heads,dim,rotated,aliased", [(32, 4, 64, 64, True), (3, 1, 20, 12, False), (2, 2, 4, 0, True)])
@pytest.mark.parametrize("lengths,starts", STEPS)
@pytest.mark.parametrize("biased,write", [(True, True), (False, False)])
def test_short_convolution_forms(dtype, heads, kv_heads, dim, rotated, aliased, lengths, starts, biased, write):
    k, channels, slots = lib(dtype), (heads + kv_heads) * dim, list(range(len(lengths), 0, -1))
    n, meta = packed(lengths, starts, slots)
    rows, conv_w = torch.randn(n, channels + 4, device="cuda"), torch.randn(channels, 4, device="cuda")
    bias, rotation = torch.randn(channels, device="cuda") if biased else None, torch.randn(800, rotated // 2, 2, device="cuda") if rotated else None
    ring, table = torch.randn(len(lengths) + 1, 4 * channels, device="cuda"), torch.randperm(50 * len(lengths), device="cuda").int().view(len(lengths), 50)
    results = []
    for offset in (4, 3):
        state = torch.zeros(len(lengths) + 1, 4 * channels + 4, device="cuda")
        state[:, offset:offset + 4 * channels] = ring
        q = torch.full((n, heads * dim), 7.0, device="cuda").to(dtype)
        caches = [torch.full((50 * len(lengths), kv_heads, 16, dim), 7.0, device="cuda").to(dtype) for _ in range(2)]
        k.short_conv_rotary(rows, bias, conv_w, 4, rotation, rotated, True, table, q, caches[0], caches[1] if aliased else None, heads, kv_heads, dim, 16,
                            write, meta, state, offset)
        results.append([q] + caches)
    for got, want in zip(*results):
        torch.testing.assert_close(got.float(), want.float(), rtol=2.0 ** -8 if dtype == torch.bfloat16 else 1e-6, atol=2e-6)


@pytest.mark.parametrize("channels,part", [(2048, 64), (260, 20), (4, 4)])
@pytest.mark.parametrize("lengths,starts", STEPS)
def test_recurrent_unit_forms(channels, part, lengths, starts):
    k, slots = lib(), list(range(len(lengths), 0, -1))
    n, meta = packed(lengths, starts, slots)
    yx, conv_w = torch.randn(n, 2 * channels, device="cuda"), torch.randn(channels, 4, device="cuda")
    x_bias, conv_b, y_bias, r_bias, i_bias, rate = (torch.randn(channels, device="cuda") for _ in range(6))
    gates, kept = torch.randn(n, 2 * channels, device="cuda"), torch.randn(len(lengths) + 1, 6 * channels, device="cuda")
    results = []
    for spare in (0, 1):
        state = torch.zeros(len(lengths) + 1, 6 * channels + spare, device="cuda")
        state[:, :6 * channels] = kept
        u = torch.full((n, channels), float("nan"), device="cuda")
        k.rglru_conv(yx, channels, x_bias, conv_w, conv_b, u, meta, state)
        # (the general form of the gates: rows that begin off 16 bytes)
        mine = torch.zeros(n * 2 * channels + spare, device="cuda")[spare:].view(n, 2 * channels).copy_(gates)
        y = yx.clone()
        k.rglru_gates(mine, u, y, y_bias, r_bias, i_bias, rate.abs(), part)
        results.append((u, mine.clone(), y))
    for got, want in zip(*results):
        torch.testing.assert_close(got, want, rtol=2e-6, atol=2e-6)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,dim", [(32, 64), (3, 128), (5, 16), (1, 32), (4, 48)])
@pytest.mark.parametrize("n", [1, 9, "many", "many and five"])      # (the wide form: two tokens an SM and more)
def test_time_mix_finish(dtype, heads, dim, n):
    many = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    n = {"many": many, "many and five": many + 5}.get(n, n)
    k, width = lib(dtype), heads * dim
    o, gate, norm = torch.randn(n, width, device="cuda"), torch.randn(n, width, device="cuda"), torch.rand(width, device="cuda") + 0.5
    out = torch.full((n, width + 8), float("nan"), device="cuda").to(dtype)
    k.time_mix_finish(o, gate, norm, 1e-5, 1.3, out, heads, dim)
    x = o.double().view(n, heads, dim)
    want = (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5)).view(n, width) * norm.double() * 1.3 * torch.nn.functional.silu(gate.double())
    assert ((out[:, :width].double() - want).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 3e-6) * want.abs() + 1e-6).all()
    assert (out[:, width:] == 0).all()
