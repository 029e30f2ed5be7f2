"""Matrix states with a decay per head at whole tiles of 64, several cells a thread in the walk over chunks, and retention
on the same kernels, against the recurrence in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def recurrence(q, k, v, log_decay, S, n_state):
    """float64: outputs [T, H, P], key-sum products [T, H] and the state after; q, k [T, H, N], v [T, H, P], log_decay [T, H]."""
    out, dots = [], []
    for t in range(len(q)):
        d = torch.exp(log_decay[t])
        S = d[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
        n_state = d[:, None] * n_state + k[t]
        out.append((q[t][:, None, :] @ S)[:, 0])
        dots.append((n_state * q[t]).sum(-1))
    return torch.stack(out), torch.stack(dots), S, n_state


# chunks of 64 that are full, end at a tile's edge of 16 or a token behind it, and are one token; states that go on; heads that
# share keys; every mechanism of the float kernel
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,groups,dim,vdim", [(3, 3, 64, 64), (4, 2, 128, 64), (2, 1, 64, 128), (2, 2, 128, 128)])
@pytest.mark.parametrize("form", ["fixed", "fixed_silu", "per_token", "forgets", "floor"])
@pytest.mark.parametrize("portions", [((64, 1, 130), (17, 65, 2)), ((200, 16, 63),)])
def test_linear_state_in_whole_tiles(dtype, heads, groups, dim, vdim, form, portions):
    from stratakv_b200.ops import kernels_for
    ops = kernels_for(dtype, 64, verbose=False)
    generator = torch.Generator(device="cuda").manual_seed(heads * dim + vdim)
    normal = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    total = [sum(p[i] for p in portions) for i in range(3)]
    width = 2 * groups * dim + heads * vdim
    rows = [normal(n, width + 4) for n in total]
    decay = torch.tensor([0.9, 0.99, 0.999, 0.0], device="cuda")[:heads].contiguous()
    if form.startswith("fixed"):
        logs = [torch.log(decay.double()).expand(n, heads) for n in total]
    else:
        logs = [-torch.rand(n, heads, generator=generator, device="cuda") * 0.1 for n in total]
        if form == "forgets":                                   # e^-60 now and then, and once everything
            for l in logs:
                l[::7] = -60.0
                l[len(l) // 2] = -4000.0
    scale, skip = [torch.rand(n, heads, generator=generator, device="cuda") for n in total], normal(heads)
    floor = [0.5 + torch.rand(n, heads, generator=generator, device="cuda") for n in total]
    per_half = heads * dim * (vdim + (form == "floor"))
    offset = 8
    state = torch.full((5, offset + 2 * per_half), 1e30, device="cuda")
    slots, want = [3, 0, 4], []
    for i in range(3):
        r = rows[i].double()
        act = torch.nn.functional.silu if form == "fixed_silu" else (lambda z: z)
        spread = lambda z: act(z).view(-1, groups, dim).repeat_interleave(heads // groups, dim=1)
        q, k, v = spread(r[:, :groups * dim]), spread(r[:, groups * dim:2 * groups * dim]), act(r[:, 2 * groups * dim:width]).view(-1, heads, vdim)
        if not form.startswith("fixed"):
            k = k * scale[i].double()[:, :, None]
        zeros = k.new_zeros(heads, dim, vdim)
        o, dots, S, n_state = recurrence(q, k, v, logs[i].double(), zeros, zeros[:, :, 0])
        # the sum of the magnitudes that a float sum's error is a fraction of
        mass = recurrence(q.abs(), k.abs(), v.abs(), logs[i].double(), zeros, zeros[:, :, 0])[0]
        if form == "floor":
            weight = torch.maximum((0.5 * dots).abs(), floor[i].double()) + 1e-6
            o, mass = 0.5 * o / weight[:, :, None], 0.5 * mass / weight[:, :, None] * 3
        elif not form.startswith("fixed"):
            o, mass = o + skip.double()[:, None] * v, mass + (skip.double()[:, None] * v).abs()
        want.append((o, mass, S))
    got, at = [[], [], []], [0, 0, 0]
    for portion in portions:
        cu = torch.tensor([0] + list(torch.tensor(portion).cumsum(0)), dtype=torch.int32, device="cuda")
        positions = torch.cat([torch.arange(at[i], at[i] + portion[i], dtype=torch.int32) for i in range(3)]).cuda()
        seqs = torch.repeat_interleave(torch.arange(3, dtype=torch.int32), torch.tensor(portion)).cuda()
        meta = (positions, seqs, cu, torch.tensor(slots, dtype=torch.int32, device="cuda"))
        pick = lambda parts: torch.cat([parts[i][at[i]:at[i] + portion[i]] for i in range(3)]).contiguous()
        more = dict(decay=decay, silu=form == "fixed_silu") if form.startswith("fixed") else dict(log_decay=pick(logs), key_scale=pick(scale))
        if form == "floor":
            more.update(floor=pick(floor), floor_eps=1e-6, out_scale=0.5)
        elif not form.startswith("fixed"):
            more.update(skip=skip)
        need = ops.linear_state_scratch(3, max(portion), heads, dim, vdim, form == "floor")
        out = torch.full((sum(portion), heads * vdim), float("nan"), device="cuda")
        ops.linear_state(pick(rows), 0, groups * dim, 2 * groups * dim, out, state, meta, heads, groups, dim, vdim, max(portion),
                         scratch=torch.full((need,), float("nan"), device="cuda"), state_offset=offset, **more)
        for i, part in enumerate(out.split(list(portion))):
            got[i].append(part)
            at[i] += portion[i]
    for i in range(3):
        o, mass, S = want[i]
        # sums of up to a few hundred products in float: a few 2^-24 of their magnitudes' sum (operands rounded to bfloat16 or to
        # sixteen bits anywhere would be off by 2^-9 or 2^-17 of a product)
        assert ((torch.cat(got[i]).double().view(-1, heads, vdim) - o).abs() <= 3e-6 * mass + 1e-6).all()
        last = state[slots[i], offset + ((total[i] - 1) & 1) * per_half:][:heads * dim * vdim].view(heads, dim, vdim)
        assert (last.double() - S).abs().max() <= 3e-6 * (S.abs().max() + 10)
    assert (state[[1, 2]] == 1e30).all() and (state[:, :offset] == 1e30).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,dim,vdim,rotated,spare", [(3, 64, 64, 32, 0), (2, 128, 64, 128, 8), (2, 64, 128, 0, 1), (2, 192, 64, 64, 0)])
def test_retention_in_whole_tiles(dtype, heads, dim, vdim, rotated, spare):
    """A head size of 192 and rows that are no whole 16 bytes stay on retention's own kernels."""
    from stratakv_b200.ops import kernels_for
    from stratakv_b200.parts.position import rope_table
    ops = kernels_for(dtype, 64, verbose=False)
    generator = torch.Generator(device="cuda").manual_seed(dim + vdim)
    lengths, eps = (130, 1, 64), 1e-5
    width = 2 * heads * (dim + vdim) + spare
    rows = [torch.randn(n, width, generator=generator, device="cuda") for n in lengths]
    decay = torch.tensor([0.9, 0.999, 1.0], device="cuda")[:heads].contiguous()
    table = torch.from_numpy(rope_table(rotated, 10000.0, 256)).cuda() if rotated else None
    state = torch.full((4, 2 * heads * dim * vdim), 1e30, device="cuda")
    slots = [2, 0, 3]
    want = []
    for r in rows:
        n = len(r)
        turn = lambda z: z
        if rotated:
            cos, sin = (table[:n, :, i].double()[:, None] for i in (0, 1))
            half = rotated // 2
            turn = lambda z: torch.cat([z[..., :half] * cos - z[..., half:rotated] * sin, z[..., half:rotated] * cos + z[..., :half] * sin, z[..., rotated:]], -1)
        q, k = (turn(r[:, i * heads * dim:(i + 1) * heads * dim].double().view(n, heads, dim)) for i in (0, 1))
        v = r[:, 2 * heads * dim:][:, :heads * vdim].double().view(n, heads, vdim)
        gate = r[:, 2 * heads * dim + heads * vdim:][:, :heads * vdim].double()
        run = lambda q, k, v: recurrence(q, k, v, torch.log(decay.double()).expand(n, heads), v.new_zeros(heads, dim, vdim), v.new_zeros(heads, dim))[0]
        o, mass = run(q, k * dim ** -0.5, v), run(q.abs(), k.abs() * dim ** -0.5, v.abs())
        factor = torch.rsqrt((o * o).mean(-1, keepdim=True) + eps)
        act = torch.nn.functional.silu(gate)
        want.append(((o * factor).reshape(n, -1) * act, (mass * factor).reshape(n, -1) * act.abs()))
    cu = torch.tensor([0, 130, 131, 195], dtype=torch.int32, device="cuda")
    positions = torch.cat([torch.arange(n, dtype=torch.int32) for n in lengths]).cuda()
    meta = (positions, torch.repeat_interleave(torch.arange(3), torch.tensor(lengths)).int().cuda(), cu, torch.tensor(slots, dtype=torch.int32, device="cuda"))
    out = torch.full((195, heads * vdim + 8), float("nan"), device="cuda").to(dtype)
    scratch = torch.full((ops.retention_scratch(3, 130, heads, dim, vdim),), float("nan"), device="cuda")
    ops.retention(torch.cat(rows).contiguous(), table, rotated, decay, eps, out, state, meta, heads, dim, vdim, 130, scratch)
    ref, mass = (torch.cat(parts) for parts in zip(*want))
    assert (out[:, heads * vdim:] == 0).all()
    # a few 2^-24 of what the float sums' terms add up to, divided by the head's root mean square as they are
    assert ((out[:, :heads * vdim].double() - ref).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * ref.abs() + 4e-6 * mass + 1e-6).all()


# one token a sequence: value heads that divide a block's columns (with fewer rows of the state than a thread has on its way, as many,
# several rounds) and one that does not; a state to go on from and none
@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128), (16, 4), (6, 1024), (200, 256), (20, 12)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_retention_of_one_token(dim, vdim, dtype):
    from stratakv_b200.ops import kernels_for
    k, heads, places = kernels_for(dtype, 64, verbose=False), 3, [0, 5, 8, 0, 1]
    n = len(places)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    fused = torch.randn(n, 2 * heads * (dim + vdim), device="cuda")
    q, key, v, gate = (t.double().view(n, heads, -1) for t in fused.split([heads * dim, heads * dim, heads * vdim, heads * vdim], -1))
    decay = torch.tensor([0.5, 0.97, 0.999], device="cuda")
    state = torch.randn(n + 1, 2 * heads * dim * vdim, device="cuda")
    before, slots = state.double().view(n + 1, 2, heads, dim, vdim), [3, 0, 5, 1, 2]
    out = torch.full((n, heads * vdim + 8), float("nan"), device="cuda").to(dtype)
    k.retention(fused, None, 0, decay, 1e-5, out, state, (i32(places), i32(range(n)), i32(range(n + 1)), i32(slots)), heads, dim, vdim, 1)
    for s, (p, slot) in enumerate(zip(places, slots)):
        old = before[slot, (p - 1) & 1] if p > 0 else torch.zeros(heads, dim, vdim, device="cuda", dtype=torch.float64)
        fresh = decay.double()[:, None, None] * old + key[s, :, :, None] * dim ** -0.5 * v[s, :, None, :]
        got = state.view(n + 1, 2, heads, dim, vdim)[slot]
        assert ((got[p & 1].double() - fresh).abs() <= 1e-6 * (1 + fresh.abs())).all()
        assert p == 0 or torch.equal(got[(p - 1) & 1].double(), old)
        o = torch.einsum("hd,hde->he", q[s], fresh)
        mass = torch.einsum("hd,hde->he", q[s].abs(), fresh.abs())
        f, g = torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-5), torch.nn.functional.silu(gate[s])
        # float sums over dim err in proportion to their mass: by d in o f, and f by at most f^2 d; then one rounding of the result
        d = 1e-6 * mass
        error = (d * f + d.amax(-1, keepdim=True) * o.abs() * f * f) * g.abs() + (2.0 ** -8 if dtype == torch.bfloat16 else 2e-6) * (o * f * g).abs() + 1e-6
        assert ((out[s, :heads * vdim].double().view(heads, vdim) - o * f * g).abs() <= error).all()
    assert (out[:, heads * vdim:] == 0).all()


# heads of a group in one block (enough blocks of them) against a sequence at a time, which has a block a head
@pytest.mark.parametrize("heads,groups,dim,vdim", [(64, 2, 128, 64), (64, 16, 64, 128)])
@pytest.mark.parametrize("floor", [False, True])
def test_heads_of_a_group_share_their_scores(heads, groups, dim, vdim, floor):
    from stratakv_b200.ops import kernels_for
    ops = kernels_for(torch.bfloat16, 64, verbose=False)
    lengths, i32 = [130, 64, 1, 65, 20] * 4, lambda values: torch.tensor(values, dtype=torch.int32, device="cuda")
    n, seqs = sum(lengths), len(lengths)
    starts = [0 if s % 3 else 7 for s in range(seqs)]
    rows = torch.randn(n, 2 * groups * dim + heads * vdim, device="cuda")
    logs, scale, least = -torch.rand(n, heads, device="cuda") * 0.1, torch.rand(n, heads, device="cuda"), 0.5 + torch.rand(n, heads, device="cuda")
    half = heads * dim * (vdim + floor)
    kept = torch.randn(seqs, 2 * half, device="cuda")

    def run(first, count):
        span, base = lengths[first:first + count], sum(lengths[:first])
        cu = [0]
        for length in span:
            cu.append(cu[-1] + length)
        meta = (i32([starts[first + s] + i for s, length in enumerate(span) for i in range(length)]), i32([s for s, length in enumerate(span) for _ in range(length)]),
                i32(cu), i32(range(first, first + count)))
        out, part = torch.full((cu[-1], heads * vdim), float("nan"), device="cuda"), slice(base, base + cu[-1])
        more = dict(floor=least[part].contiguous(), floor_eps=1e-6, out_scale=0.5) if floor else {}
        need = ops.linear_state_scratch(count, max(span), heads, dim, vdim, floor)
        ops.linear_state(rows[part].contiguous(), 0, groups * dim, 2 * groups * dim, out, state, meta, heads, groups, dim, vdim, max(span),
                         scratch=torch.full((need,), float("nan"), device="cuda"), log_decay=logs[part].contiguous(), key_scale=scale[part].contiguous(), **more)
        return out

    state = kept.clone()
    together, after = run(0, seqs), state
    state = kept.clone()
    apart = torch.cat([run(s, 1) for s in range(seqs)])
    # (a sequence of one token alone is a step of another kernel: its sums have another order)
    torch.testing.assert_close(together, apart, rtol=2e-5, atol=2e-5 * float(apart.abs().max()))
    torch.testing.assert_close(after, state, rtol=1e-5, atol=1e-5)
