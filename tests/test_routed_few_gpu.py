"""The experts of few pairs against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def lib(dtype=torch.bfloat16):
    from stratakv_b200.ops import kernels_for
    return kernels_for(dtype, 64, verbose=False)


# pairs at both ends of what the streaming kernel takes and one beyond; experts without rows, with up to 8, with several rounds;
# inner sizes of one load, one step, part of a round and several; outputs that end inside a tile
@pytest.mark.parametrize("n,top,experts,N,K", [(1, 2, 8, 64, 8), (8, 2, 8, 88, 2816), (16, 2, 8, 40, 520), (32, 1, 8, 24, 2048), (11, 1, 3, 16, 4104),
                                               (64, 1, 16, 72, 1032), (65, 1, 16, 16, 1032), (40, 2, 80, 16, 64),
                                               (41, 2, 80, 16, 64)])
@pytest.mark.parametrize("form", ["relu2", "gated", "gated_clamp", "weighted", "float"])
@pytest.mark.parametrize("crowded", [False, True])
def test_experts_of_few_pairs(n, top, experts, N, K, form, crowded):
    k = lib()
    pairs = n * top
    h = torch.randn(n, K, device="cuda").bfloat16()
    gated = form in ("gated", "gated_clamp", "weighted")
    w = (torch.randn(experts, 2 * N if gated else N, K, device="cuda") / math.sqrt(K)).bfloat16()
    chosen = torch.stack([torch.randperm(experts, device="cuda")[:top] for _ in range(n)]).int()
    if crowded and top == 1:
        chosen[:] = experts - 1
    offsets, order = torch.empty(experts + 1, dtype=torch.int32, device="cuda"), torch.empty(pairs, dtype=torch.int32, device="cuda")
    place, weights = torch.empty(n, top, dtype=torch.int32, device="cuda"), torch.rand(n, top, device="cuda")
    k.sort_by_expert(chosen, experts, offsets, order, place)
    few = k.expert_few(pairs, experts, K)
    assert few == (pairs <= (4 if K >= 1024 else 1) * experts)
    rows = h[order.long()]
    more = dict(rows=order)
    if form == "weighted":
        factor = torch.empty(pairs, device="cuda")
        factor[place.reshape(-1).long()] = weights.reshape(-1)
        rows = (rows.float() * factor[:, None]).bfloat16()                 # (rounded as the kernel rounds it)
        more = dict(rows=order, place=place, weights=weights) if few else dict(rows=None)
    source = h if more["rows"] is not None else rows
    activation = {"relu2": "relu2", "gated": "silu", "gated_clamp": "swiglu_clamp", "weighted": "swiglu_clamp", "float": None}[form]
    out = torch.full((pairs, N), float("nan"), device="cuda", dtype=torch.float32 if form == "float" else torch.bfloat16)
    k.expert_linear(source, w, offsets, out, activation=activation, gated=gated, activation_param=7.0 if "clamp" in (activation or "") else 0.0, **more)
    expert = torch.empty(pairs, dtype=torch.long, device="cuda")
    expert[place.reshape(-1).long()] = chosen.reshape(-1).long()
    z = torch.einsum("pk,pnk->pn", rows.double(), w.double()[expert])
    if gated:
        tiles = z.view(pairs, -1, 2, 8)
        g, u = tiles[:, :, 0].reshape(pairs, N), tiles[:, :, 1].reshape(pairs, N)
        if activation == "silu":
            ref = torch.nn.functional.silu(g) * u
        else:
            ref = g.clamp(max=7.0) * torch.sigmoid(1.702 * g.clamp(max=7.0)) * (u.clamp(-7.0, 7.0) + 1.0)
    else:
        ref = torch.relu(z) ** 2 if form == "relu2" else z
    # float sums of products that add up to order one, then one rounding to bfloat16
    assert ((out.double() - ref).abs() <= (2.0 ** -8 if form != "float" else 0.0) * ref.abs() + 2e-5 * (1 + ref.abs())).all()


# tokens at a block's edges; dot products of one, two and several tiles and beyond a round of them, with and without the shared gate;
# rows of one step, of fewer steps than warps, of several rounds, and of a width that is no multiple of 32 (a block a token)
@pytest.mark.parametrize("n", [1, 16, 17, 40])
@pytest.mark.parametrize("experts,shared,groups", [(1, True, 0), (8, False, 2), (8, True, 0), (15, True, 0), (17, False, 0), (70, True, 7), (1024, False, 0)])
@pytest.mark.parametrize("hidden", [32, 480, 2080, 4096, 72])
@pytest.mark.parametrize("softmax", [False, True])
def test_router(n, experts, shared, groups, hidden, softmax):
    k, top = lib(), min(2, experts)
    h, w = torch.randn(n, hidden, device="cuda").bfloat16(), (torch.randn(experts, hidden, device="cuda") / math.sqrt(hidden)).bfloat16()
    correction, gate = torch.randn(experts, device="cuda"), torch.randn(hidden, device="cuda").bfloat16() if shared else None
    share = torch.full((n,), float("nan"), device="cuda") if shared else None
    chosen, weights = torch.full((n, top), -1, dtype=torch.int32, device="cuda"), torch.full((n, top), float("nan"), device="cuda")
    keep = groups // 2 if groups else 0
    k.route_tokens(h, w, correction, top, 1.5, True, chosen, weights, gate, share, softmax=softmax, groups=groups, keep=keep)
    z = h.double() @ w.double().T
    score = torch.softmax(z, -1) if softmax else torch.sigmoid(z)
    choice = score + correction.double()
    if groups:
        best = choice.view(n, groups, -1).amax(-1)
        kept = torch.zeros_like(best).scatter_(1, best.topk(keep, -1).indices, 1.0).repeat_interleave(experts // groups, -1)
        choice = torch.where(kept > 0, choice, -math.inf)
    want = choice.topk(top, -1)
    got = choice.gather(1, chosen.long())
    # a float sum of products of order one errs by a few 1e-7: only scores that close may change places
    assert (got - want.values).abs().max() <= 1e-5 and all(len(set(row)) == top for row in chosen.tolist())
    picked = score.gather(1, chosen.long())
    torch.testing.assert_close(weights.double(), 1.5 * picked / picked.sum(-1, keepdim=True), rtol=1e-5, atol=1e-7)
    if shared:
        torch.testing.assert_close(share.double(), torch.sigmoid(h.double() @ gate.double()), rtol=2e-5, atol=1e-6)
