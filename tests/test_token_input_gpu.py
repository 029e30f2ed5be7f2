"""The per-token input on tensor cores against float64: widths that fill one block, part of a cluster and eight blocks,
token counts at the edges of 16 and 32, and where many-token blocks take over."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,hidden", [(16, 64), (32, 192), (64, 2048), (32, 3072), (64, 4096), (16, 8192), (64, 1984)])
@pytest.mark.parametrize("n,next_norm", [(1, True), (5, False), (16, True), (17, True), (256, False), (257, True), (300, False)])
def test_token_side_on_tensor_cores(dim, hidden, n, next_norm):
    from stratakv_b200.ops import kernels_for
    k = kernels_for(torch.bfloat16, 64, verbose=False)
    vocab, stride, offset, eps = 50, 3 * dim, dim, 1e-5
    x = 3 * torch.randn(n, hidden, device="cuda")
    ids = torch.randint(0, vocab, (n,), device="cuda", dtype=torch.int32)
    table = torch.randn(vocab, stride, device="cuda").bfloat16()
    gate = (torch.randn(dim, hidden, device="cuda") / math.sqrt(hidden)).bfloat16()
    proj_t = torch.randn(dim, hidden, device="cuda").bfloat16()
    norm, gamma = 1 + 0.1 * torch.randn(hidden, device="cuda"), 1 + 0.1 * torch.randn(hidden, device="cuda")
    gated = torch.nn.functional.gelu(x.double() @ gate.double().T, approximate="tanh") * table[ids.long(), offset:offset + dim].double()
    y = gated @ proj_t.double()
    want = x.double() + y * torch.rsqrt((y * y).mean(-1, keepdim=True) + eps) * norm.double()
    got = x.clone()
    out = torch.full((n, hidden), float("nan"), device="cuda", dtype=torch.bfloat16) if next_norm else None
    k.token_side(got, ids, table, offset, dim, gate, proj_t, norm, eps, next_gamma=gamma if next_norm else None, next_eps=eps, next_out=out)
    # float sums over hidden (of order-three numbers with weights of order 1/sqrt(hidden)) and over dim, then a unit row:
    # a few 2^-24 of each, as with FMA; a stream rounded to bfloat16 anywhere would be off by 1e-3
    assert (got.double() - want).abs().max() <= 2e-5
    if next_norm:
        normed = want * torch.rsqrt((want * want).mean(-1, keepdim=True) + eps) * gamma.double()
        assert ((out.double() - normed).abs() <= 2.0 ** -8 * normed.abs() + 2e-5).all()


# the last count whose clusters all have SMs to themselves, the first that takes the form of fewer registers, and the most
@pytest.mark.parametrize("dim,hidden", [(64, 2048), (32, 4096), (32, 8192), (64, 4096)])
@pytest.mark.parametrize("n", [240, 241, 256])
def test_token_side_where_two_blocks_share_an_sm(dim, hidden, n):
    test_token_side_on_tensor_cores(dim, hidden, n, True)


def test_token_side_skips_an_unknown_id():
    from stratakv_b200.ops import kernels_for
    k = kernels_for(torch.bfloat16, 64, verbose=False)
    x = torch.randn(3, 128, device="cuda")
    before = x.clone()
    w = torch.randn(32, 128, device="cuda").bfloat16()
    ids = torch.tensor([2, -1, 7], dtype=torch.int32, device="cuda")
    k.token_side(x, ids, torch.randn(7, 32, device="cuda").bfloat16(), 0, 32, w, w, torch.ones(128, device="cuda"), 1e-5)
    assert torch.equal(x[1:], before[1:]) and not torch.equal(x[0], before[0])


@pytest.mark.parametrize("hidden", [256, 4096])
@pytest.mark.parametrize("choose", ["argmax", "sample"])
def test_ids_chosen_by_the_kernels_in_front(hidden, choose):
    """The chooser, the embedding and the token input one behind the other on a stream: each may start before the one in front has
    finished, and none may read the ids before they are there."""
    from stratakv_b200.ops import kernels_for
    k = kernels_for(torch.bfloat16, 64, verbose=False)
    n, dim, vocab = 8, 32, 100000
    g = torch.Generator(device="cuda").manual_seed(3)
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    logits, embedding, table = normal(n, vocab), normal(vocab, hidden).bfloat16(), normal(vocab, dim).bfloat16()
    gate, proj_t, norm = normal(dim, hidden).bfloat16(), normal(dim, hidden).bfloat16(), torch.ones(hidden, device="cuda")
    counters = torch.zeros(n, dtype=torch.int32, device="cuda")

    def step(ids):
        x = torch.empty(n, hidden, device="cuda")
        if ids is not settled:
            if choose == "argmax":
                k.argmax(logits, ids)
            else:
                k.sample(logits, ids, 1.0, 1, 1.0, 0, counters, counters)
        k.embed(embedding, ids, x)
        k.token_side(x, ids, table, 0, dim, gate, proj_t, norm, 1e-5)
        return x

    settled = logits.argmax(-1).int()
    torch.cuda.synchronize()
    want, stale = step(settled), ((settled + 1) % vocab).int()
    busy = torch.empty(1 << 28, device="cuda")
    for _ in range(10):
        ids = stale.clone()
        torch.cuda.synchronize()
        busy.add_(1.0)                                   # (the three launches queue up behind it)
        assert torch.equal(step(ids), want)
        assert torch.equal(ids, settled)
