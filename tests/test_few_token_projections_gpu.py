"""Projections of at most 16 tokens, whose blocks walk the weight's tiles, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles of 16 rows: as many as two blocks an SM of 148 hold, one more, several rounds with a last tile that is not whole; inner sizes of
# a part of a step, of one half of a warp's steps, of an odd number of halves, the longest that is walked and one beyond
@pytest.mark.parametrize("M", [1, 7, 8])
@pytest.mark.parametrize("N", [4736, 4752, 9250, 16384])
@pytest.mark.parametrize("K", [8, 1000, 2048, 2056, 3072, 3080])
def test_tiles_are_walked(M, N, K):
    check(M, N, K)


@pytest.mark.parametrize("M,N,K", [(8, 6146, 4096), (9, 6144, 4096), (16, 6146, 4096), (16, 6142, 4096), (13, 3072, 12288), (12, 40000, 648)])
def test_up_to_sixteen_tokens_over_large_weights(M, N, K):
    check(M, N, K)


# tiles of 16 rows around one and two blocks an SM of 148 and beyond; inner sizes around what a warp's activations in registers and its
# slots hold (4, 8 steps of 16 warps), and shorter than a warp's first step
@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N", [16, 2368, 2384, 4736, 4768])
@pytest.mark.parametrize("K", [24, 512, 2048, 2056, 4096, 4104, 5632])
def test_blocks_walk_and_slots_wrap(M, N, K):
    check(M, N, K)


@pytest.mark.parametrize("M,N,K", [(16, 6416, 512), (8, 12304, 4104)])
def test_the_last_block_finishes_wide_rows(M, N, K):
    """Rows too wide for every consumer to add their partial sums up: the writer's last block leaves the factors, and the counter at zero."""
    from types import SimpleNamespace
    from stratakv_b200 import ops
    from stratakv_b200.residual import ResidualStats
    k = ops.kernels_for(torch.bfloat16, 64, verbose=False)
    stats = ResidualStats.allocate(lambda name, shape, dtype, zero=False: torch.zeros(shape, dtype=dtype, device="cuda"), M, N, torch.bfloat16)
    norm = SimpleNamespace(gamma=1 + 0.2 * torch.randn(N, device="cuda"), spec=SimpleNamespace(eps=1e-5))
    for _ in range(2):
        a, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
        x, plain = torch.ones(M, N, device="cuda"), torch.ones(M, N, device="cuda")
        stats.expect(norm)
        k.linear(a, w, x, ops.MODE_ADD_F32, stats=stats)
        k.linear(a, w, plain, ops.MODE_ADD_F32)
        assert stats.n_partials == 0 and int(stats.counter) == 0 and torch.equal(x, plain)
        assert torch.equal(stats.scaled, (x * norm.gamma).bfloat16())
        want = torch.rsqrt((x.double() ** 2).mean(-1) + 1e-5)
        assert ((stats.row_scale.double() - want).abs() <= 1e-5 * want).all()


def check(M, N, K):
    from stratakv_b200 import ops
    k = ops.kernels_for(torch.bfloat16, 64, verbose=False)
    a, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
    ref, bound = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    error = 2e-6 * (1 + bound)                                  # float sums, in proportion to the products' magnitudes
    out = torch.full((M, N), float("nan"), device="cuda")
    k.linear(a, w, out, ops.MODE_STORE_F32)
    assert ((out.double() - ref).abs() <= error).all()
    base = torch.randn(M, N, device="cuda")
    total = base.clone()
    k.linear(a, w, total, ops.MODE_ADD_F32)
    assert ((total.double() - base.double() - ref).abs() <= error + 1e-6 * base.abs()).all()
    rounded = torch.full((M, N), float("nan"), device="cuda").bfloat16()
    k.linear(a, w, rounded, ops.MODE_ACT, "relu2")
    want = torch.relu(ref) ** 2
    assert ((rounded.double() - want).abs() <= 2 * error * torch.relu(ref) + error ** 2 + 2.0 ** -8 * want).all()
    if N % 16 == 0:
        gated = torch.full((M, N // 2), float("nan"), device="cuda").bfloat16()
        k.linear(a, w, gated, ops.MODE_GATED, "silu")           # tiles of 8 gate rows and their 8 up rows
        tiles, slack = ref.view(M, -1, 2, 8), error.view(M, -1, 2, 8)
        g, u, eg, eu = (x.reshape(M, N // 2) for x in (tiles[:, :, 0], tiles[:, :, 1], slack[:, :, 0], slack[:, :, 1]))
        want = torch.nn.functional.silu(g) * u
        assert ((gated.double() - want).abs() <= 1.2 * eg * u.abs() + torch.nn.functional.silu(g).abs() * eu + 2.0 ** -8 * want.abs() + 1e-6).all()
    assert int(k.error_flag) == 0


@pytest.mark.parametrize("M,partials", [(1, 1464), (8, 2000), (8, 2001), (16, 1403)])
def test_any_number_of_partial_sums(M, partials):
    """A folded norm's factors from more partial sums than a block could stage: they are added up as they are read."""
    from stratakv_b200 import ops
    from stratakv_b200.residual import NormedRows
    k, N, K, eps = ops.kernels_for(torch.bfloat16, 64, verbose=False), 2400, 1024, 1e-5
    a, w = torch.randn(M, K, device="cuda").bfloat16(), (torch.randn(N, K, device="cuda") / math.sqrt(K)).bfloat16()
    sums = torch.rand(M, partials, device="cuda")
    out = torch.full((M, N), float("nan"), device="cuda")
    k.linear(NormedRows(a, torch.ones(M, device="cuda"), partials=sums, n_partials=partials, eps=eps), w, out, ops.MODE_STORE_F32)
    factor = torch.rsqrt(sums.double().sum(-1, keepdim=True) / K + eps)
    ref, bound = a.double() @ w.double().T * factor, a.double().abs() @ w.double().abs().T * factor
    assert ((out.double() - ref).abs() <= 2e-6 * (1 + bound)).all()
