"""Projections of at most 16 tokens where blocks walk the weight's tiles (at most 8 tokens), and of 8 to 16 tokens over weights around
48 MB, against float64."""
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
