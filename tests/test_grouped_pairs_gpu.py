"""Products of rows sorted by group with each group's own matrix on pairs of blocks (256 rows a tile) and on single ones, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# groups without rows, of one row, around a tile and half a tile; columns and inner sizes that end inside a tile; and groups too small for pairs
@pytest.mark.parametrize("counts", [[2700, 0, 1, 257, 2500], [1256, 512, 1255, 2384, 129], [300, 300, 300, 300, 300], [64, 0, 200, 1, 130]])
@pytest.mark.parametrize("N,K", [(2600, 2048), (2816, 264), (4096, 1000)])
@pytest.mark.parametrize("form", ["float", "relu2", "gated"])
def test_groups(counts, N, K, form):
    from stratakv_b200 import ops
    k = ops.kernels_for(torch.bfloat16, 64, verbose=False)
    rows, groups = sum(counts), len(counts)
    a = torch.randn(rows, K, device="cuda").bfloat16()
    w = (torch.randn(groups, 2 * N if form == "gated" else N, K, device="cuda") / math.sqrt(K)).bfloat16()
    offsets = torch.tensor([0] + [sum(counts[:i + 1]) for i in range(groups)], dtype=torch.int32, device="cuda")
    out = torch.full((rows, N), float("nan"), device="cuda", dtype=torch.float32 if form == "float" else torch.bfloat16)
    k.expert_linear(a, w, offsets, out, activation={"float": None, "relu2": "relu2", "gated": "silu"}[form], gated=form == "gated")
    z = torch.cat([a[lo:hi].double() @ w[e].double().T for e, (lo, hi) in enumerate(zip(offsets.tolist(), offsets.tolist()[1:]))])
    if form == "gated":
        tiles = z.view(rows, -1, 2, 8)
        g, u = tiles[:, :, 0].reshape(rows, N), tiles[:, :, 1].reshape(rows, N)
        want = torch.nn.functional.silu(g) * u
    else:
        want = torch.relu(z) ** 2 if form == "relu2" else z
    # sums kept in tensor memory (cut off at each of K / 16 steps: at most 2^-23 of a sum of order one each), then one rounding to bfloat16
    slack = 4 * (K / 16) * 2.0 ** -23 + 1e-6
    assert ((out.double() - want).abs() <= (2.0 ** -8 if form != "float" else 0.0) * want.abs() + slack * 8 * (1 + want.abs())).all()
    assert int(k.error_flag) == 0
