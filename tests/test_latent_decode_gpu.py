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
