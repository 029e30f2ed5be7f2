"""How many parts a decode step over a latent's cached rows is cut into."""
import ctypes

import pytest

from stratakv_b200.csrc import build
from stratakv_b200.parts.latent_attention import decode_parts


def test_two_parts_only_where_they_run_on_tensor_cores():
    """A latent of 512 with a rotated part of 64 in a large batch went through memory in two parts for a kernel that does not serve it."""
    assert decode_parts(64 * 128, 1000, 148, False) == 1 and decode_parts(64 * 128, 1000, 148, True) == 2
    assert decode_parts(8 * 32, 40, 148, False) == 1
    # short contexts: the kernel for parts and the merge take longer than the walk over a few keys
    assert decode_parts(8 * 32, 32, 148, True) == 1 and decode_parts(8 * 32, 33, 148, True) == 2
    assert decode_parts(8 * 32, 780, 148, False) == decode_parts(8 * 32, 780, 148, True) == 13
    assert decode_parts(4, 100000, 148, True) == 64


@pytest.mark.parametrize("dim,vdim,serves", [(272, 256, True), (320, 256, True), (16, 16, True), (576, 512, False), (336, 256, False),
                                             (288, 272, False), (280, 256, False), (272, 250, False), (32, 48, False)])
def test_what_the_tensor_core_form_serves(dim, vdim, serves):
    for dtype in ("bfloat16", "float32"):
        path = build.find_built(dtype, 64)
        if path is None:
            pytest.skip("not compiled yet")
        assert ctypes.CDLL(str(path)).skv_attention_latent_serves(dim, vdim) == int(serves and dtype == "bfloat16")
