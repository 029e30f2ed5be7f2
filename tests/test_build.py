"""What is compiled per head size, and that the libraries of one dtype share the rest."""
import ctypes
import re
import subprocess

import pytest
import torch

from stratakv_b200.csrc import build


def test_only_what_reads_the_head_size_is_compiled_per_head_size():
    """Sixteen libraries of every kernel were 441 MB, too much to carry; only the attention files differ between them."""
    sources = {path.name for path in build.CSRC.glob("*.cu")}
    assert sources == set(build.HEAD_SOURCES) | set(build.COMMON_SOURCES) and not set(build.HEAD_SOURCES) & set(build.COMMON_SOURCES)
    for name in sources:
        text = (build.CSRC / name).read_text()
        assert bool(re.search(r"\bSKV_HEAD_DIM\b", text)) == (name in build.HEAD_SOURCES), name
        assert ('#include "head_size.cuh"' in text) == (name in build.HEAD_SOURCES), name
    assert build.common_library_name("bfloat16") != build.common_library_name("float32")
    assert build.library_name("bfloat16", 64) != build.library_name("bfloat16", 128)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_one_handle_has_both_libraries_and_one_message(dtype):
    path = build.find_built(dtype, 64)
    if path is None:
        pytest.skip("not compiled yet")
    common = path.parent / build.common_library_name(dtype)
    assert path.stat().st_size < common.stat().st_size / 4
    lib = ctypes.CDLL(str(path))
    lib.skv_last_error.restype = ctypes.c_char_p
    assert lib.skv_library_head_dim() == 64 and lib.skv_library_dtype() == build.DTYPE_CODES[dtype]
    null = ctypes.c_void_p(0)
    # a refusal of the attention library, then one of the common library: no kernel is reached
    one = ctypes.c_int(1)
    assert lib.skv_attention(null, null, null, null, one, null, null, null, one, one, one, ctypes.c_int(48), ctypes.c_int(16),
                             ctypes.c_float(1.0), ctypes.c_int(0), null) != 0
    assert lib.skv_last_error().startswith(b"skv_attention:")
    assert lib.skv_rmsnorm(null, null, ctypes.c_float(1.0), null, null, one, ctypes.c_int(0), one, null) != 0
    assert lib.skv_last_error().startswith(b"skv_rmsnorm:")


# in the package's own folder; the one for temporary files is shared with other copies of the package
@pytest.mark.parametrize("own", [True, False])
def test_a_new_library_replaces_those_of_older_sources(own, tmp_path, monkeypatch):
    monkeypatch.setattr(build, "CSRC", tmp_path if own else tmp_path / "elsewhere")
    folder = tmp_path / "_build"
    folder.mkdir()
    names = ["libstratakv_bf16_0123456789ab.so", "libstratakv_bf16_ba9876543210.so", "libstratakv_bf16_hd64_0123456789ab.so",
             "libstratakv_bf16_hd64_ba9876543210.so", "libstratakv_bf16_hd6_0123456789ab.so", "libstratakv_f32_0123456789ab.so"]
    for name in names:
        (folder / name).write_text("")
    build.drop_older(folder / names[0])
    assert {path.name for path in folder.iterdir()} == set(names) - ({names[1]} if own else set())
    build.drop_older(folder / names[2])
    assert {path.name for path in folder.iterdir()} == set(names) - ({names[1], names[3]} if own else set())


def test_shared_memory_is_asked_for_on_every_device():
    """A kernel's limit belongs to a device: a status kept once per process left a second GPU's launches refused."""
    for path in build.CSRC.glob("*.cu"):
        assert "static const cudaError_t" not in path.read_text(), path.name


# (blocks, keys, parts): more blocks than SMs, short pieces and long ones; as many blocks as SMs
@pytest.mark.parametrize("head_dim,pairs", [(64, False), (80, True), (128, True), (192, False)])
def test_narrow_blocks_of_fused_decode_where_two_share_an_sm(head_dim, pairs):
    """At 192 two blocks of four warps take 250 KB, more than an SM has: they ran alone, with half the bytes on their way."""
    path = build.find_built("bfloat16", head_dim)
    if path is None:
        pytest.skip("not compiled yet")
    warps = ctypes.CDLL(str(path)).skv_attention_decode_fused_warps
    assert warps(192, 448, 1, 148) == warps(2 * 148, 4096, 1, 148) == (4 if pairs else 8)
    assert warps(148, 448, 1, 148) == 8 and warps(384, 1024, 1, 148) == 8


# (pairs, experts, inner size, the most rows an expert may have): spread over the experts, or perhaps all on a few of them
@pytest.mark.parametrize("step,serves", [((32, 8, 2048, 16), True), ((32, 8, 2048, 0), True), ((33, 8, 2048, 0), False), ((64, 64, 512, 16), True),
                                         ((256, 64, 2048, 0), True), ((256, 64, 2048, 128), False), ((68, 64, 2048, 17), False), ((4, 8, 2044, 2), False)])
def test_experts_of_few_pairs_and_few_tokens(step, serves):
    """128 tokens that all choose the same 2 of 64 experts were sixteen rounds over the same weights."""
    path = build.find_built("bfloat16", 64)
    if path is None:
        pytest.skip("not compiled yet")
    assert ctypes.CDLL(str(path)).skv_expert_few_serves(*step) == int(serves)


# (vocabulary, top-k, top-p): short rows, where passes over the row are faster, and long ones
@pytest.mark.parametrize("call,serves", [((1000, 20, 1.0), False), ((1000, 20, 0.9), True), ((1000, 200, 0.9), True), ((1000, 256, 0.95), False),
                                         ((2000, 200, 1.0), False), ((2200, 20, 1.0), True), ((32000, 256, 1.0), True), ((128256, 257, 0.9), False),
                                         ((128256, 0, 0.9), False), ((1, 1, 0.9), False), ((2, 2, 0.5), False)])
def test_rows_that_are_sampled_from_a_short_list(call, serves):
    path = build.find_built("bfloat16", 64)
    if path is None:
        pytest.skip("not compiled yet")
    vocab, top_k, top_p = call
    assert bool(ctypes.CDLL(str(path)).skv_sample_few_serves(vocab, top_k, ctypes.c_float(top_p))) == serves


def test_tensor_memory_is_touched_behind_a_fence():
    """What a barrier's phase tells of another thread's tensor-core work is ordered with this thread's accesses to tensor memory by a fence
    on every path between the two: not one inside a branch.  (A missing one shows in no result: program order has held so far.)"""
    text = re.sub(r"//[^\n]*", "", (build.CSRC / "attention_prefill_tc.cu").read_text().split("prefill_attention_tc_kernel(")[1])
    waits = 0
    for wait in re.finditer(r"a_wait\(bar\(", text):
        depth = 0
        for token in re.finditer(r"[{}]|tcgen05\.fence::after_thread_sync|a_wait\(|\ba_(?:ld|st|mma)\w*\(", text[wait.end():]):
            word = token.group()
            depth += (word == "{") - (word == "}")
            if word == "a_wait(" or (word.startswith("tcgen05") and depth <= 0):
                waits += word != "a_wait("
                break
            assert not re.match(r"a_(ld|st|mma)", word), text[wait.start():wait.end() + token.end()]
    assert waits >= 5                                   # scores, probabilities, the products' ends


@pytest.mark.gpu
def test_a_build_with_other_registers_leaves_prompts_to_the_other_kernel(tmp_path):
    """The tensor-memory prompt kernel's warpgroups share out the registers that a block is launched with.  Where the compiler gives it another
    number the library says that it has no such kernel, so that prompts go to the one without (nothing is launched here)."""
    from stratakv_b200.ops import kernels_for
    lib = kernels_for(torch.bfloat16, 64, verbose=False).lib
    assert lib.skv_has_attention_prefill_tc() == 1
    text = (build.CSRC / "attention_prefill_tc.cu").read_text()
    assert text.count("A_REGS = 128") == 1
    (tmp_path / "other.cu").write_text(text.replace("A_REGS = 128", "A_REGS = 120"))
    folder = build.find_built("bfloat16", 64).parent
    subprocess.run([build.find_nvcc(), *build.ARCH_FLAGS, *build.COMMON_FLAGS, "-shared", *build._defines("bfloat16", 64), f"-I{build.CSRC}",
                    str(tmp_path / "other.cu"), "-o", str(tmp_path / "other.so"), "-L", str(folder),
                    f"-l:{build.common_library_name('bfloat16')}", "-Xlinker", f"-rpath={folder}"], check=True)
    other = ctypes.CDLL(str(tmp_path / "other.so"))
    assert other.skv_has_attention_prefill_tc() == 0


# (rows, vocabulary, top-k): one row, as many as two blocks each leave SMs for, more; short rows; more than a shared list's top-k
@pytest.mark.parametrize("call,ranks", [((1, 128256, 40), 8), ((1, 128256, 80), 4), ((1, 128256, 128), 2), ((1, 128256, 129), 1), ((64, 128256, 40), 2),
                                        ((67, 128256, 40), 2), ((68, 128256, 40), 1), ((16, 128256, 40), 8), ((17, 128256, 40), 4), ((1, 23999, 1), 1), ((1, 24000, 1), 2),
                                        ((1, 128256, 0), 1)])
def test_blocks_that_share_a_row_of_logits(call, ranks):
    path = build.find_built("bfloat16", 64)
    if path is None:
        pytest.skip("not compiled yet")
    rows, vocab, top_k = call
    assert ctypes.CDLL(str(path)).skv_sample_few_ranks(rows, vocab, top_k, ctypes.c_float(0.95), 148) == ranks


# (query tiles, heads, table width, block size, window): few tiles over long tables, short tables, windows, more tiles
@pytest.mark.parametrize("call,splits", [((1, 32, 32, 64, 0), 4), ((1, 32, 31, 64, 0), 2), ((1, 32, 15, 64, 0), 1), ((1, 32, 128, 64, 700), 1), ((1, 32, 128, 64, 896), 2),
                                         ((1, 32, 128, 64, 1920), 4), ((4, 32, 128, 64, 0), 2), ((5, 32, 128, 64, 0), 1), ((2, 37, 128, 64, 0), 4), ((3, 25, 128, 64, 0), 2)])
def test_blocks_that_share_a_query_tiles_keys(call, splits):
    path = build.find_built("bfloat16", 64)
    if path is None:
        pytest.skip("not compiled yet")
    assert ctypes.CDLL(str(path)).skv_attention_prefill_tc_splits(*call, 148) == splits
