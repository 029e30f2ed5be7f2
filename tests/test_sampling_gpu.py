"""The sampling kernels against the distribution the reference's sampler draws from."""
import ctypes
import numpy as np
import pytest
import torch

import plain_llama

pytestmark = pytest.mark.gpu


def kernels():
    from stratakv_b200.ops import kernels_for
    return kernels_for(torch.float32, 64, verbose=False)


def draw(logits_row, n, temperature, top_k, top_p, seed=3):
    k = kernels()
    logits = torch.tensor(logits_row, dtype=torch.float32, device="cuda").repeat(n, 1).contiguous()
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    streams = torch.zeros(n, dtype=torch.int32, device="cuda")
    counters = torch.arange(n, dtype=torch.int32, device="cuda")
    k.sample(logits, out, temperature, top_k, top_p, seed, streams, counters)
    return out.cpu().numpy()


@pytest.mark.parametrize("temperature,top_k,top_p", [(1.0, 0, 1.0), (0.7, 5, 1.0), (1.3, 0, 0.8), (0.8, 40, 0.95),
                                                     (1.0, 1000, 0.999)])
def test_frequencies_match_the_reference_distribution(temperature, top_k, top_p):
    rng = np.random.default_rng(0)
    logits = (rng.standard_normal(331) * 2.0).astype(np.float32)
    expected = plain_llama.sample_reference(logits, temperature, top_k, top_p)
    n = 40000
    counts = np.bincount(draw(logits, n, temperature, top_k, top_p), minlength=331)
    assert counts[expected == 0].sum() == 0                   # nothing outside the kept set
    sigma = np.sqrt(n * expected * (1 - expected)) + 1.0
    assert (np.abs(counts - n * expected) < 5 * sigma).all()


def test_top_k_and_top_p_keep_what_the_reference_keeps():
    logits = np.log(np.array([0.5, 0.3, 0.15, 0.05], dtype=np.float32))
    assert set(draw(logits, 2000, 1.0, 2, 1.0)) == {0, 1}                 # tests/phase7_smoke.cpp:69-74
    assert set(draw(logits, 2000, 1.0, 0, 0.6)) == {0, 1}                 # the crossing token stays, :76-92
    assert set(draw(logits, 2000, 1.0, 0, 0.4)) == {0}
    assert set(draw(np.zeros(6, dtype=np.float32), 2000, 1.0, 2, 1.0)) == {0, 1}    # equal values: lower index first
    assert set(draw(logits, 200, 1.0, 1, 0.1)) == {0}


def test_draws_depend_on_seed_stream_and_counter_only():
    rng = np.random.default_rng(1)
    logits = torch.tensor(rng.standard_normal((6, 1000)), dtype=torch.float32, device="cuda")
    k = kernels()
    streams = torch.tensor([0, 1, 2, 3, 4, 5], dtype=torch.int32, device="cuda")
    counters = torch.tensor([9, 9, 9, 3, 3, 3], dtype=torch.int32, device="cuda")
    out = torch.zeros(6, dtype=torch.int32, device="cuda")
    k.sample(logits, out, 1.0, 0, 1.0, 11, streams, counters)
    first = out.clone()
    k.sample(logits, out, 1.0, 0, 1.0, 11, streams, counters)
    assert torch.equal(out, first)
    # a row alone gives the same token as in the batch
    one = torch.zeros(1, dtype=torch.int32, device="cuda")
    k.sample(logits[4:5].contiguous(), one, 1.0, 0, 1.0, 11, streams[4:5].contiguous(), counters[4:5].contiguous())
    assert int(one) == int(first[4])
    k.sample(logits, out, 1.0, 0, 1.0, 12, streams, counters)
    assert not torch.equal(out, first)


def test_non_finite_logits_raise_the_flag():
    k = kernels()
    logits = torch.zeros(2, 50, device="cuda")
    logits[1, 3] = float("inf")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(2, dtype=torch.int32, device="cuda")
    zeros = torch.zeros(2, dtype=torch.int32, device="cuda")
    k.sample(logits, out, 1.0, 0, 1.0, 0, zeros, zeros, flag)
    assert int(flag) & 2


def test_long_rows_and_ties_take_the_other_paths_of_the_kernel():
    """Rows longer than the kernel keeps in shared memory are read again on every walk; many equal values make the
    passes over the index bits run; a top-k above what the list of elements in play holds keeps it from being made."""
    vocab = 50000
    rng = np.random.default_rng(5)
    logits = (-30.0 + 0.01 * rng.standard_normal(vocab)).astype(np.float32)
    logits[[7, 31000, 49999]] = [3.0, 2.5, 2.0]
    n = 6000
    drawn = draw(logits, n, 1.0, 3, 1.0)
    assert set(drawn) == {7, 31000, 49999}
    expected = np.exp([3.0, 2.5, 2.0]) / np.exp([3.0, 2.5, 2.0]).sum()
    counts = np.array([(drawn == i).sum() for i in (7, 31000, 49999)])
    assert (np.abs(counts - n * expected) < 5 * np.sqrt(n * expected * (1 - expected))).all()
    assert set(draw(logits, 500, 1.0, 0, 0.3)) == {7}                    # its share is 0.51: it crosses 0.3 alone
    assert set(draw(logits, 2000, 1.0, 0, 0.6)) == {7, 31000}            # 0.51 + 0.31 crosses 0.6
    # all values equal: the k lowest indices stay, whatever k
    flat = np.zeros(vocab, dtype=np.float32)
    assert set(draw(flat, 3000, 1.0, 5, 1.0)) == {0, 1, 2, 3, 4}
    assert set(draw(flat, 400, 0.7, 1, 1.0)) == {0}
    # more survivors than the list of elements in play holds
    slope = (-1e-4 * np.arange(vocab)).astype(np.float32)
    many = draw(slope, 4000, 1.0, 6000, 1.0)
    assert many.max() < 6000 and many.min() < 300 and (many > 3000).sum() > 1000
    # and the same three tokens on a row that does fit
    short = logits[:32000].copy()
    short[[7, 31000, 31999]] = [3.0, 2.5, 2.0]
    assert set(draw(short, 3000, 1.0, 3, 1.0)) == {7, 31000, 31999}


@pytest.mark.parametrize("vocab,top_k,top_p", [(2, 1, 1.0), (37, 36, 0.9), (513, 40, 1.0), (160, 40, 0.9), (1000, 200, 0.9), (2401, 40, 1.0), (32000, 40, 0.95), (32001, 200, 0.9), (50257, 256, 0.5),
                                               (128256, 20, 0.95)])
@pytest.mark.parametrize("ties", [False, True])
def test_a_short_list_draws_what_the_whole_row_draws(vocab, top_k, top_p, ties):
    """A small top-k is chosen from a short list; a row whose other logits are sunk to where they weigh 2^-40 of the largest
    goes through every element of the row and must give the same tokens.  With ties more values equal the bound than the
    list holds in the long rows, and the lower indices win."""
    rng = np.random.default_rng(vocab + top_k)
    rows = 24
    logits = (rng.standard_normal((rows, vocab)) * 2).astype(np.float32)
    if ties:
        logits = np.round(logits)
    order = np.argsort(-logits, axis=1, kind="stable")
    sunk = np.full_like(logits, -1e4)
    kept = []
    for r in range(rows):
        probabilities = plain_llama.sample_reference(logits[r], 0.8, top_k, 1.0)
        cumulative = np.cumsum(probabilities[order[r]])
        if top_p < 1.0 and np.abs(cumulative - top_p).min() < 1e-5:
            continue                                       # the cut falls within rounding: either side is right
        count = min(top_k, int(np.searchsorted(cumulative, top_p)) + 1) if top_p < 1.0 else top_k
        sunk[r, order[r, :count]] = logits[r, order[r, :count]]
        kept.append(r)
    k, outs = kernels(), []
    streams = torch.arange(rows, dtype=torch.int32, device="cuda")
    for values, limit, mass in ((logits, top_k, top_p), (sunk, 0, 1.0)):
        out = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
        k.sample(torch.tensor(values, device="cuda"), out, 0.8, limit, mass, 5, streams, streams)
        outs.append(out.cpu().numpy())
    # (a drawn number falls within the 2^-40 x vocab of the sunk logits about once in 10^7 rows)
    assert kept and (outs[0][kept] == outs[1][kept]).all()


def test_a_short_list_flags_what_is_not_finite():
    k = kernels()
    for bad in (float("nan"), float("inf"), float("-inf"), 3e38):
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        logits = torch.zeros(2, 1001, device="cuda")
        logits[1, 777] = bad
        out = torch.full((2,), -1, dtype=torch.int32, device="cuda")
        zeros = torch.zeros(2, dtype=torch.int32, device="cuda")
        k.sample(logits, out, 0.5, 40, 0.9, 0, zeros, zeros, flag)      # (3e38 / 0.5 overflows)
        assert int(flag) == 2 and int(out[1]) == 0


@pytest.mark.parametrize("vocab", [5000, 32000, 128256])
@pytest.mark.parametrize("allowed", [3, 39, 41, 700])
def test_masked_rows_with_few_logits_left(vocab, allowed):
    """Fewer than top-k logits that are not the mask's: the others are equal, and the list cannot hold them."""
    rng = np.random.default_rng(vocab + allowed)
    rows = 8
    logits = np.full((rows, vocab), -1e30, dtype=np.float32)
    sunk = np.full((rows, vocab), -1e4, dtype=np.float32)
    for r in range(rows):
        places = rng.choice(vocab, allowed, replace=False)
        logits[r, places] = rng.standard_normal(allowed) * 2
        best = places[np.argsort(-logits[r, places], kind="stable")[:40]]
        sunk[r, best] = logits[r, best]
    k, outs = kernels(), []
    streams = torch.arange(rows, dtype=torch.int32, device="cuda")
    for values, limit in ((logits, 40), (sunk, 0)):
        out = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
        k.sample(torch.tensor(values, device="cuda"), out, 1.0, limit, 1.0, 9, streams, streams)
        outs.append(out.cpu().numpy())
    assert (outs[0] == outs[1]).all()


def test_two_blocks_of_the_kernel_share_an_sm():
    """More rows than SMs: with one block an SM they take half as long again."""
    assert kernels().lib.skv_sample_blocks_per_sm() >= 2


@pytest.mark.parametrize("vocab,top_k", [(24000, 1), (32000, 40), (50257, 40), (65539, 97), (128256, 40), (128256, 128)])
@pytest.mark.parametrize("kind", ["plain", "ties", "masked", "one_part"])
def test_blocks_that_share_a_row_draw_what_one_block_draws(vocab, top_k, kind):
    """A row of a small batch is walked by two, four or eight blocks, a row of a large one by one: the tokens are the same,
    whatever part the largest logits lie in, and a logit that is not finite is found in every part."""
    rng = np.random.default_rng(vocab + top_k)
    rows = 300
    logits = (rng.standard_normal((rows, vocab)) * 3).astype(np.float32)
    if kind == "ties":
        logits = np.round(logits * 8) / 8
    elif kind == "masked":
        logits[:, 100:] = -1e30
        logits[::2, -30:] = 1.0
    elif kind == "one_part":
        for r in range(rows):
            logits[r, (r * 997) % (vocab - 600):][:600] += 30.0
    k = kernels()
    streams = torch.arange(rows, dtype=torch.int32, device="cuda")
    device = torch.tensor(logits, device="cuda")

    def tokens(first, count):
        out = torch.full((count,), -1, dtype=torch.int32, device="cuda")
        k.sample(device[first:first + count], out, 0.9, top_k, 0.95, 7, streams[first:first + count], streams[first:first + count])
        return out

    whole = tokens(0, rows)
    ranks = lambda count: k.lib.skv_sample_few_ranks(count, vocab, top_k, ctypes.c_float(0.95), torch.cuda.get_device_properties(0).multi_processor_count)
    assert ranks(rows) == 1 and ranks(1) > 1 and ranks(60) > 1
    for count in (1, 3, 16, 17, 60, 130):
        assert torch.equal(tokens(rows - count, count), whole[rows - count:]), count
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    for place in (0, vocab // 2 - 1, vocab // 2 + 1, vocab - 1):
        row = device[:1].clone()
        row[0, place] = float("nan")
        out = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        flag.zero_()
        k.sample(row, out, 0.9, top_k, 0.95, 7, streams[:1], streams[:1], flag)
        assert int(flag) == 2 and int(out) == 0, place
