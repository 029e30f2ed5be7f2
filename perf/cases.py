"""The work this library is timed at: requests served through ``Engine.step`` and tokens chosen by ``Sampler``.

A served case is one batch of requests from its prompts to the logits of its last decoded token, as a serving program
drives the engine: open a sequence per request, run the prompts in one step (or in portions), then one step per new
token, then close the sequences.  The tokens fed are given, so that two implementations walk the same path; every
logit row that such a program looks at comes back.  The engine with its weights is what the program keeps; a state is
a batch of requests to it, made from the seed.  A sampling case is one choice of a token per row of logits.

The ranges (``draw``): the seven registered decoders, at the layer sizes of this repository's benchmark; bfloat16, and
float32 for small models; batches of 1 to 64; prompts of 16 to 8,192 tokens, whole or in portions, of one length or
ragged; 0 to 32 decoded tokens; sampling over 1 to 128 rows of 1,000 to 128,256 logits.
"""
import math
import random

import torch

from stratakv_b200 import Engine, EngineConfig, StepEntry, ops
from stratakv_b200.config.registry import resolve_architecture
from stratakv_b200.engine.model import expected_tensors
from stratakv_b200.sampling import Sampler, SamplingParams
from stratakv_b200.weights import random_tensors

# Layer sizes: TinyLlama's and Llama-3-8B's, one with a key head per query head, and Llama-2-7B's.
SIZES = {
    "2048": dict(hidden=2048, heads=32, kv_heads=4, head_dim=64, ff=5632, vocab=32000),
    "4096": dict(hidden=4096, heads=32, kv_heads=8, head_dim=128, ff=14336, vocab=128256),
    "3072": dict(hidden=3072, heads=24, kv_heads=24, head_dim=128, ff=8192, vocab=32000),
    "4096mha": dict(hidden=4096, heads=32, kv_heads=32, head_dim=128, ff=11008, vocab=32000),
}
KINDS = {"llama": ("attention",), "zepavik": ("attention",), "povusun": ("attention", "latent_attention", "rglru"),
         "kedelorn": ("retention", "latent_attention"), "fidolix": ("attention", "parallel"),
         "tobozen": ("attention", "mamba2", "lightning"), "vekanex": ("gla", "mlstm", "parallel")}
EPS = 1e-5


def served(name, model, size, layers, batch, prompt, new, portion=0, ragged=True, dtype="bfloat16"):
    return dict({"name": name} if name else {}, op="serve", model=model, size=size, layers=layers, dtype=dtype, batch=batch,
                prompt=prompt, ragged=ragged, portion=portion, new=new)


def listed():
    return [
        # one short question to the TinyLlama shape: launches and latency
        served("llama-chat-1", "llama", "2048", 22, 1, 33, 16),
        # the headline shape: eight requests of unequal length that are decoded together
        served("llama-serve-8", "llama", "2048", 22, 8, 1000, 32),
        # one long document in portions, then an answer
        served("llama-long-1", "llama", "2048", 22, 1, 8100, 16, portion=2048),
        # a full batch on layers of the Llama-3-8B shape with its vocabulary
        served("llama8b-batch-64", "llama", "4096", 8, 64, 512, 8),
        # the exact 32-bit path
        served("llama-float32", "llama", "2048", 4, 3, 250, 16, dtype="float32"),
        # the other decoders: all their kinds of layer, prompts and decoding, small and middle batches
        served("zepavik-serve-8", "zepavik", "3072", 4, 8, 511, 16),
        served("povusun-serve-8", "povusun", "2048", 6, 8, 600, 16),
        served("kedelorn-serve-8", "kedelorn", "2048", 4, 8, 777, 16),
        served("fidolix-serve-4", "fidolix", "2048", 4, 4, 1024, 16),
        served("tobozen-serve-16", "tobozen", "4096", 3, 16, 200, 16),
        served("vekanex-prompt-1", "vekanex", "2048", 3, 1, 2000, 24, ragged=False),
        # temperature, top-k and top-p over a batch's logits
        dict(name="sample-64", op="sample", rows=64, vocab=128256, temperature=0.8, top_k=40, top_p=0.95),
    ]


def draw(rng):
    if rng.random() < 0.1:
        return dict(op="sample", rows=round(2 ** rng.uniform(0, 7)), vocab=rng.choice((1000, 32000, 50257, 128256)),
                    temperature=rng.choice((0.6, 0.8, 1.0)), top_k=rng.choice((0, 0, 20, 40, 200)), top_p=rng.choice((1.0, 0.9, 0.95)))
    model = rng.choice(("llama",) * 4 + tuple(KINDS)[1:])
    dtype = "float32" if rng.random() < 0.1 else "bfloat16"
    size = rng.choice(("2048", "3072")) if dtype == "float32" else rng.choice(tuple(SIZES))
    kinds = len(KINDS[model])
    case = served("", model, size, kinds * rng.randint(1, 2) if kinds > 1 else rng.randint(1, 8),
                  max(1, round(2 ** rng.uniform(0, 6))), round(2 ** rng.uniform(4, 13)), rng.choice((0, 1, 4, 16, 32)),
                  rng.choice((0, 0, 512, 2048)), rng.random() < 0.7, dtype)
    while cost(case) > DRAWN_MOST or exact_seconds(case) > 12:
        case["batch" if case["batch"] > 1 and rng.random() < 0.5 else "prompt"] //= 2
    return case


# ---- the models ------------------------------------------------------------------------------------------------------

def model_dict(model, size, layers):
    """The ``config.json`` of a model, all its layers' kinds in turn."""
    s = SIZES[size]
    d, heads, kv, width, ff, vocab = s["head_dim"], s["heads"], s["kv_heads"], s["hidden"], s["ff"], s["vocab"]
    if model == "llama":
        return dict(architectures=["LlamaForCausalLM"], hidden_size=width, intermediate_size=ff, num_hidden_layers=layers,
                    num_attention_heads=heads, num_key_value_heads=kv, head_dim=d, vocab_size=vocab, rms_norm_eps=EPS,
                    rope_theta=10000.0, max_position_embeddings=8192 + 64, tie_word_embeddings=False, hidden_act="silu")
    vocab = 32000
    half, quarter, scale = ff // 2 // 64 * 64, ff // 4 // 64 * 64, d ** -0.5
    grouped = dict(heads=heads, kv_heads=kv, dim=d, vdim=d, scale=scale)
    stretched = {"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0}
    slow = [1.0 - 2.0 ** (-5.0 - 3.0 * h / max(heads - 1, 1)) for h in range(heads)]
    top2 = {"experts": 8, "top": 2}
    raw = dict(architecture=model.capitalize(), vocab=vocab, width=width, norm={"eps": EPS})
    mixers, mlp, first_mlp = {}, None, None
    if model == "zepavik":
        raw.update(max_positions=8192 + 64, logit_scale=1.0, embedding={"bigram": {"buckets": 65521, "mul_prev": 40503, "mul_cur": 9973}})
        mixers["attention"] = dict(grouped, mask={"size": 4096})
        mlp = {"kind": "dense", "ff": ff * 3 // 2}
    elif model == "povusun":
        raw.update(token_side={"dim": 32})
        mixers = {"attention": dict(grouped, softcap=30.0, q_temp={"coef": 0.1, "every": 512}),
                  "latent_attention": dict(heads=heads, dim=d, vdim=d, kv_rank=min(256, 4 * d), scale=scale),
                  "rglru": dict(width=width, blocks=heads, conv=4)}
        mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    elif model == "kedelorn":
        raw.update(streams=2)
        mixers = {"retention": dict(heads=heads, dim=d, vdim=d, rot={"dims": d, "base": 10000.0}, decay=slow),
                  "latent_attention": dict(heads=heads, dim=d - d // 4, rot_dim=d // 4, vdim=d, kv_rank=min(256, 4 * d), scale=scale,
                                           rot={"dims": d // 4, "base": 10000.0, "scaling": stretched})}
        mlp = {"kind": "moe", "expert": {"ff": half}, "router": dict(top2, scale=1.0), "shared": {"ff": half}}
    elif model == "fidolix":
        raw.update(embedding={"scale": 3.0}, token_side={"dim": 64})
        left = dict(grouped, conv=4, mask={"size": 1024}, rot={"dims": d, "base": 10000.0, "scaling": stretched})
        mixers = {"attention": dict(grouped, softcap=30.0),
                  "parallel": dict(left=left, right={"heads": heads, "dim": d, "rank": 64}, left_scale=0.8, right_scale=1.1)}
        mlp = {"kind": "moe", "expert": {"ff": half}, "router": dict(top2, groups={"count": 2, "keep": 1})}
        first_mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    elif model == "tobozen":
        raw["norm"]["groups"] = 2
        mixers = {"attention": dict(grouped, rot={"dims": d, "base": 10000.0}, v_mix=True),
                  "mamba2": dict(heads=2 * width // 64, vdim=64, state=128, groups=8, conv=4, norm_groups=8),
                  "lightning": dict(heads=heads, dim=d, vdim=d, decay=slow)}
        mlp = {"kind": "moe", "expert": {"ff": half, "limit": 7.0}, "router": top2}
    else:
        raw.update(residual_mult=0.7, logit_softcap=30.0)
        mixers = {"gla": dict(heads=heads, dim=d, vdim=d, tau=16.0, rank=16), "mlstm": dict(heads=heads, dim=d, vdim=d, gate_cap=15.0),
                  "parallel": dict(left=dict(grouped, rot={"dims": d, "base": 10000.0}),
                                   right=dict(heads=heads, kv_heads=heads, dim=d, vdim=d, conv=4, decay_rank=d, gate_rank=d),
                                   left_scale=0.8, right_scale=0.6)}
        mlp = {"kind": "moe", "expert": {"ff": quarter}, "router": top2, "shared": {"ff": half}}
    kinds = KINDS[model]
    made = [{"type": kinds[i % len(kinds)], "mixer": dict(mixers[kinds[i % len(kinds)]]),
             "mlp": first_mlp if i == 0 and first_mlp else mlp} for i in range(layers)]
    if model in ("povusun", "kedelorn") and layers == 2 * len(kinds):
        borrower = len(kinds) if model == "povusun" else 3          # the second layer of its kind reads the first one's cache
        made[borrower]["mixer"]["kv_from"] = borrower - len(kinds)
    return dict(raw, layers=made)


def spec_of(case):
    """(architecture's name, typed configuration, model description) of a case."""
    raw = model_dict(case["model"], case["size"], case["layers"])
    arch = resolve_architecture("LlamaForCausalLM" if case["model"] == "llama" else raw["architecture"])
    config = arch.config_class.from_dict(raw)
    return raw, config, arch.build_spec(config)


def is_output(name):
    return name.endswith(("o_proj.weight", "down_proj.weight", "mix.o", "left.o", "right.o", ".down"))


def weights_of(case):
    """Weights as a trained model has them in what matters here: projections that end in the stream are scaled by the
    number of layers, a token's own vector stays visible in the stream, and routers are decisive (an expert answers to a
    direction, and a token's vector leans towards two of them), so that rounding does not decide which experts run."""
    raw, _, spec = spec_of(case)
    dtype = getattr(torch, case["dtype"])
    P = random_tensors(expected_tensors(spec), seed=1, dtype=dtype, device="cuda")
    generator = torch.Generator(device="cuda").manual_seed(2)
    normal = lambda *shape: torch.randn(shape, generator=generator, device="cuda")
    width = SIZES[case["size"]]["hidden"]
    for name in P:
        if is_output(name):
            P[name] = (P[name].float() * (2 * case["layers"]) ** -0.5).to(dtype)
        elif name.endswith("mix.lam"):                      # decays of 0.9 to 0.999 at half-open gates
            P[name] = (normal(*P[name].shape) - 5.0).to(dtype)
        elif name in ("pos", "bigram", "side.embed"):
            P[name] = normal(*P[name].shape).mul_(0.5).to(dtype)
    table = "model.embed_tokens.weight" if case["model"] == "llama" else "embed"
    embed = normal(*P[table].shape)
    routers = [name for name in P if name.endswith("mlp.router")]
    if routers:
        direction = torch.nn.functional.normalize(normal(8, width), dim=-1)
        first = torch.arange(embed.shape[0], device="cuda") % 8
        second = first // 4 * 4 + (first + 1 + embed.shape[0] // 8 % 3) % 4          # of the same four experts
        embed += width ** 0.5 * (0.35 * direction[first] + 0.21 * direction[second])
        for name in routers:
            P[name] = (0.5 * direction + 0.002 * normal(8, width)).to(dtype)
    P[table] = embed.to(dtype)
    return P


# The program's engine: one model is loaded at a time.
_LOADED = {}


def engine_of(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _LOADED:
        _LOADED.clear()
        _, _, spec = spec_of(case)
        tokens = sum(-(-(n + case["new"]) // 64) * 64 for n in lengths(case))
        _LOADED[key] = Engine(spec, weights_of(case), EngineConfig(max_tokens=tokens, dtype=case["dtype"], max_batch=case["batch"],
                                                                   max_context=8192 + 64), verbose=False)
    return _LOADED[key]


def vocab_of(case):
    return SIZES[case["size"]]["vocab"] if case["model"] == "llama" else 32000


def lengths(case):
    """The prompts' lengths: all ``prompt``, or spread between half of it and it."""
    n, spread = case["prompt"], max(1, case["prompt"] // 2)
    return [max(1, n - (i * 37) % spread) if case["ragged"] else n for i in range(case["batch"])]


def tokens_of(case, seed):
    """The prompts and, per decode step, the token each request is fed."""
    rng = random.Random(seed)
    vocab = vocab_of(case)
    prompts = [[rng.randrange(vocab) for _ in range(n)] for n in lengths(case)]
    return prompts, [[rng.randrange(vocab) for _ in prompts] for _ in range(case["new"])]


def prepare(case, seed):
    if case["op"] == "sample":
        generator = torch.Generator(device="cuda").manual_seed(seed)
        logits = 2.0 * torch.randn(case["rows"], case["vocab"], generator=generator, device="cuda")
        params = SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=seed)
        flags = torch.zeros(1, dtype=torch.int32, device="cuda")
        rows = torch.arange(case["rows"], dtype=torch.int32, device="cuda")
        return dict(sampler=Sampler(ops.kernels_for(torch.bfloat16, 64), params, flags), logits=logits, streams=rows, counters=rows % 7)
    prompts, fed = tokens_of(case, seed)
    portion = case["portion"] or max(map(len, prompts))
    return dict(engine=engine_of(case), prompts=prompts, fed=fed, portion=portion)


def run(state):
    if "sampler" in state:
        return state["sampler"].sample(state["logits"], state["streams"], state["counters"])
    engine, prompts, portion = state["engine"], state["prompts"], state["portion"]
    slots = [engine.open_sequence() for _ in prompts]
    first = [None] * len(prompts)
    for start in range(0, max(map(len, prompts)), portion):
        entries, ends = [], []
        for i, prompt in enumerate(prompts):
            part = prompt[start:start + portion]
            if part:
                last = start + portion >= len(prompt)
                entries.append(StepEntry(slots[i], part, [len(part) - 1] if last else []))
                ends += [i] * last
        logits = engine.step(entries)
        if ends:
            logits = logits.clone()
        for row, i in enumerate(ends):
            first[i] = logits[row]
    decoded = [engine.step([StepEntry(slot, [token], [0]) for slot, token in zip(slots, fed)]).clone() for fed in state["fed"]]
    for slot in slots:
        engine.close_sequence(slot)
    return [torch.stack(first)] + ([torch.stack(decoded)] if decoded else [])


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def work(case):
    if case["op"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"] + 12.0 * case["rows"], "flops": 4.0 * case["rows"] * case["vocab"]}
    raw, _, spec = spec_of(case)
    size, counts = SIZES[case["size"]], lengths(case)
    width, item = size["hidden"], 4 if case["dtype"] == "float32" else 2
    layers = raw.get("layers") or [{"type": "attention", "mixer": dict(heads=size["heads"], kv_heads=size["kv_heads"],
                                                                       dim=size["head_dim"], vdim=size["head_dim"])}] * case["layers"]
    dense = experts = head = 0
    for name, request in expected_tensors(spec).items():
        n = math.prod(request.shape)
        if name in ("lm_head.weight", "head") or (name == "embed" and case["model"] in ("povusun", "tobozen")):
            head += n
        elif ".mlp.e" in name:
            experts += n
        elif "embed" not in name and name not in ("pos", "bigram"):
            dense += n
    steps = [[n for n in counts]] + [[1] * len(counts)] * case["new"]
    total_bytes = total_flops = 0.0
    for step, news in enumerate(steps):
        tokens = sum(news)
        context = [n + step for n in counts]
        # weights once a step (of the experts, as many as the step's tokens can choose), the embedding rows, the logits
        total_bytes += item * (dense + head + experts * min(1.0, 2 * tokens / 8) + tokens * width) + 4.0 * vocab_of(case) * len(counts)
        total_flops += 2.0 * (dense + experts / 4) * tokens + 2.0 * head * len(counts)
        for layer in layers:
            for m in ([layer["mixer"]] if layer["type"] != "parallel" else [layer["mixer"]["left"], layer["mixer"]["right"]]):
                if "scale" in m or case["model"] == "llama":                   # softmax attention over the context
                    kept = m["kv_rank"] + m.get("rot_dim", 0) if "kv_rank" in m else m["kv_heads"] * (m["dim"] + m["vdim"])
                    window = (m.get("mask") or {}).get("size", 1 << 30)
                    total_bytes += item * kept * sum(min(c, window) + q for c, q in zip(context, news))
                    total_flops += 2.0 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"]) * sum(
                        q * min(window, c - (q - 1) / 2) for c, q in zip(context, news))
                elif "blocks" not in m:                                        # a matrix state per head
                    state = m["heads"] * m.get("state", m.get("dim", 0)) * m.get("vdim", m.get("dim", 0))
                    total_bytes += 8.0 * state * len(counts)
                    total_flops += 4.0 * state * tokens
    return {"bytes": total_bytes, "flops": total_flops}


def cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / (50 if case.get("dtype") != "float32" else 2))


DRAWN_MOST = 0.5 * cost(listed()[3])


def tolerance(case):
    """Four times what the engine's logits are off from ``exact``: 1.2e-6 in float32, 0.002 to 0.005 in bfloat16 (up to 0.006 where
    every branch is normed again before it joins the stream)."""
    if case["op"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.025 if case["model"] in ("povusun", "vekanex") else 0.02}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------

def exact_seconds(case):
    """About how long ``exact`` takes: arithmetic, and a few launches per token of a recurrent layer."""
    if case["op"] == "sample":
        return 0.0
    recurrent = sum(kind in ("rglru", "retention", "mamba2", "lightning", "gla", "mlstm", "parallel")
                    for kind in KINDS[case["model"]]) * case["layers"] / len(KINDS[case["model"]])
    return work(case)["flops"] / 15e12 + recurrent * 1.5e-4 * sum(n + case["new"] for n in lengths(case))


def exact(case, seed):
    """Plain torch in float64 on the very same weights and tokens: whole sequences, no cache, one after the other."""
    if case["op"] == "sample" or exact_seconds(case) > 25:
        return None
    raw = model_dict(case["model"], case["size"], case["layers"])
    P = Doubles(weights_of(case))
    prompts, fed = tokens_of(case, seed)
    rows = []
    for i, prompt in enumerate(prompts):
        tokens = torch.tensor(prompt + [step[i] for step in fed], device="cuda")
        x = (llama_stream if case["model"] == "llama" else decoder_stream)(raw, P, tokens)[len(prompt) - 1:]
        rows.append(logits(raw, P, x))
    rows = torch.stack(rows, dim=1)                                            # [1 + new, batch, vocab]
    return [rows[0]] + ([rows[1:]] if case["new"] else [])


class Doubles(dict):
    """Weights that widen when they are read."""

    def __getitem__(self, name):
        return super().__getitem__(name).double()


def unit(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def grouped_norm(x, weight, groups=1, eps=EPS):
    return unit(x.reshape(*x.shape[:-1], groups, -1), eps).reshape(x.shape) * weight


def silu(z):
    return z * torch.sigmoid(z)


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


softplus = torch.nn.functional.softplus


def rotate(x, rot, interleaved=False):
    """The first rot.dims numbers of every head: halves against each other, or neighbours."""
    dims, base, magnitude = rot["dims"], rot["base"], 1.0
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    f = base ** (-2.0 * i / dims)
    if rot.get("scaling"):
        s = rot["scaling"]
        pair = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, magnitude = f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0
    angle = torch.arange(x.shape[0], device=x.device).double()[:, None] * f
    shape = (x.shape[0],) + (1,) * (x.dim() - 2) + (dims // 2,)
    cos, sin = (angle.cos() * magnitude).view(shape), (angle.sin() * magnitude).view(shape)
    out = x.clone()
    u, v = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., u], out[..., v] = x[..., u] * cos - x[..., v] * sin, x[..., v] * cos + x[..., u] * sin
    return out


def attend(q, k, v, scale, cap=0.0, window=0, sink=None, penalty=None):
    """Causal softmax attention; ``sink`` per head counts in the denominator; ``penalty(head, distance)`` leaves the scores."""
    T, H = q.shape[:2]
    distance = torch.arange(T, device=q.device)[:, None] - torch.arange(T, device=q.device)
    hidden = (distance < 0) | (distance >= (window or T))
    out = q.new_zeros(T, H, v.shape[2])
    for h in range(H):
        g = h * k.shape[1] // H
        scores = (q[:, h] @ k[:, g].T).mul_(scale)
        scores = cap * torch.tanh(scores / cap) if cap else scores
        scores = scores - penalty(h, distance.clamp(min=0)) if penalty else scores
        scores.masked_fill_(hidden, -math.inf)
        if sink is not None:
            scores = torch.cat([scores, sink[h].expand(T, 1)], dim=1)
        out[:, h] = torch.softmax(scores, dim=-1)[:, :T] @ v[:, g]
    return out


def convolve(u, taps):
    """Causal short convolution, a filter per channel; the last tap weighs the token itself."""
    padded = torch.cat([u.new_zeros(taps.shape[1] - 1, u.shape[1]), u])
    return sum(padded[j:j + u.shape[0]] * taps[:, j] for j in range(taps.shape[1]))


def memory(q, k, v, decay, beta=None, bonus=None):
    """S_t = decay_t S_(t-1) + k_t v_t^T, o_t = S_t^T q_t; ``beta``: what S says about the key is taken off the value first
    (the delta rule); ``bonus``: o_t reads S_(t-1) and the token itself by this weight per key channel."""
    T, H, n = k.shape
    S, out = k.new_zeros(H, n, v.shape[2]), k.new_zeros(T, H, v.shape[2])
    for t in range(T):
        kt, vt, before = k[t][:, :, None], v[t][:, None, :], S
        S = decay[t].view(H, -1, 1) * S
        if beta is not None:
            vt = beta[t][:, None, None] * (vt - kt.transpose(1, 2) @ S)
        S = S + kt * vt
        read = S if bonus is None else before + bonus[:, :, None] * kt * vt
        out[t] = (q[t][:, None, :] @ read)[:, 0]
    return out


def llama_stream(c, P, tokens):
    T, H, G, d = len(tokens), c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    x, rot = P["model.embed_tokens.weight"][tokens], {"dims": d, "base": c["rope_theta"]}
    for i in range(c["num_hidden_layers"]):
        w = lambda name: P["model.layers.%d.%s.weight" % (i, name)]
        h = unit(x) * w("input_layernorm")
        q, k, v = (h @ w("self_attn.%s_proj" % s).T for s in "qkv")
        o = attend(rotate(q.view(T, H, d), rot), rotate(k.view(T, G, d), rot), v.view(T, G, d), d ** -0.5)
        x = x + o.reshape(T, -1) @ w("self_attn.o_proj").T
        h = unit(x) * w("post_attention_layernorm")
        x = x + (silu(h @ w("mlp.gate_proj").T) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
    return x


def logits(c, P, x):
    if "architecture" not in c:
        return (unit(x) * P["model.norm.weight"]) @ P["lm_head.weight"].T
    name = c["architecture"]
    weight = P["final.norm"] + (1.0 if name == "Kedelorn" else 0.0)
    y = grouped_norm(x, weight, c["norm"].get("groups", 1)) @ P["embed" if name in ("Povusun", "Tobozen") else "head"].T
    cap = c.get("logit_softcap")
    return cap * torch.tanh(y / cap) if cap else y * c.get("logit_scale", 1.0)


def grouped_attention(name, h, P, p, m, kept, i):
    """The attention layers of Zepavik, Povusun, Fidolix and Tobozen."""
    T, H, G, d = len(h), m["heads"], m["kv_heads"], m["dim"]
    bias = name in ("Zepavik", "Fidolix")
    project = lambda s: h @ P[p + s].T + (P[p + s + ".b"] if bias else 0.0)
    q, (k, v) = project("q"), kept[m["kv_from"]] if "kv_from" in m else (project("k"), project("v"))
    if name in ("Fidolix", "Tobozen"):
        q, k = unit(q) * P[p + "q.norm"], unit(k) * P[p + "k.norm"]
    q, k, v, penalty, sink = q.view(T, H, d), k.view(T, G, d), v.view(T, G, -1), None, None
    if name == "Zepavik":
        r1, r2, v = P[p + "r1"], P[p + "r2"], unit(v)
        penalty = lambda head, distance: r1[head] * torch.log1p(r2[head] * distance)
    elif name == "Povusun":
        kept[i] = k, v
        q, k = unit(q), unit(k)
        steps = (torch.arange(T, device=h.device) + 1) // m["q_temp"]["every"]
        q = q * (1.0 + m["q_temp"]["coef"] * torch.log(steps.double() + 1.0))[:, None, None]
    elif name == "Tobozen":
        q, k, sink = rotate(q, m["rot"], True), rotate(k, m["rot"], True), h.new_zeros(H)
        own, v = v, (1.0 - P[p + "vmix"]) * v + P[p + "vmix"] * kept["values"] if "values" in kept else v
        kept.setdefault("values", own)
    out = attend(q, k, v, m["scale"], m.get("softcap", 0.0), (m.get("mask") or {}).get("size", 0), sink, penalty)
    if name == "Zepavik":
        out = out * torch.sigmoid(h @ P[p + "g"].T)[:, :, None]
    out = out.reshape(T, -1)
    return (out * torch.sigmoid(h @ P[p + "g"].T) if name in ("Povusun", "Fidolix") else out) @ P[p + "o"].T


def latent_attention(h, P, p, m, kept, i):
    T, H, d, rank = len(h), m["heads"], m["dim"], m["kv_rank"]
    turned = m.get("rot_dim", 0)
    if "kv_from" in m:
        c, k_rot = kept[m["kv_from"]]
    else:
        down = h @ P[p + "dkv"].T
        c, k_rot = unit(down[:, :rank]) * P[p + "dkv.norm"], rotate(down[:, rank:], m["rot"]) if turned else None
    kept[i] = c, k_rot
    q, k = (h @ P[p + "q"].T).view(T, H, d + turned), (c @ P[p + "uk"].T).view(T, H, d)
    v = (c @ P[p + "uv"].T).view(T, H, m["vdim"])
    if turned:
        q = torch.cat([q[..., :d], rotate(q[..., d:], m["rot"])], dim=-1)
        k = torch.cat([k, k_rot[:, None, :].expand(T, H, turned)], dim=-1)
    out = attend(q, k, v, m["scale"], sink=P[p + "sink"] if turned else None)
    if turned:
        out = out * torch.sigmoid(h @ P[p + "g"].T)[:, :, None]
    return out.reshape(T, -1) @ P[p + "o"].T


def rglru(h, P, p, m):
    T, blocks = len(h), m["blocks"]
    u = convolve(h @ P[p + "x"].T + P[p + "x.b"], P[p + "conv"]) + P[p + "conv.b"]
    gate = lambda s: torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(T, blocks, -1), P[p + s]) + P[p + s + ".b"]).reshape(T, -1)
    a = torch.exp(-8.0 * gate("ra") * softplus(P[p + "lam"]))
    driven, state, states = torch.sqrt(1.0 - a * a) * gate("ri") * u, h.new_zeros(m["width"]), []
    for t in range(T):
        state = a[t] * state + driven[t]
        states.append(state)
    return (torch.stack(states) * gelu(h @ P[p + "y"].T + P[p + "y.b"])) @ P[p + "o"].T


def heads_of(h, P, p, m, names="qkv"):
    return [(h @ P[p + s].T).view(len(h), m["heads"], -1) for s in names]


def retention(h, P, p, m):
    q, k, v = heads_of(h, P, p, m)
    decay = torch.tensor(m["decay"], dtype=torch.float64, device=h.device).expand(len(h), -1)
    o = unit(memory(rotate(q, m["rot"]), rotate(k, m["rot"]) * m["dim"] ** -0.5, v, decay)).reshape(len(h), -1)
    return (o * silu(h @ P[p + "g"].T)) @ P[p + "o"].T


def lightning(h, P, p, m):
    q, k, v = (silu(z) for z in heads_of(h, P, p, m))
    decay = torch.tensor(m["decay"], dtype=torch.float64, device=h.device).expand(len(h), -1)
    o = unit(memory(q, k, v, decay).reshape(len(h), -1)) * P[p + "norm"]
    return (o * torch.sigmoid(h @ P[p + "g"].T)) @ P[p + "o"].T


def mamba2(h, P, p, m):
    T, H, dv, N, G = len(h), m["heads"], m["vdim"], m["state"], m["groups"]
    z, xbc, dt = (h @ P[p + "in"].T).split([H * dv, H * dv + 2 * G * N, H], dim=1)
    x, B, C = silu(convolve(xbc, P[p + "conv"]) + P[p + "conv.b"]).split([H * dv, G * N, G * N], dim=1)
    dt, x = softplus(dt + P[p + "dt_bias"]), x.view(T, H, dv)
    spread = lambda y: y.reshape(T, G, N).repeat_interleave(H // G, dim=1)
    y = memory(spread(C), dt[:, :, None] * spread(B), x, torch.exp(-torch.exp(P[p + "A_log"]) * dt)) + P[p + "D"][:, None] * x
    return grouped_norm(y.reshape(T, -1) * silu(z), P[p + "norm"], m["norm_groups"]) @ P[p + "o"].T


def fidolix_pair(h, P, p, m):
    T, left, right = len(h), m["left"], m["right"]
    w = lambda s: P[p + "left." + s]
    q, k = (convolve(h @ w(s).T + w(s + ".b"), w(s + ".conv")) for s in "qk")
    q, k = q.view(T, left["heads"], -1), k.view(T, left["kv_heads"], -1)
    o = attend(rotate(q, left["rot"], True), rotate(k, left["rot"], True), k, left["scale"], window=left["mask"]["size"], sink=w("sink"))
    one = o.reshape(T, -1) @ w("o").T
    w = lambda s: P[p + "right." + s]
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    mix = {s: h + (before - h) * w("mu." + s) for s in "rkvgw"}
    r, k, v = ((mix[s] @ w(s).T).view(T, right["heads"], -1) for s in "rkv")
    decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w("w1").T) @ w("w2").T + w("w0")))
    o = unit(memory(r, k, v, decay, bonus=w("u").view(right["heads"], -1))).reshape(T, -1)
    return m["left_scale"] * one + m["right_scale"] * ((o * w("norm") * silu(mix["g"] @ w("g").T)) @ w("o").T)


def gla(h, P, p, m):
    q, k, v = heads_of(h, P, p, m)
    decay = torch.exp(torch.nn.functional.logsigmoid((h @ P[p + "a1"].T) @ P[p + "a2"].T + P[p + "a2.b"]) / m["tau"])
    o = (unit(memory(q * m["dim"] ** -0.5, k, v, decay)) * P[p + "norm"]).reshape(len(h), -1)
    return (o * silu(h @ P[p + "g"].T)) @ P[p + "o"].T


def mlstm(h, P, p, m):
    T, H, cap = len(h), m["heads"], m["gate_cap"]
    q, k, v = heads_of(h, P, p, m)
    capped = lambda s: cap * torch.tanh((h @ P[p + s].T + P[p + s + ".b"]) / cap)
    i, f, q = capped("i"), torch.nn.functional.logsigmoid(capped("f")), q * m["dim"] ** -0.5
    v = torch.cat([v, v.new_ones(T, H, 1)], dim=-1)                          # the last column sums the keys
    top, tops = h.new_zeros(H), []
    for t in range(T):
        top = torch.maximum(f[t] + top, i[t])
        tops.append(top)
    tops = torch.stack(tops)
    decay = torch.exp(f + torch.cat([torch.zeros_like(tops[:1]), tops[:-1]]) - tops)
    o = memory(q, torch.exp(i - tops)[:, :, None] * k, v, decay)
    o = o[..., :-1] / (torch.maximum(o[..., -1].abs(), torch.exp(-tops)) + 1e-6)[..., None]
    return (unit(o).reshape(T, -1) * P[p + "norm"] * torch.sigmoid(h @ P[p + "g"].T)) @ P[p + "o"].T


def vekanex_pair(h, P, p, m):
    T, left, right = len(h), m["left"], m["right"]
    w = lambda s: P[p + "left." + s]
    q, k, v = (h @ w(s).T + w(s + ".b") for s in "qkv")
    q, k = (unit(q) * w("q.norm")).view(T, left["heads"], -1), (unit(k) * w("k.norm")).view(T, left["kv_heads"], -1)
    o = attend(rotate(q, left["rot"]), rotate(k, left["rot"]), v.view(T, left["kv_heads"], -1), left["scale"])
    one = o.reshape(T, -1) @ w("o").T + w("o.b")
    w = lambda s: P[p + "right." + s]
    q, k, v = (silu(convolve(h @ w(s).T, w(s + ".conv"))).view(T, right["heads"], -1) for s in "qkv")
    q, k = (z / torch.sqrt((z * z).sum(dim=-1, keepdim=True) + 1e-6) for z in (q, k))
    step = softplus((h @ w("a1").T) @ w("a2").T + w("dt_bias")).view(T, right["heads"], -1)
    o = memory(q * right["dim"] ** -0.5, k, v, torch.exp(-torch.exp(w("A_log"))[:, None] * step), beta=torch.sigmoid(h @ w("b").T))
    o = (unit(o) * w("norm")).reshape(T, -1) * torch.sigmoid((h @ w("g1").T) @ w("g2").T)
    return m["left_scale"] * one + m["right_scale"] * (o @ w("o").T)


def feed_forward(name, h, P, p, m):
    clamped = lambda g, u, limit: g.clamp(max=limit) * torch.sigmoid(1.702 * g.clamp(max=limit)) * (u.clamp(-limit, limit) + 1.0)
    if m["kind"] == "dense":
        if name == "Zepavik":
            return torch.relu(h @ P[p + "up"].T) ** 2 @ P[p + "down"].T
        return clamped(h @ P[p + "gate"].T, h @ P[p + "up"].T, m["limit"]) @ P[p + "down"].T

    def expert(x, q):
        if name == "Kedelorn":
            return torch.relu(x @ P[q + "up"].T) ** 2 @ P[q + "down"].T
        g, u = x @ P[q + "gate"].T, x @ P[q + "up"].T
        return (clamped(g, u, m["expert"]["limit"]) if name == "Tobozen" else silu(g) * u) @ P[q + "down"].T

    z = h @ P[p + "router"].T
    if name == "Kedelorn":
        scores = torch.sigmoid(z)
        chosen = (scores + P[p + "correction"]).topk(2, dim=-1).indices
        share = scores.gather(1, chosen)
    elif name == "Fidolix":
        scores = torch.softmax(z, dim=-1).view(-1, 2, 4)
        best = scores.max(dim=-1).values
        scores = torch.where((best == best.max(dim=-1, keepdim=True).values)[:, :, None], scores, -1.0).view(-1, 8)
        share, chosen = scores.topk(2, dim=-1)
        share = share / (share.sum(dim=-1, keepdim=True) + 1e-20)
    else:
        share, chosen = z.topk(2, dim=-1)
        share = torch.sigmoid(share) if name == "Tobozen" else torch.softmax(share, dim=-1)
    y = torch.zeros_like(h)
    for e in range(8):
        t, c = torch.nonzero(chosen == e, as_tuple=True)
        if len(t):
            s = share[t, c][:, None]
            q = "%se%d." % (p, e)
            y.index_add_(0, t, expert(s * h[t], q) if name == "Tobozen" else s * expert(h[t], q))
    if m.get("shared"):
        shared = expert(h, p + "shared.")
        y = y + (torch.sigmoid(h @ P[p + "shared.sg"].T) * shared if name == "Kedelorn" else shared)
    return y


def decoder_stream(c, P, tokens):
    """The stream after the last layer of any decoder but Llama."""
    name, eps, groups = c["architecture"], c["norm"]["eps"], c["norm"].get("groups", 1)
    x, kept = P["embed"][tokens] * (c.get("embedding") or {}).get("scale", 1.0), {}
    if name == "Zepavik":
        pair = c["embedding"]["bigram"]
        rows = (tokens[:-1] * pair["mul_prev"] + tokens[1:] * pair["mul_cur"]) % pair["buckets"]
        x = x + P["bigram"][torch.cat([rows.new_tensor([pair["buckets"]]), rows])] + P["pos"][:len(tokens)]
    streams = x[None].repeat(c.get("streams", 1), 1, 1)
    for i, layer in enumerate(c["layers"]):
        p, m, kind = "l%d." % i, layer["mixer"], layer["type"]
        norm = lambda x, s: grouped_norm(x, P[p + s] + (1.0 if name == "Kedelorn" else 0.0), groups, eps)

        def mixer(h):
            q = p + "mix."
            if kind == "attention":
                return grouped_attention(name, h, P, q, m, kept, i)
            if kind == "latent_attention":
                return latent_attention(h, P, q, m, kept, i)
            pair = vekanex_pair if name == "Vekanex" else fidolix_pair
            return dict(rglru=rglru, retention=retention, lightning=lightning, mamba2=mamba2, gla=gla, mlstm=mlstm, parallel=pair)[kind](h, P, q, m)

        ffn = lambda h: feed_forward(name, h, P, p + "mlp.", layer["mlp"])
        if name == "Zepavik":
            h = norm(x, "norm1")
            x = x + mixer(h) + ffn(h)
        elif name == "Povusun":
            x = x + norm(mixer(norm(x, "norm1")), "norm1b")
            x = x + norm(ffn(norm(x, "norm2")), "norm2b")
        elif name == "Kedelorn":
            for s, sub in (("1", mixer), ("2", ffn)):
                y = sub(norm(torch.einsum("s,stw->tw", P[p + "hc" + s + ".in"], streams), "norm" + s))
                streams = torch.einsum("sr,stw->rtw", P[p + "hc" + s + ".mix"], streams) + P[p + "hc" + s + ".out"][:, None, None] * y
            x = streams.sum(dim=0)
        elif name == "Fidolix":
            x = x + mixer(norm(x, "norm1")) + ffn(norm(x, "norm2"))
        elif name == "Tobozen":
            x = x + mixer(norm(x, "norm1"))
            x = x + ffn(norm(x, "norm2"))
        else:
            x = x + c["residual_mult"] * norm(mixer(x), "norm1")
            x = x + c["residual_mult"] * norm(ffn(x), "norm2")
        if c.get("token_side"):
            dim = c["token_side"]["dim"]
            e = P["side.embed"][tokens][:, i * dim:(i + 1) * dim]
            x = x + unit((gelu(x @ P[p + "side.gate"].T) * e) @ P[p + "side.proj"].T) * P[p + "side.norm"]
    return x
