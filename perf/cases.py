"""The work whose speed counts: requests as a user's program hands them to an `Engine`, from the smallest to the largest.

A pass is one batch of requests from beginning to end: slots are taken, all prompts run in one step, then come `steps`
single tokens for every sequence, in two-turn requests a follow-up of `turn` tokens and `steps` further single tokens,
and the slots are given back.  The tokens are given (the next token of a sequence does not hang on a rounding of its
logits), and every logit that a sampler would have read is an output.  One case goes through `generate_token_ids`.

Models are of the shapes of this repository's benchmark and tests: Qwen3 of 8B and 14B shape (in full depth or with
fewer of their equal layers), the small 32-bit model of the tests, and the Fagunex models of the design benchmark
(latent attention, a gated recurrence, routed experts with a shared one) for the parts that Qwen3 does not have.
"""
import math
import random
import zlib

import numpy as np
import torch

import qwen3_b200 as q

VOCAB = 151936
QWEN3 = {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "hidden_act": "silu", "torch_dtype": "bfloat16",
         "num_hidden_layers": 36, "hidden_size": 4096, "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 128,
         "intermediate_size": 12288, "vocab_size": VOCAB, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6,
         "tie_word_embeddings": False, "max_position_embeddings": 40960, "attention_bias": False,
         "use_sliding_window": False, "sliding_window": None, "rope_scaling": None, "bos_token_id": 1, "eos_token_id": 2}
MODELS = {
    "8b": QWEN3,
    "14b": dict(QWEN3, hidden_size=5120, num_attention_heads=40, intermediate_size=17408),
    "tiny": dict(QWEN3, hidden_size=96, num_attention_heads=8, num_key_value_heads=1, head_dim=32, intermediate_size=160,
                 vocab_size=384, rms_norm_eps=1e-5, max_position_embeddings=256),
}
FAGUNEX_WIDTHS = {"fagunex-2k": (2048, 8192), "fagunex-4k": (4096, 12288)}
FAGUNEX_VOCAB, EXPERTS, TOP, HEAD, SIDE = 32768, 16, 2, 128, 64
ROUTED_BY = 32             # columns of the hidden state that the routers read (see `_fagunex_weights`)


def listed():
    return [
        # a unit-test-sized model in 32-bit, sampled at a temperature: the smallest calls, latency alone
        {"name": "tiny_generate", "model": "tiny", "layers": 3, "dtype": "float32", "lengths": "1,9,33,64", "steps": 12,
         "turn": 0, "want": "sampled"},
        # one person's chat, two turns of it: latency of a single sequence
        {"name": "chat_two_turns", "model": "8b", "layers": 36, "dtype": "bfloat16", "lengths": "217", "steps": 24, "turn": 45,
         "want": "last"},
        # the benchmark's decode: 8 sequences of unequal context of thousands of tokens
        {"name": "decode_8_long", "model": "8b", "layers": 36, "dtype": "bfloat16",
         "lengths": "4000,3241,3017,3733,3100,3500,3999,3368", "steps": 64, "turn": 0, "want": "last"},
        # a busy server: 64 short requests that decode together
        {"name": "decode_64", "model": "8b", "layers": 36, "dtype": "bfloat16", "lengths": _ragged(64, 16, 200), "steps": 24,
         "turn": 0, "want": "last"},
        # time to the first token of one prompt of the benchmark's size
        {"name": "prompt_2048", "model": "8b", "layers": 36, "dtype": "bfloat16", "lengths": "2048", "steps": 0, "turn": 0,
         "want": "last"},
        # a handful of short prompts of unequal length that start together
        {"name": "prompts_short", "model": "8b", "layers": 36, "dtype": "bfloat16", "lengths": "33,261,8,130,95", "steps": 0,
         "turn": 0, "want": "last"},
        # scoring a text: the logits of every position
        {"name": "score_700", "model": "8b", "layers": 12, "dtype": "bfloat16", "lengths": "700", "steps": 0, "turn": 0,
         "want": "all"},
        # a long document and an answer about it
        {"name": "document_24k", "model": "8b", "layers": 9, "dtype": "bfloat16", "lengths": "24571", "steps": 48, "turn": 0,
         "want": "last"},
        # the larger shape, 16 sequences (10 of its 40 layers)
        {"name": "decode_16_14b", "model": "14b", "layers": 10, "dtype": "bfloat16", "lengths": _ragged(16, 256, 1500),
         "steps": 48, "turn": 0, "want": "last"},
        # the 32-bit check path at full width: prompts, then single tokens
        {"name": "float32_check", "model": "8b", "layers": 4, "dtype": "float32", "lengths": "141,37,5", "steps": 16, "turn": 0,
         "want": "last"},
        # prompts through routed experts, latent attention and the recurrence
        {"name": "routed_prompts", "model": "fagunex-4k", "layers": 4, "dtype": "bfloat16", "lengths": "2048,911,1203",
         "steps": 0, "turn": 0, "want": "last"},
        # single tokens of 8 sequences through the same
        {"name": "routed_decode_8", "model": "fagunex-2k", "layers": 4, "dtype": "bfloat16", "lengths": _ragged(8, 64, 700),
         "steps": 96, "turn": 0, "want": "last"},
    ]


def draw(rng):
    most = max(_cost(c) for c in listed())

    def between(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))

    while True:
        kind = rng.choice(["requests", "requests", "requests", "prompts", "prompts", "score", "tiny", "float32", "routed", "routed"])
        case = {"model": "8b", "layers": rng.randint(4, 36), "dtype": "bfloat16", "steps": 0, "turn": 0, "want": "last"}
        if kind == "requests":
            batch = between(1, 64)
            case.update(steps=between(8, 96), turn=between(2, 300) if rng.random() < 0.25 else 0)
            lengths = _lengths(rng, batch, between(8, 256), between(256, min(24576, 49152 // batch)))
        elif kind == "prompts":
            lengths = _lengths(rng, between(1, 12), between(4, 128), between(128, 4096))
        elif kind == "score":
            case.update(layers=rng.randint(4, 12), want="all")
            lengths = [between(100, 1500)]
        elif kind == "tiny":
            case.update(model="tiny", layers=rng.randint(2, 4), dtype="float32", steps=rng.randint(4, 32), want="sampled")
            lengths = _lengths(rng, between(1, 8), 1, between(2, 150))
        elif kind == "float32":
            case.update(layers=rng.randint(2, 4), dtype="float32", steps=between(1, 24))
            lengths = _lengths(rng, between(1, 8), between(4, 40), between(40, 160))
        else:
            case.update(model=rng.choice(sorted(FAGUNEX_WIDTHS)), layers=rng.choice([2, 4]))
            if rng.random() < 0.5:
                lengths = _lengths(rng, between(1, 4), between(30, 300), between(300, 2500))
            else:
                case.update(steps=between(16, 96))
                lengths = _lengths(rng, between(1, 32), between(8, 100), between(100, 700))
        if kind in ("requests", "prompts") and rng.random() < 0.25:
            case.update(model="14b", layers=rng.randint(4, 12))
        case["lengths"] = ",".join(str(n) for n in lengths)
        if _cost(case) <= most:
            return case


def _lengths(rng, count, lo, hi):
    return [rng.randint(lo, max(lo, hi)) for _ in range(count)]


def _ragged(count, lo, hi):
    return ",".join(str(n) for n in _lengths(random.Random(count * 1000003 + hi), count, lo, hi))


def _prompt_lengths(case):
    return [int(n) for n in case["lengths"].split(",")]


def _vocab(case):
    return FAGUNEX_VOCAB if case["model"] in FAGUNEX_WIDTHS else MODELS[case["model"]]["vocab_size"]


def _config(case):
    if case["model"] in FAGUNEX_WIDTHS:
        return _fagunex(case)
    return dict(MODELS[case["model"]], num_hidden_layers=case["layers"], torch_dtype=case["dtype"])


def _fagunex(case):
    width, ff = FAGUNEX_WIDTHS[case["model"]]
    latent = {"heads": 16, "dim": HEAD, "rot_dim": HEAD // 2, "vdim": width // 16, "kv_rank": 3 * HEAD // 2,
              "scale": (HEAD + HEAD // 2) ** -0.5, "rot": {"base": 1000000.0, "dims": HEAD // 2}}
    order = [{"type": "latent_attention", "mixer": dict(latent, q_rank=width * 3 // 4, mask={"size": 1024})},
             {"type": "hgrn2", "mixer": {"heads": width // HEAD, "dim": HEAD, "vdim": HEAD}},
             {"type": "latent_attention_2", "mixer": latent},
             {"type": "hgrn2", "mixer": {"heads": width // HEAD, "dim": HEAD, "vdim": HEAD}}]
    moe = {"kind": "moe", "expert": {"ff": ff // 4}, "router": {"experts": EXPERTS, "top": TOP}, "shared": {"ff": ff // 4}}
    return {"architecture": "Fagunex", "vocab": FAGUNEX_VOCAB, "width": width, "norm": {"eps": 1e-6},
            "token_side": {"dim": SIDE}, "layers": [dict(order[i % 4], mlp=moe) for i in range(case["layers"])]}


# ------------------------------------------------------------------------------------------------ inputs
def _tokens(case, seed):
    """For every sequence (prompt, its single tokens, its follow-up, the single tokens after that)."""
    rng = np.random.default_rng(seed)
    vocab, turn = _vocab(case), case["turn"]
    later = case["steps"] if turn else 0
    return [tuple(rng.integers(0, vocab, size=n) for n in (length, case["steps"], turn, later))
            for length in _prompt_lengths(case)]


def _weights(case, seed):
    """Every tensor of the model by its checkpoint name, on the GPU, in the type the model computes in."""
    specs = q.build_model(q.config_from_dict(_config(case)).plan()).weight_specs()
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    out = {}
    for name in sorted(specs):
        spec = specs[name]
        gen = torch.Generator(device="cuda")
        gen.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
        if case["model"] in FAGUNEX_WIDTHS:
            out[name] = _fagunex_weight(name, spec, gen).to(dtype)
            continue
        tensor = torch.empty(spec.shape, dtype=dtype, device="cuda")
        tensor.normal_(*_qwen3_spread(name, spec, case["layers"]), generator=gen)
        out[name] = tensor
    return out


def _qwen3_spread(name, spec, layers):
    """(mean, deviation) of a tensor: norms around 1, matrices N(0, 1/columns).  As in a trained model the hidden state is
    large beside what any one layer adds to it: the products that add to it are smaller by the root of their number."""
    if spec.role == "norm":
        return 1.0, 0.1
    if "embed_tokens" in name:
        return 0.0, 1.0
    return 0.0, (spec.shape[-1] * (2 * layers if "o_proj" in name or "down_proj" in name else 1)) ** -0.5


def _fagunex_weight(name, spec, gen):
    """Matrices N(0, 1/columns), norms around 1, slopes around 1, shifts and lower bounds over [0, 0.9], sinks N(0, 1).

    A trained router decides clearly; a random one is full of near ties that any other rounding decides otherwise.  So the
    first columns of the embedding hold +-16, which no sublayer's output turns and which every norm's tanh takes to +-1, and
    the routers read these columns: which experts a token goes to differs from token to token and layer to layer, about
    evenly, and does not hang on a rounding."""
    tail = name.rsplit(".", 1)[-1]
    value = torch.randn(spec.shape, generator=gen, device="cuda", dtype=torch.float32)
    if tail == "alpha":
        return 1.0 + 0.3 * torch.tanh(value)
    if tail in ("shift", "lower"):
        return 0.9 * torch.rand(spec.shape, generator=gen, device="cuda")
    if tail == "sink":
        return value
    if spec.role == "norm":
        value = 1.0 + 0.1 * value
        if name.endswith(".norm2"):
            value[:ROUTED_BY] = 1.0
        return value
    if spec.role == "bias":
        value = 0.1 * value
        if name.endswith(".norm2.b"):
            value[:ROUTED_BY] = 0.0
        return value
    if tail == "router":
        value[:, ROUTED_BY:] = 0.0
        return 0.5 * value
    if name == "embed":
        value[:, :ROUTED_BY] = 16.0 * torch.sign(value[:, :ROUTED_BY])
        return value
    return value if name == "side.embed" else value / spec.shape[-1] ** 0.5


def prepare(case, seed):
    config = q.config_from_dict(_config(case))
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    model = q.build_model(config.plan())
    model.bind(_weights(case, seed), dtype, "cuda:0")
    tokens = _tokens(case, seed)
    longest = max(sum(len(part) for part in parts) for parts in tokens) + (case["steps"] if case["want"] == "sampled" else 0)
    pages = -(-longest // q.PAGE_TOKENS)
    engine = q.Engine(model, config, max_tokens=len(tokens) * pages * q.PAGE_TOKENS, max_seq_len=longest, n_slots=len(tokens))
    state = {"engine": engine, "case": case, "seed": seed}
    prompts = [[int(t) for t in parts[0]] for parts in tokens]
    if case["want"] == "sampled":
        return dict(state, prompts=prompts)
    wanted = [list(range(len(p))) if case["want"] == "all" else [len(p) - 1] for p in prompts]
    single = lambda k: [[[int(parts[k][i])] for parts in tokens] for i in range(len(tokens[0][k]))]  # noqa: E731
    steps = [(prompts, wanted)] + [(row, [[0]] * len(row)) for row in single(1)]
    if case["turn"]:
        steps.append(([[int(t) for t in parts[2]] for parts in tokens], [[case["turn"] - 1]] * len(tokens)))
        steps += [(row, [[0]] * len(row)) for row in single(3)]
    logits = [torch.empty((sum(len(w) for w in want), _vocab(case)), dtype=torch.float32, device="cuda") for _, want in steps]
    return dict(state, steps=steps, logits=logits)


def run(state):
    engine = state["engine"]
    if state["case"]["want"] == "sampled":
        got = q.generate_token_ids(engine, state["prompts"], q.SamplingParams(mode="sample", temperature=0.7, seed=state["seed"] % 1000),
                                   q.GenerationOptions(max_new_tokens=state["case"]["steps"]))
        return np.array([r.token_ids for r in got], dtype=np.int64)
    slots = [engine.new_sequence() for _ in state["steps"][0][0]]
    for (tokens, wanted), keep in zip(state["steps"], state["logits"]):
        entries = [q.StepEntry(slot, new, want) for slot, new, want in zip(slots, tokens, wanted)]
        keep.copy_(engine.step(entries))                # what `step` returns is valid until the next step
    for slot in slots:
        engine.release(slot)
    return _whole(case=state["case"], logits=state["logits"])


def _whole(case, logits):
    """The prompts' logits and, where there are any, those of all later steps in the order in which they came."""
    out = {"prompt": logits[0]}
    if len(logits) > 1:
        out["later"] = torch.cat(logits[1:])
    return out


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _layer_values(case):
    """(matrix values of a layer that every token uses, matrix values of one routed expert, multiplications a token makes
    in a layer's matrices, cached values per token and layer, multiplications per token and key it looks at) on average."""
    if case["model"] in FAGUNEX_WIDTHS:
        h, ff = FAGUNEX_WIDTHS[case["model"]]
        heads, rank, rot, qr = 16, 3 * HEAD // 2, HEAD // 2, h * 3 // 4
        latent = h * (rank + rot) + heads * (HEAD + h // 16) * rank + h * h
        first = latent + h * qr + qr * heads * (HEAD + rot) + h * h
        second = latent + h * heads * (HEAD + rot)
        recurrent = 4 * h * h
        mixers = [(first, rank + rot, heads * (2 * rank + rot)), (recurrent, 0, 0), (second, rank + rot, heads * (2 * rank + rot)),
                  (recurrent, 0, 0)]
        used = [mixers[i % 4] for i in range(case["layers"])]
        common = 3 * h * (ff // 4) + (EXPERTS + 1) * h + 2 * h * SIDE
        expert = 3 * h * (ff // 4)
        n = len(used)
        dense = sum(m[0] for m in used) / n + common
        return dense, expert, dense + TOP * expert, sum(m[1] for m in used) / n, sum(m[2] for m in used) / n
    c = _config(case)
    h, i, d, nq, nkv = c["hidden_size"], c["intermediate_size"], c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"]
    dense = (nq + 2 * nkv) * d * h + h * nq * d + 3 * h * i
    return dense, 0, dense, 2 * nkv * d, 2 * nq * d


def work(case):
    """Every step reads each matrix that it uses once (a step's tokens hang on the step before), the cached keys and values
    of its sequences once, and writes its rows of the cache and the logits that are wanted."""
    size = 4 if case["dtype"] == "float32" else 2
    dense, expert, per_token, cached, per_key = _layer_values(case)
    width = FAGUNEX_WIDTHS[case["model"]][0] if case["model"] in FAGUNEX_WIDTHS else _config(case)["hidden_size"]
    lengths, vocab, layers = _prompt_lengths(case), _vocab(case), case["layers"]
    steps = [list(lengths)] + [[1] * len(lengths)] * (case["steps"] - 1 if case["want"] == "sampled" else case["steps"])
    if case["turn"]:
        steps += [[case["turn"]] * len(lengths)] + [[1] * len(lengths)] * case["steps"]
    bytes_, flops, past = 0.0, 0.0, [0] * len(lengths)
    for new in steps:
        n = sum(new)
        rows = n if case["want"] == "all" else len(new)
        experts = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** n) if expert else 0.0
        keys = sum(t * p + t * (t + 1) // 2 for t, p in zip(new, past))
        bytes_ += size * (layers * (dense + experts * expert) + vocab * width + n * width)
        bytes_ += size * layers * cached * (sum(past) + n) + 4.0 * rows * vocab
        flops += 2.0 * layers * (per_token * n + per_key * keys) + 2.0 * rows * vocab * width
        past = [p + t for p, t in zip(past, new)]
    return {"bytes": bytes_, "flops": flops}


def _cost(case):
    """Seconds that the work takes at about the rates of this GPU: the measure by which drawn cases are held below the largest."""
    w = work(case)
    rate = 3e13 if case["dtype"] == "float32" else 1.2e15
    calls = 1 + case["steps"] * (2 if case["turn"] else 1)
    return w["bytes"] / 5e12 + w["flops"] / rate + calls * 1e-4


def tolerance(case):
    if case["want"] == "sampled":
        return {"rel": 0.0, "differ": 0.01}
    if case["dtype"] == "float32":
        return {"rel": 7e-6, "max": 6e-5}                 # 1.7e-6 and 1.4e-5 away from 64 bits
    # Two forms of every product, which round the same 16-bit values after sums in another order, give logits 0.010 apart
    # (0.08 at most) in 36 layers and 0.005 in 9 or in the Fagunex models; 64 bits are 0.015 and 0.006 away.
    return {"rel": 0.03, "max": 0.3} if case["model"] not in FAGUNEX_WIDTHS else {"rel": 0.02, "max": 0.17}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    if case["want"] == "sampled":
        return None                                        # token ids have no value in 64 bits
    w = _weights(case, seed)
    parts = _tokens(case, seed)
    tokens = [np.concatenate(p) for p in parts]
    spans, at = [], 0
    for t in tokens:
        spans.append((at, at + len(t)))
        at += len(t)
    ids = torch.from_numpy(np.concatenate(tokens)).cuda()
    # which rows' logits come back, in the order in which the steps give them
    first, steps, turn = [], case["steps"], case["turn"]
    for (lo, _), length in zip(spans, _prompt_lengths(case)):
        first += list(range(lo, lo + length)) if case["want"] == "all" else [lo + length - 1]
    later = []
    ends = [lo + length for (lo, _), length in zip(spans, _prompt_lengths(case))]
    for i in range(steps):
        later += [e + i for e in ends]
    if turn:
        later += [e + steps + turn - 1 for e in ends]
        for i in range(steps):
            later += [e + steps + turn + i for e in ends]
    forward = _fagunex_exact if case["model"] in FAGUNEX_WIDTHS else _qwen3_exact
    hidden, head = forward(_config(case), w, ids, spans, first + later)
    logits = torch.empty((hidden.shape[0], head.shape[0]), dtype=torch.float64, device="cuda")
    for lo in range(0, head.shape[0], 16384):
        logits[:, lo:lo + 16384] = hidden @ head[lo:lo + 16384].double().t()
    out = {"prompt": logits[:len(first)]}
    if later:
        out["later"] = logits[len(first):]
    return out


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _times(x, w):
    return x @ w.double().t()


def _positions(spans):
    return torch.cat([torch.arange(hi - lo, device="cuda", dtype=torch.float64) for lo, hi in spans])


def _turned(x, positions, base, dims, pairs):
    """Rotate the first `dims` values of x [T, heads, d]: pairs (2i, 2i + 1) for `pairs`, else (i, i + dims / 2)."""
    half = dims // 2
    angle = positions[:, None] * torch.tensor([base ** (-2.0 * i / dims) for i in range(half)], dtype=torch.float64, device="cuda")
    c, s = angle.cos()[:, None, :], angle.sin()[:, None, :]
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, half), slice(half, dims))
    out = x.clone()
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _attended(qs, ks, vs, scale, spans, window=None, sink=None):
    """Causal softmax attention inside every span: qs [T, H, d], ks [T, G, d], vs [T, G, v] -> [T, H, v]."""
    heads, groups = qs.shape[1], ks.shape[1]
    out = torch.empty((qs.shape[0], heads, vs.shape[2]), dtype=torch.float64, device="cuda")
    for lo, hi in spans:
        piece = max(1, min(1024, (1 << 27) // (heads * (hi - lo))))
        for at in range(lo, hi, piece):
            to = min(hi, at + piece)
            since = lo if window is None else max(lo, at - window + 1)
            k = ks[since:to].permute(1, 2, 0)                                       # [G, d, keys]
            v = vs[since:to].permute(1, 0, 2)                                       # [G, keys, v]
            x = qs[at:to].reshape(to - at, groups, heads // groups, -1).permute(1, 2, 0, 3).reshape(groups, -1, qs.shape[2])
            s = (x @ k * scale).view(groups, heads // groups, to - at, to - since)
            apart = torch.arange(at, to, device="cuda")[:, None] - torch.arange(since, to, device="cuda")[None, :]
            hidden = apart < 0 if window is None else (apart < 0) | (apart >= window)
            s.masked_fill_(hidden, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                z = sink.double().view(groups, heads // groups, 1, 1)
                top = torch.maximum(top, z)
            s.sub_(top).exp_()
            total = s.sum(-1, keepdim=True)
            if sink is not None:
                total = total + (z - top).exp()
            y = (s.view(groups, -1, to - since) @ v).view(groups, heads // groups, to - at, -1) / total
            out[at:to] = y.permute(2, 0, 1, 3).reshape(to - at, heads, -1)
    return out


def _qwen3_exact(c, w, ids, spans, rows):
    d, nq, nkv, eps = c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"], c["rms_norm_eps"]
    positions = _positions(spans)
    x = w["model.embed_tokens.weight"][ids].double()
    for i in range(c["num_hidden_layers"]):
        t = lambda name: w["model.layers.%d.%s.weight" % (i, name)]  # noqa: E731,B023
        h = _rms(x, eps) * t("input_layernorm").double()
        qs = _rms(_times(h, t("self_attn.q_proj")).view(-1, nq, d), eps) * t("self_attn.q_norm").double()
        ks = _rms(_times(h, t("self_attn.k_proj")).view(-1, nkv, d), eps) * t("self_attn.k_norm").double()
        vs = _times(h, t("self_attn.v_proj")).view(-1, nkv, d)
        qs, ks = (_turned(y, positions, c["rope_theta"], d, False) for y in (qs, ks))
        y = _attended(qs, ks, vs, d ** -0.5, spans)
        x = x + _times(y.reshape(-1, nq * d), t("self_attn.o_proj"))
        h = _rms(x, eps) * t("post_attention_layernorm").double()
        g = _times(h, t("mlp.gate_proj"))
        g = g.mul_(torch.sigmoid(g)).mul_(_times(h, t("mlp.up_proj")))
        x = x + _times(g, t("mlp.down_proj"))
    x = _rms(x[torch.tensor(rows, device="cuda")], eps) * w["model.norm.weight"].double()
    return x, w["lm_head.weight"]


def _fagunex_exact(c, w, ids, spans, rows):
    eps, width = c["norm"]["eps"], c["width"]
    positions = _positions(spans)
    starts = torch.tensor([lo for lo, _ in spans], device="cuda")

    def norm(x, name):
        return torch.tanh(w[name + ".alpha"].double() * x) * w[name].double() + w[name + ".b"].double()

    def feed_forward(h, p):
        g = _times(h, w[p + "gate"])
        return _times(g * torch.sigmoid(g) * _times(h, w[p + "up"]), w[p + "down"])

    x = w["embed"][ids].double()
    for i, layer in enumerate(c["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        h = norm(x, p + "norm1")
        before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        before[starts] = 0.0
        h = h + (before - h) * w[p + "shift"].double()
        t = lambda name: w[p + "mix." + name]  # noqa: E731,B023
        heads, d, vd = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "hgrn2":
            qs = _times(h, t("q")).view(-1, heads, d)
            qs = qs * torch.sigmoid(qs)
            vs = _times(h, t("v")).view(-1, heads, vd)
            low = t("lower").double()
            f = (low + (1.0 - low) * torch.sigmoid(_times(h, t("f")) + t("f.b").double())).view(-1, heads, d)
            y = torch.empty((len(ids), heads, vd), dtype=torch.float64, device="cuda")
            # all sequences side by side, token by token
            longest, lows = max(hi - lo for lo, hi in spans), [lo for lo, _ in spans]
            state = torch.zeros((len(spans), heads, d, vd), dtype=torch.float64, device="cuda")
            for k in range(longest):
                live = [s for s, (lo, hi) in enumerate(spans) if lo + k < hi]
                at = torch.tensor([lows[s] + k for s in live], device="cuda")
                who = slice(None) if len(live) == len(spans) else torch.tensor(live, device="cuda")
                fk = f[at]
                new = torch.addcmul((1.0 - fk)[..., None] * vs[at][:, :, None, :], fk[..., None], state[who])
                state[who] = new
                y[at] = (qs[at][:, :, None, :] @ new)[:, :, 0]
            y = (_rms(y, eps) * t("norm").double()).reshape(len(ids), heads * vd)
        else:
            gated, rot, rank = layer["type"] == "latent_attention", m["rot"], m["kv_rank"]
            if m.get("q_rank"):
                qs = _times(_rms(_times(h, t("dq")), eps) * t("dq.norm").double(), t("uq"))
            else:
                qs = _times(h, t("q"))
            qs = qs.view(-1, heads, d + m["rot_dim"])
            down = _times(h, t("dkv"))
            latent = _rms(down[:, :rank], eps) * t("dkv.norm").double()
            q_turned = _turned(qs[:, :, d:], positions, rot["base"], rot["dims"], gated)
            k_turned = _turned(down[:, None, rank:], positions, rot["base"], rot["dims"], gated)
            ks = torch.cat([_times(latent, t("uk")).view(-1, heads, d), k_turned.expand(-1, heads, -1)], -1)
            vs = _times(latent, t("uv")).view(-1, heads, vd)
            y = _attended(torch.cat([qs[:, :, :d], q_turned], -1), ks, vs, m["scale"], spans,
                          m["mask"]["size"] if m.get("mask") else None, t("sink") if gated else None).reshape(len(ids), heads * vd)
            if gated:
                y = y * torch.sigmoid(_times(h, t("g")))
        x = x + norm(_times(y, t("o")), p + "norm1b")
        h = norm(x, p + "norm2")
        z, chosen = _times(h, w[p + "mlp.router"]).topk(TOP, -1)
        share = torch.softmax(z, -1)
        y = torch.sigmoid(_times(h, w[p + "mlp.shared.sg"])) * feed_forward(h, p + "mlp.shared.")
        for e in range(EXPERTS):
            who, place = (chosen == e).nonzero(as_tuple=True)
            y.index_add_(0, who, share[who, place][:, None] * feed_forward(h[who], "%smlp.e%d." % (p, e)))
        x = x + norm(y, p + "norm2b")
        side = w["side.embed"][ids][:, i * SIDE:(i + 1) * SIDE].double()
        g = torch.nn.functional.gelu(_times(x, w[p + "side.gate"]), approximate="tanh") * side
        x = x + _rms(_times(g, w[p + "side.proj"]), eps) * w[p + "side.norm"].double()
    return norm(x[torch.tensor(rows, device="cuda")], "final.norm"), w["head"]
