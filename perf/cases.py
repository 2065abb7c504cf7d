"""What users of this framework run, as measurable cases: decode steps and prompts of the models it serves.

A *decode* case is a serving loop: a batch whose contexts are already cached takes `steps` tokens, one call of
`step` each (host ids in, host tokens out), from the captured step graph. A *prompt* case is the processing of
new prompts: `prefill` for a batch of equal lengths, `forward` for ragged ones in portions. Both go through the
engines that the model registry hands out.

Weights and cached contexts are random at the scale that the mechanisms meet; every tensor is made from the
seed alone. `exact` restates the models in 64-bit torch.
"""

from __future__ import annotations

import math
from typing import Dict, List

import torch

from llm_compiler_b200 import bazirax, lozanex, qwen2
from llm_compiler_b200.engine import Qwen2Engine
from llm_compiler_b200.hybrid_engine import HybridEngine

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}

# width, feed-forward, heads and head size of the designs that bench.py puts beside Qwen2
HYBRID_SIZES = {
    "0.5b": dict(width=896, ff=4864, heads=14, dim=64, kv_heads=2, q_rank=448, kv_rank=256, experts=16, active=2),
    "1.5b": dict(width=2048, ff=8192, heads=16, dim=128, kv_heads=2, q_rank=768, kv_rank=512, experts=32, active=4),
}
HYBRID_VOCABULARY = 32768
CONV_TAPS, GATE_RANK = 4, 16

# The largest contexts and prompts of the drawn cases (tokens in all sequences together).
CONTEXT_TOKENS = 64 * 4096
PROMPT_TOKENS = {"qwen2-0.5b": 4 * 4096, "qwen2-7b-4l": 4096, "bazirax-0.5b": 8192, "lozanex-0.5b": 8192,
                 "bazirax-1.5b": 8192, "lozanex-1.5b": 8192}


def _decode(name, model, batch, context, *, dtype="bf16", ragged=False, paged=False, steps=8) -> dict:
    return dict(name=name, task="decode", model=model, dtype=dtype, batch=batch, context=context, ragged=ragged,
                paged=paged, steps=steps)


def _prompt(name, model, batch, tokens, *, dtype="bf16", ragged=False, portion=0) -> dict:
    return dict(name=name, task="prompt", model=model, dtype=dtype, batch=batch, tokens=tokens, ragged=ragged,
                portion=portion)


def listed() -> List[dict]:
    return [
        # one user's conversation: a single sequence, every launch on the critical path
        _decode("decode-single", "qwen2-0.5b", 1, 1000),
        # the benchmark's serving batch: equal contexts, a step bound by weights and cached keys and values
        _decode("decode-batch", "qwen2-0.5b", 64, 4096),
        # a server with block tables: an odd number of sequences of very different ages
        _decode("decode-ragged-paged", "qwen2-0.5b", 23, 6000, ragged=True, paged=True),
        # the larger model (four of its layers), heads of 128, contexts spread up to 8192
        _decode("decode-7b-ragged", "qwen2-7b-4l", 64, 8192, ragged=True),
        # a full-precision model, as for checks against the reference
        _decode("decode-fp32", "qwen2-0.5b", 4, 600, dtype="fp32"),
        # a chat turn: one short prompt, where launches and host work count
        _prompt("prompt-short", "qwen2-0.5b", 1, 77),
        # documents: the largest prompts of the benchmark
        _prompt("prompt-long", "qwen2-0.5b", 4, 4096),
        # a half-precision checkpoint
        _prompt("prompt-fp16", "qwen2-0.5b", 2, 515, dtype="fp16"),
        # recurrent and latent-attention layers: a served batch, and prompts arriving in portions
        _decode("decode-bazirax", "bazirax-1.5b", 32, 4096),
        _prompt("prompt-bazirax-portions", "bazirax-0.5b", 5, 1500, ragged=True, portion=512),
        # delta rule, attention and experts: ragged decoding and whole prompts
        _decode("decode-lozanex", "lozanex-1.5b", 24, 3000, ragged=True),
        _prompt("prompt-lozanex", "lozanex-1.5b", 4, 2048),
    ]


def _spread(rng, low: int, high: int) -> int:
    """An integer between low and high, spread evenly over its logarithm."""

    return min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))


def draw(rng) -> dict:
    family = rng.choice(["qwen2", "qwen2", "bazirax", "lozanex"])
    size = rng.choice(["0.5b", "0.5b", "7b-4l"] if family == "qwen2" else ["0.5b", "1.5b"])
    model = f"{family}-{size}"
    dtype = rng.choice(["bf16"] * 5 + (["fp16", "fp32"] if model == "qwen2-0.5b" else ["fp32"]))
    if rng.random() < 0.5:
        batch = _spread(rng, 1, 64 if dtype == "bf16" else 8)
        context = _spread(rng, 16, min(8192, CONTEXT_TOKENS // batch) if dtype == "bf16" else 1024)
        paged = family == "qwen2" and dtype == "bf16" and rng.random() < 0.3
        case = _decode("", model, batch, context, dtype=dtype, ragged=rng.random() < 0.5, paged=paged,
                       steps=rng.randint(4, 8))
    else:
        most = PROMPT_TOKENS[model] if dtype == "bf16" else 1024
        batch = _spread(rng, 1, 8 if dtype == "bf16" else 2)
        ragged = family != "qwen2" and rng.random() < 0.5
        tokens = _spread(rng, 4, min(4096, most // batch))
        case = _prompt("", model, batch, tokens, dtype=dtype, ragged=ragged,
                       portion=rng.choice([0, 256, 512]) if ragged else 0)
    del case["name"]
    return case


# ------------------------------------------------------------------- models and inputs ----
def _is_qwen(case: dict) -> bool:
    return case["model"].startswith("qwen2")


def _config(model: str):
    if model == "qwen2-0.5b":
        return qwen2.QWEN2_0_5B
    if model == "qwen2-7b-4l":
        full = qwen2.QWEN2_7B
        return qwen2.Qwen2Config(hidden_size=full.hidden_size, intermediate_size=full.intermediate_size, num_layers=4,
                                 num_heads=full.num_heads, num_kv_heads=full.num_kv_heads,
                                 rms_norm_eps=full.rms_norm_eps, rope_theta=full.rope_theta,
                                 vocab_size=full.vocab_size)
    family, size = model.split("-")
    size = HYBRID_SIZES[size]
    heads, dim = size["heads"], size["dim"]
    delta = dict(heads=heads, kv_heads=heads, dim=dim, vdim=dim, conv=CONV_TAPS)
    if family == "bazirax":
        retention = dict(heads=heads, dim=dim, vdim=dim, rot=dict(base=1e4, dims=dim),
                         decay=[1 - 2.0 ** -(5 + i * 5 / heads) for i in range(heads)])
        latent = dict(heads=heads, dim=dim, vdim=dim, q_rank=size["q_rank"], kv_rank=size["kv_rank"],
                      scale=dim ** -0.5)
        kinds = [("channel_delta", delta), ("retention", retention), ("latent_attention", latent)] * 2
        kinds[5] = ("latent_attention", dict(latent, kv_from=2))
        layers = tuple(bazirax.LayerSpec(kind, spec, size["ff"]) for kind, spec in kinds)
        return bazirax.BaziraxConfig(vocab_size=HYBRID_VOCABULARY, hidden_size=size["width"], norm_eps=1e-5,
                                     layers=layers)
    attention = dict(heads=heads, kv_heads=size["kv_heads"], dim=dim, vdim=dim, scale=dim ** -0.5,
                     rot=dict(base=1e6, dims=dim), mask=dict(size=8192))
    mlp = dict(kind="moe", expert=dict(ff=size["ff"] // 2 // size["active"]),
               router=dict(experts=size["experts"], top=size["active"]), shared=dict(ff=size["ff"] // 2))
    kinds = [("delta", delta), ("attention", attention), ("delta", delta), ("delta", delta),
             ("attention", dict(attention, kv_from=1)), ("delta", delta)]
    layers = tuple(lozanex.LayerSpec(kind, spec, mlp) for kind, spec in kinds)
    return lozanex.LozanexConfig(vocab_size=HYBRID_VOCABULARY, hidden_size=size["width"], norm_eps=1e-5, layers=layers)


def _weights(case: dict, seed: int) -> Dict[str, torch.Tensor]:
    config, dtype = _config(case["model"]), DTYPES[case["dtype"]]
    if _is_qwen(case):
        return qwen2.make_weights(config, seed=seed, dtype=dtype, device="cuda", reproducible=False)
    if case["model"].startswith("bazirax"):
        return bazirax.make_weights(config, seed=seed, dtype=dtype, device="cuda", gate_rank=GATE_RANK)
    weights = lozanex.make_weights(config, seed=seed, dtype=dtype, device="cuda")
    # As in trained models, what a layer adds is small against the stream. (Were it as large, every expert that
    # rounding swaps for its runner-up would change all that follows, and no two results could be compared.)
    for name in weights:
        if name.endswith((".norm1", ".norm2")):
            weights[name] *= 0.25 if name.endswith(".norm1") else 0.1
    return weights


def _lengths(case: dict, longest: int, seed: int) -> List[int]:
    """Tokens of every sequence: `longest` each, or uniform up to it."""

    if not case["ragged"]:
        return [longest] * case["batch"]
    generator = torch.Generator().manual_seed(seed)
    return torch.randint(max(1, longest // 16), longest + 1, (case["batch"],), generator=generator).tolist()


def _ids(case: dict, shape, seed: int) -> torch.Tensor:
    return torch.randint(0, _config(case["model"]).vocab_size, shape, generator=torch.Generator().manual_seed(seed + 1))


def _capacity(case: dict) -> int:
    return case["context"] + case["steps"] if case["task"] == "decode" else case["tokens"]


def _random(generator, shape, scale, dtype) -> torch.Tensor:
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, scale, generator=generator)


def _qwen_context(case: dict, seed: int):
    """Cached keys and values of every layer, [batch, capacity, kv_heads, head_dim], layer by layer."""

    config, generator = _config(case["model"]), torch.Generator(device="cuda").manual_seed(seed + 2)
    shape = (case["batch"], _capacity(case), config.num_kv_heads, config.head_dim)
    scale = 0.02 * config.hidden_size ** 0.5  # what projections of normed rows have
    for _ in range(config.num_layers):
        yield tuple(_random(generator, shape, scale, DTYPES[case["dtype"]]) for _ in range(2))


def _hybrid_context(case: dict, seed: int) -> List[Dict[str, torch.Tensor]]:
    """What every layer keeps of its sequences: recurrent state, inputs of the short convolutions (by position
    modulo their number), cached latents, or cached keys and values. Zeros in front of a prompt."""

    generator = torch.Generator(device="cuda").manual_seed(seed + 2)
    batch, dtype, scale = case["batch"], DTYPES[case["dtype"]], 1.0 if case["task"] == "decode" else 0.0
    kept = []
    for layer in _config(case["model"]).layers:
        m = layer.mixer
        state = {}
        if "delta" in layer.type or layer.type == "retention":
            state["state"] = _random(generator, (batch, m["heads"], m["dim"], m["vdim"]), 0.1 * scale, torch.float32)
        if "delta" in layer.type:
            channels = 2 * m["kv_heads"] * m["dim"] + m["heads"] * m["vdim"]
            state["ring"] = _random(generator, (batch, m["conv"], channels), scale, dtype)
        if layer.type == "latent_attention" and m.get("kv_from") is None:
            state["latent"] = _random(generator, (batch, _capacity(case), m["kv_rank"]), scale, dtype)
        if layer.type == "attention" and m.get("kv_from") is None:
            for name in ("keys", "values"):
                state[name] = _random(generator, (batch, _capacity(case), m["kv_heads"], m["dim"]), scale, dtype)
        kept.append(state)
    return kept


# ------------------------------------------------------------------------------ cases ----
def prepare(case: dict, seed: int) -> dict:
    """The engine as a serving program holds it; for decoding with its contexts cached and its step captured."""

    config, weights = _config(case["model"]), _weights(case, seed)
    batch, capacity = case["batch"], _capacity(case)
    if _is_qwen(case):
        layout = dict(kv_layout="paged") if case.get("paged") else {}
        engine = Qwen2Engine(config, weights, batch=batch, capacity=capacity, **layout)
    else:
        engine = HybridEngine(config, weights, batch=batch, capacity=capacity)
    state = dict(case=case, engine=engine)
    if case["task"] == "prompt":
        state["ids"] = _ids(case, (batch, case["tokens"]), seed)
        state["prompts"] = [row[:n].tolist() for row, n in zip(state["ids"], _lengths(case, case["tokens"], seed))]
        return state
    lengths = torch.tensor(_lengths(case, case["context"], seed))
    state["lengths"] = lengths
    state["ids"] = _ids(case, (case["steps"], batch), seed)
    engine.load_context(lengths)
    if _is_qwen(case):
        for layer, cached in enumerate(_qwen_context(case, seed)):
            for buffer, rows in zip((engine.state.keys[layer], engine.state.values[layer]), cached):
                if not case["paged"]:
                    buffer.copy_(rows)
                    continue
                size, table = engine.state.block_size, engine.state.block_table
                for sequence, tokens in enumerate(lengths.tolist()):
                    for first in range(0, tokens, size):
                        count = min(size, tokens - first)
                        buffer[int(table[sequence, first // size])][:count].copy_(rows[sequence, first:first + count])
    else:
        # the part of a context that decoding rewrites is put back in front of every pass, as a program that
        # starts from a cached prefix does
        state["rewritten"] = []
        for buffers, made in zip(engine.state.layers, _hybrid_context(case, seed)):
            for name, tensor in made.items():
                buffers[name].copy_(tensor)
                if name in ("state", "ring"):
                    state["rewritten"].append((buffers[name], tensor))
    engine.capture()
    return state


def run(state: dict):
    case, engine = state["case"], state["engine"]
    if case["task"] == "decode":
        return _run_decode(case, engine, state)
    if not case["ragged"]:
        logits = engine.prefill(state["ids"])
    else:
        logits = _run_portions(case, engine, state["prompts"])
    if _is_qwen(case):
        return {"logits": logits, "keys": list(engine.state.keys), "values": list(engine.state.values)}
    return {"logits": logits, "state": engine.state.layers}


def _run_decode(case: dict, engine, state: dict):
    engine.load_context(state["lengths"])
    for buffer, tensor in state.get("rewritten", ()):
        buffer.copy_(tensor)
    logits, tokens = [], []
    for ids in state["ids"]:
        tokens.append(engine.step(ids).clone())
        logits.append(engine.logits.clone())
    result = {"logits": logits, "tokens": torch.stack(tokens)}
    if not _is_qwen(case):
        result["state"] = [buffer for buffer, _ in state["rewritten"]]
    elif not case["paged"] and not case["ragged"]:
        new = slice(case["context"], case["context"] + case["steps"])
        result["keys"] = [rows[:, new] for rows in engine.state.keys]
        result["values"] = [rows[:, new] for rows in engine.state.values]
    return result


def _run_portions(case: dict, engine, prompts: List[List[int]]) -> List[torch.Tensor]:
    """The prompts side by side, each call up to `portion` tokens of every sequence that has some left."""

    slots = [engine.open() for _ in prompts]
    portion = case["portion"] or case["tokens"]
    logits: List[torch.Tensor] = [None] * len(prompts)
    for first in range(0, max(map(len, prompts)), portion):
        active = [i for i, prompt in enumerate(prompts) if len(prompt) > first]
        rows = engine.forward([(slots[i], prompts[i][first:first + portion]) for i in active])
        for row, i in enumerate(active):
            logits[i] = rows[row]
    for slot in slots:
        engine.close(slot)
    return logits


def work(case: dict) -> dict:
    """Weights, contexts and results once; products of the projections and of attention."""

    config, size = _config(case["model"]), DTYPES[case["dtype"]].itemsize
    decode = case["task"] == "decode"
    passes = case["steps"] if decode else 1
    # (ragged sequences: uniform between a sixteenth and all of the longest)
    mean = (17 / 32 if case["ragged"] else 1.0) * (case["context"] if decode else case["tokens"])
    rows = case["batch"] * (1 if decode else mean)
    seen = case["batch"] * (mean if decode else mean * mean / 2)  # pairs of query and key
    context = case["batch"] * (mean if decode else 0)
    written = rows
    if _is_qwen(case):
        c = config
        layer = c.hidden_size * (c.q_size + 2 * c.kv_size) + c.q_size * c.hidden_size + \
            3 * c.hidden_size * c.intermediate_size
        used = weights = c.num_layers * layer
        cached = c.num_layers * (context + written) * 2 * c.kv_size * size
        attention = c.num_layers * 4 * seen * c.q_size
        vocabulary = c.vocab_size
    else:
        vocabulary, used, weights, cached, attention = HYBRID_VOCABULARY, 0, 0, 0, 0
        width = config.hidden_size
        for layer in config.layers:
            m = layer.mixer
            inner = m["heads"] * m["dim"]
            if layer.type in ("channel_delta", "retention", "delta"):
                mixer = width * inner * (4 if layer.type == "channel_delta" else 5)
                cached += case["batch"] * m["heads"] * m["dim"] * m["vdim"] * 4 * (2 if decode else 1)
                attention += rows * 4 * inner * m["dim"]
            elif layer.type == "latent_attention":
                mixer = (width + inner) * m["q_rank"] + (2 * inner + width) * m["kv_rank"] + width * inner
                cached += (context + written) * m["kv_rank"] * size
                attention += 4 * seen * inner
            else:
                mixer = 2 * width * (inner + m["kv_heads"] * m["dim"])
                cached += (context + written) * 2 * m["kv_heads"] * m["dim"] * size
                attention += 4 * seen * inner
            if case["model"].startswith("bazirax"):
                dense, experts, active = 3 * width * layer.ff, 0, 0
            else:
                dense = 3 * width * layer.mlp["shared"]["ff"]
                expert, router = 3 * width * layer.mlp["expert"]["ff"], layer.mlp["router"]
                hit = 1 - (1 - router["top"] / router["experts"]) ** rows  # share of experts that get a row
                experts, active = hit * router["experts"] * expert, router["top"] * expert
            used += mixer + dense + active
            weights += mixer + dense + experts
    results = case["batch"] * vocabulary
    head = config.hidden_size * vocabulary
    return {"bytes": passes * ((weights + head + results) * size + cached),
            "flops": passes * (2 * rows * used + 2 * case["batch"] * head + attention)}


def tolerance(case: dict) -> dict:
    """Four times what rounding shows against `exact`: 16-bit results are rounded at every operator, through all
    layers (bf16 0.010 for Qwen2 and 0.015 for Bazirax, fp16 0.0012, fp32 3.4e-6). Lozanex's experts and the greedy
    tokens are chosen by scores that rounding can swap."""

    if case["dtype"] == "bf16":
        rel = {"qwen2": 0.04, "bazirax": 0.06, "lozanex": 0.15}[case["model"].split("-")[0]]
    else:
        rel = {"fp16": 5e-3, "fp32": 1.5e-5}[case["dtype"]]
    return {"rel": rel, "differ": 0.5} if case["task"] == "decode" else {"rel": rel}


# ------------------------------------------------------------- the models in 64 bits ----
def exact(case: dict, seed: int):
    weights = {name: value.double() for name, value in _weights(case, seed).items()}
    if _is_qwen(case):
        return _exact_qwen_decode(case, weights, seed) if case["task"] == "decode" \
            else _exact_qwen_prompt(case, weights, seed)
    return _exact_hybrid(case, weights, seed)


def _norm(x, weight, epsilon, offset=0.0):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + epsilon)
    return y if weight is None else y * (offset + weight)


def _rotate(x, positions, base, dims):
    """x [batch, tokens, heads, size] at positions [batch, tokens]: pair (i, i + dims / 2) of the first `dims`
    dimensions turned by position * base^(-2 i / dims)."""

    half = dims // 2
    steps = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)
    angle = positions.double()[:, :, None, None] * steps
    u, v = x[..., :half], x[..., half:dims]
    c, s = angle.cos(), angle.sin()
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], dim=-1)


def _attend(q, keys, values, positions, scale, *, chunk=None, sink=None):
    """q [batch, tokens, heads, size] over keys [batch, cached, groups, size]: those up to a row's position, with
    `chunk` only those of its own chunk; the denominator of a head also holds exp(sink)."""

    batch, tokens, heads, size = q.shape
    groups, rows = keys.shape[2], []
    places = torch.arange(keys.shape[1], device=q.device)
    for b in range(batch):
        visible = places <= positions[b][:, None]
        if chunk is not None:
            visible &= places >= positions[b][:, None] // chunk * chunk
        scores = torch.einsum("tgnd,cgd->gntc", q[b].view(tokens, groups, -1, size), keys[b]) * scale
        scores = scores.masked_fill(~visible, -math.inf)
        top = scores.amax(-1, keepdim=True)
        extra = 0.0
        if sink is not None:
            column = sink.view(groups, -1, 1, 1)
            top = torch.maximum(top, column)
            extra = (column - top).exp()
        scores = (scores - top).exp()
        scores = scores / (scores.sum(-1, keepdim=True) + extra)
        rows.append(torch.einsum("gntc,cgd->tgnd", scores, values[b]).reshape(tokens, heads, -1))
    return torch.stack(rows)


def _silu(x):
    return x * torch.sigmoid(x)


def _gated(x, gate, up, down):
    return (_silu(x @ gate.T) * (x @ up.T)) @ down.T


def _exact_qwen_layers(config, w, x, positions, caches):
    """x [batch, tokens, hidden] through the layers; caches: (keys, values) of every layer, in 64 bits, which take
    the new rows at `positions`."""

    batch, tokens, _ = x.shape
    which = torch.arange(batch, device=x.device)[:, None]
    for layer in range(config.num_layers):
        p = f"decoder.layers.{layer}."
        h = _norm(x, w[p + "input_layernorm.weight"], config.rms_norm_eps)
        q, k, v = ((h @ w[p + f"self_attn.{n}_proj.weight"].T + w[p + f"self_attn.{n}_proj.bias"])
                   .view(batch, tokens, -1, config.head_dim) for n in "qkv")
        keys, values = caches(layer)
        keys[which, positions] = _rotate(k, positions, config.rope_theta, config.head_dim)
        values[which, positions] = v
        q = _rotate(q, positions, config.rope_theta, config.head_dim)
        mixed = _attend(q, keys, values, positions, config.head_dim ** -0.5)
        x = x + mixed.reshape(batch, tokens, -1) @ w[p + "self_attn.o_proj.weight"].T
        h = _norm(x, w[p + "post_attention_layernorm.weight"], config.rms_norm_eps)
        x = x + _gated(h, *(w[p + f"mlp.{n}_proj.weight"] for n in ("gate", "up", "down")))
    return x


def _exact_qwen_logits(config, w, x):
    return _norm(x[:, -1], w["decoder.norm.weight"], config.rms_norm_eps) @ w["lm_head.weight"].T


def _exact_qwen_prompt(case, w, seed):
    config, ids = _config(case["model"]), _ids(case, (case["batch"], case["tokens"]), seed).cuda()
    shape = (case["batch"], case["tokens"], config.num_kv_heads, config.head_dim)
    kept = [tuple(torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(2))
            for _ in range(config.num_layers)]
    positions = torch.arange(case["tokens"], device="cuda").expand(case["batch"], -1)
    x = _exact_qwen_layers(config, w, w["embed_tokens.weight"][ids], positions, kept.__getitem__)
    return {"logits": _exact_qwen_logits(config, w, x), "keys": [k for k, _ in kept], "values": [v for _, v in kept]}


def _exact_qwen_decode(case, w, seed):
    config = _config(case["model"])
    lengths = torch.tensor(_lengths(case, case["context"], seed), device="cuda")
    cached = list(_qwen_context(case, seed))
    new = [[[], []] for _ in cached]
    logits = []
    for step, ids in enumerate(_ids(case, (case["steps"], case["batch"]), seed).cuda()):
        positions = (lengths + step)[:, None]

        def caches(layer):
            """This layer's context in 64 bits, with the rows of earlier steps as they were computed."""

            wide = tuple(t.double() for t in cached[layer])
            for buffer, rows in zip(wide, new[layer]):
                rows.append(buffer)
                for earlier, row in enumerate(rows[:-1]):
                    at = lengths + earlier
                    buffer[torch.arange(len(at)), at] = row
            return wide

        x = _exact_qwen_layers(config, w, w["embed_tokens.weight"][ids][:, None], positions, caches)
        logits.append(_exact_qwen_logits(config, w, x))
        for layer in new:
            for rows in layer:  # of the whole buffer only the step's row is kept
                rows[-1] = rows[-1][torch.arange(len(lengths)), lengths + step].clone()
    result = {"logits": logits, "tokens": None}
    if not case["paged"] and not case["ragged"]:
        result["keys"], result["values"] = ([torch.stack(layer[i], dim=1) for layer in new] for i in range(2))
    return result


def _short_conv(x, taps, ring, first, counts):
    """The filter over the inputs x [batch, tokens, channels] and those that `ring` [batch, taps, channels] holds of
    earlier positions (by position modulo taps); the ring takes each sequence's last inputs."""

    n = taps.shape[1]
    batch, tokens, _ = x.shape
    which = torch.arange(batch, device=x.device)
    before = torch.stack([torch.where((first >= b)[:, None], ring[which, (first - b) % n], 0.0)
                          for b in range(n - 1, 0, -1)], dim=1)
    window = torch.cat([before, x], dim=1)
    for t in range(tokens):
        keep = t < counts
        ring[which[keep], (first[keep] + t) % n] = x[keep, t]
    return sum(window[:, j:j + tokens] * taps[:, j] for j in range(n))


def _scan(q, k, v, decay, beta, state, counts):
    """S = g S (delta rule: + k (beta (v - S^T k))^T, else + k v^T), read-out S^T q, token by token; q, k
    [batch, tokens, heads, dim], decay broadcast over them, state [batch, heads, dim, vdim] in place."""

    rows = []
    for t in range(q.shape[1]):
        next_state = decay[:, t, :, :, None] * state
        u = v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - torch.einsum("bhdv,bhd->bhv", next_state, k[:, t]))
        next_state = next_state + k[:, t, :, :, None] * u[:, :, None, :]
        rows.append(torch.einsum("bhdv,bhd->bhv", next_state, q[:, t]))
        state.copy_(torch.where((t < counts)[:, None, None, None], next_state, state))
    return torch.stack(rows, dim=1)


def _exact_delta(w, spec, h, kept, first, counts, epsilon):
    batch, tokens, _ = h.shape
    heads, dim = spec["heads"], spec["dim"]
    inputs = torch.cat([h @ w[n].T for n in "qkv"], dim=-1)
    taps = torch.cat([w[n + ".conv"] for n in "qkv"])
    mixed = _silu(_short_conv(inputs, taps, kept["ring"], first, counts))
    q, k, v = (part.view(batch, tokens, -1, dim) for part in mixed.split(heads * dim, dim=-1))
    q, k = (part * torch.rsqrt(part.square().sum(-1, keepdim=True) + 1e-6) for part in (q, k))
    low_rank = "a1" in w
    rates = (h @ w["a1"].T) @ w["a2"].T if low_rank else h @ w["a"].T
    rates = torch.nn.functional.softplus(rates + w["dt_bias"], threshold=1e9).view(batch, tokens, heads, -1)
    decay = torch.exp(-w["A_log"].exp()[:, None] * rates)
    out = _scan(q * dim ** -0.5, k, v, decay, torch.sigmoid(h @ w["b"].T), kept["state"], counts)
    gate = torch.sigmoid((h @ w["g1"].T) @ w["g2"].T) if low_rank else _silu(h @ w["g"].T)
    return (_norm(out, w["norm"], epsilon).flatten(2) * gate) @ w["o"].T


def _exact_retention(w, spec, h, kept, positions, counts, epsilon):
    batch, tokens, _ = h.shape
    q, k, v = ((h @ w[n].T).view(batch, tokens, spec["heads"], -1) for n in "qkv")
    q, k = (_rotate(x, positions, spec["rot"]["base"], spec["rot"]["dims"]) for x in (q, k))
    decay = torch.tensor(spec["decay"], dtype=torch.float64, device=h.device)[:, None].expand(batch, tokens, -1, 1)
    out = _scan(q, k * spec["dim"] ** -0.5, v, decay, None, kept["state"], counts)
    return (_norm(out, None, epsilon).flatten(2) * _silu(h @ w["g"].T)) @ w["o"].T


def _store(cache, rows, positions, counts):
    for b, count in enumerate(counts.tolist()):
        cache[b, positions[b, :count]] = rows[b, :count]


def _exact_latent(w, spec, h, caches, layer, positions, counts, epsilon):
    batch, tokens, _ = h.shape
    heads, dim = spec["heads"], spec["dim"]
    source = spec.get("kv_from")
    if source is None:
        _store(caches[layer]["latent"], _norm(h @ w["dkv"].T, w["dkv.norm"], epsilon), positions, counts)
    latent = caches[layer if source is None else source]["latent"]
    q = (_norm(h @ w["dq"].T, w["dq.norm"], epsilon) @ w["uq"].T).view(batch, tokens, heads, dim)
    keys, values = ((latent @ w[n].T).view(batch, -1, heads, dim) for n in ("uk", "uv"))
    return _attend(q, keys, values, positions, spec["scale"], sink=w["sink"]).flatten(2) @ w["o"].T


def _exact_attention(w, spec, h, caches, layer, positions, counts, epsilon):
    batch, tokens, _ = h.shape
    turn = (positions, spec["rot"]["base"], spec["rot"]["dims"])
    source = spec.get("kv_from")
    if source is None:
        k = _norm(h @ w["k"].T + w["k.b"], w["k.norm"], epsilon).view(batch, tokens, spec["kv_heads"], -1)
        v = (h @ w["v"].T + w["v.b"]).view(batch, tokens, spec["kv_heads"], -1)
        _store(caches[layer]["keys"], _rotate(k, *turn), positions, counts)
        _store(caches[layer]["values"], v, positions, counts)
    cache = caches[layer if source is None else source]
    q = _norm(h @ w["q"].T + w["q.b"], w["q.norm"], epsilon).view(batch, tokens, spec["heads"], -1)
    mixed = _attend(_rotate(q, *turn), cache["keys"], cache["values"], positions, spec["scale"],
                    chunk=spec["mask"]["size"])
    return mixed.flatten(2) @ w["o"].T + w["o.b"]


def _exact_experts(w, spec, h):
    rows = h.flatten(0, 1)
    scores, chosen = torch.sigmoid(rows @ w["router"].T).topk(spec["router"]["top"], dim=-1)
    parts = lambda prefix: (w[prefix + name] for name in ("gate", "up", "down"))
    out = _gated(rows, *parts("shared."))
    for expert in range(spec["router"]["experts"]):
        row, place = (chosen == expert).nonzero(as_tuple=True)
        if len(row):
            out.index_add_(0, row, _gated(rows[row] * scores[row, place, None], *parts(f"e{expert}.")))
    return out.view_as(h)


def _exact_hybrid_pass(config, w, ids, first, counts, caches):
    """Logits of every sequence's last token; ids [batch, tokens] of which `counts` count, behind `first` cached
    tokens."""

    is_bazirax, epsilon = isinstance(config, bazirax.BaziraxConfig), config.norm_eps
    offset = 1.0 if is_bazirax else 0.0
    positions = first[:, None] + torch.arange(ids.shape[1], device=ids.device)
    positions = torch.minimum(positions, (first + counts - 1)[:, None])  # (what follows a sequence does not matter)
    x = w["embed"][ids]
    if not is_bazirax:
        x = _norm(x, w["embed.norm"], epsilon)
    for i, layer in enumerate(config.layers):
        p, spec = f"l{i}.", layer.mixer
        under = lambda prefix: {n[len(prefix):]: t for n, t in w.items() if n.startswith(prefix)}
        mix = under(p + "mix.")
        h = _norm(x, w[p + "norm1"], epsilon, offset) if is_bazirax else x
        if layer.type == "retention":
            y = _exact_retention(mix, spec, h, caches[i], positions, counts, epsilon)
        elif layer.type == "latent_attention":
            y = _exact_latent(mix, spec, h, caches, i, positions, counts, epsilon)
        elif layer.type == "attention":
            y = _exact_attention(mix, spec, h, caches, i, positions, counts, epsilon)
        else:
            y = _exact_delta(mix, spec, h, caches[i], first, counts, epsilon)
        mlp = under(p + "mlp.")
        if is_bazirax:
            x = x + _norm(y, w[p + "norm1b"], epsilon, offset)
            h = _norm(x, w[p + "norm2"], epsilon, offset)
            x = x + _norm(_gated(h, mlp["gate"], mlp["up"], mlp["down"]), w[p + "norm2b"], epsilon, offset)
        else:
            x = x + _norm(y, w[p + "norm1"], epsilon)
            x = x + _norm(_exact_experts(mlp, layer.mlp, x), w[p + "norm2"], epsilon)
    last = x[torch.arange(len(counts)), counts - 1]
    return _norm(last, w["final.norm"], epsilon, offset) @ w["head"].T


def _exact_hybrid(case, w, seed):
    config, batch = _config(case["model"]), case["batch"]
    caches = [{name: t.double() for name, t in layer.items()} for layer in _hybrid_context(case, seed)]
    if case["task"] == "prompt":
        ids = _ids(case, (batch, case["tokens"]), seed).cuda()
        counts = torch.tensor(_lengths(case, case["tokens"], seed), device="cuda")
        logits = _exact_hybrid_pass(config, w, ids, torch.zeros_like(counts), counts, caches)
        return {"logits": list(logits) if case["ragged"] else logits, "state": caches}
    first = torch.tensor(_lengths(case, case["context"], seed), device="cuda")
    ones, logits = torch.ones_like(first), []
    for step, ids in enumerate(_ids(case, (case["steps"], batch), seed).cuda()):
        logits.append(_exact_hybrid_pass(config, w, ids[:, None], first + step, ones, caches))
    rewritten = [layer[name] for layer in caches for name in layer if name in ("state", "ring")]
    return {"logits": logits, "tokens": None, "state": rewritten}
