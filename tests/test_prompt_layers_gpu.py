"""The native prompt loop (csrc/prompt_layers.cu) against its operators called one by one: the same launches but for RoPE
and KV store in one kernel, whose roundings are the same, so every result is equal bit for bit. Every projection of more
than 64 rows sums K in one chain, so a prompt's results do not depend on the prompts beside it either."""

import contextlib

import pytest
import torch

from llm_compiler_b200 import _lib, kernels, qwen2
from llm_compiler_b200.engine import Qwen2Engine

pytestmark = pytest.mark.gpu


def _operator_by_operator(engine, ids):
    cfg = engine.config
    batch, tokens = ids.shape
    x = kernels.b200_embedding(engine.embed, ids.cuda())
    positions = torch.arange(tokens, device="cuda").repeat(batch, 1)
    cosine, sine = kernels.b200_rope_table(positions, engine.inv_freq, engine.dtype)
    norm = dict(epsilon=cfg.rms_norm_eps, round_before_weight=True, numerical_mode=engine.mode)
    cached = []
    for layer in engine.layers:
        qkv = kernels.b200_linear(kernels.b200_rms_norm(x, layer["input_norm"], **norm), layer["qkv_w"], layer["qkv_b"])
        q, k, v = (part.view(batch, tokens, -1, cfg.head_dim).transpose(1, 2)
                   for part in qkv.split([cfg.q_size, cfg.kv_size, cfg.kv_size], dim=-1))
        q, k = kernels.b200_rope(q, k, cosine, sine)
        cached.append((k.transpose(1, 2), v.transpose(1, 2)))
        mixed = kernels.b200_prefill_attention(q, k, v, None, scale=engine.scale, causal=True, numerical_mode=engine.mode)
        x = kernels.b200_linear(mixed.transpose(1, 2).reshape(batch, tokens, -1), layer["o_w"], residual=x, epilogue="residual")
        gated = kernels.b200_linear(kernels.b200_rms_norm(x, layer["post_norm"], **norm), layer["gate_up_w"], epilogue="swiglu")
        x = kernels.b200_linear(gated, layer["down_w"], residual=x, epilogue="residual")
    return kernels.b200_linear(kernels.b200_rms_norm(x[:, -1], engine.final_norm, **norm), engine.lm_head), cached


@pytest.mark.parametrize("dtype,heads,kv_heads,dim,layout,mode", [
    (torch.bfloat16, 14, 2, 64, "contiguous", "fast"), (torch.bfloat16, 6, 3, 128, "contiguous", "fast"),
    (torch.bfloat16, 14, 2, 64, "paged", "fast"), (torch.bfloat16, 4, 2, 64, "contiguous", "pytorch_compatible"),
    (torch.float16, 14, 2, 64, "contiguous", "fast"), (torch.float32, 4, 4, 32, "contiguous", "fast"),
    (torch.bfloat16, 4, 2, 16, "contiguous", "fast"), (torch.float32, 2, 1, 256, "contiguous", "fast")])
@pytest.mark.parametrize("batch,tokens", [(1, 1), (3, 9), (1, 77), (1, 130), (2, 600)])
def test_equals_the_operators_one_by_one(dtype, heads, kv_heads, dim, layout, mode, batch, tokens):
    config = qwen2.Qwen2Config(hidden_size=heads * dim, intermediate_size=3 * heads * dim, num_layers=3, num_heads=heads,
                               num_kv_heads=kv_heads, vocab_size=1000)
    weights = qwen2.make_weights(config, seed=tokens, dtype=dtype, device="cuda", reproducible=False)
    engine = Qwen2Engine(config, weights, batch=batch, capacity=640, kv_layout=layout, numerical_mode=mode)
    ids = torch.randint(0, 1000, (batch, tokens), generator=torch.Generator().manual_seed(batch))
    expected, cached = _operator_by_operator(engine, ids)
    for _ in range(2):  # (the second prompt runs on used caches)
        assert torch.equal(engine.prefill(ids), expected)
        for layer, (keys, values) in enumerate(cached):
            for buffer, rows in ((engine.state.keys[layer], keys), (engine.state.values[layer], values)):
                for b in range(batch):
                    stored = buffer[b] if layout == "contiguous" else buffer[engine.state.block_table[b].long()].flatten(0, 1)
                    assert torch.equal(stored[:tokens], rows[b])
    kernels.runtime().check_status()


@pytest.mark.parametrize("tokens", [65, 77, 130, 300])
def test_a_prompt_is_the_same_bit_for_bit_beside_others(tokens):
    config = qwen2.Qwen2Config(hidden_size=896, intermediate_size=4864, num_layers=2, num_heads=14, num_kv_heads=2,
                               vocab_size=1000)
    weights = qwen2.make_weights(config, seed=3, dtype=torch.bfloat16, device="cuda", reproducible=False)
    ids = torch.randint(0, 1000, (5, tokens), generator=torch.Generator().manual_seed(tokens))
    alone = Qwen2Engine(config, weights, batch=1, capacity=320).prefill(ids[:1], all_logits=True)
    beside = Qwen2Engine(config, weights, batch=5, capacity=320).prefill(ids, all_logits=True)
    assert torch.equal(alone[0], beside[0])


@pytest.mark.parametrize("switch", ["scope", "environment"])
@pytest.mark.parametrize("batch,tokens", [(1, 9), (1, 77), (2, 300)])
def test_named_variants_reach_the_layers(batch, tokens, switch, monkeypatch):
    config = qwen2.Qwen2Config(hidden_size=896, intermediate_size=2048, num_layers=2, num_heads=14, num_kv_heads=2,
                               vocab_size=1000)
    weights = qwen2.make_weights(config, seed=tokens, dtype=torch.bfloat16, device="cuda", reproducible=False)
    engine = Qwen2Engine(config, weights, batch=batch, capacity=320)
    ids = torch.randint(0, 1000, (batch, tokens), generator=torch.Generator().manual_seed(batch))
    own = engine.prefill(ids).clone()
    scope = contextlib.nullcontext()
    if switch == "scope":
        scope = kernels.kernel_variants(linear="mma.sync", prefill_attention="mma.sync")
    else:
        monkeypatch.setenv("B200_LINEAR_PATH", "mma.sync")
        monkeypatch.setenv("B200_PREFILL_ATTENTION_PATH", "mma.sync")
    with scope:
        expected, cached = _operator_by_operator(engine, ids)
        assert torch.equal(engine.prefill(ids), expected)
        for layer, (keys, values) in enumerate(cached):
            assert torch.equal(engine.state.keys[layer][:, :tokens], keys)
            assert torch.equal(engine.state.values[layer][:, :tokens], values)
    assert not torch.equal(own, expected)  # (the variants sum K in other orders)
    kernels.runtime().check_status()


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_named_variants_reach_the_decode_step(dtype, monkeypatch):
    config = qwen2.Qwen2Config(hidden_size=256, intermediate_size=512, num_layers=2, num_heads=4, num_kv_heads=2,
                               vocab_size=1000)
    weights = qwen2.make_weights(config, seed=4, dtype=dtype, device="cuda", reproducible=False)
    engine = Qwen2Engine(config, weights, batch=2, capacity=64)
    engine.prefill(torch.randint(0, 1000, (2, 5), generator=torch.Generator().manual_seed(2)))
    modes, linear = [], kernels.b200_linear

    def recorded(*args, **options):
        modes.append(_lib.load().b200_get_launch_mode())
        return linear(*args, **options)

    monkeypatch.setattr(kernels, "b200_linear", recorded)
    with kernels.kernel_variants(linear="mma.sync"):
        engine.decode_step()
    engine.decode_step()
    half = len(modes) // 2
    assert half > 0 and all(mode & _lib.LAUNCH_LINEAR_WARP_LEVEL for mode in modes[:half])
    assert not any(mode & _lib.LAUNCH_LINEAR_WARP_LEVEL for mode in modes[half:])


def _refused(engine, ids, **changed):
    cfg = engine.config
    batch, tokens = ids.shape
    cosine, sine = kernels.b200_rope_table(torch.arange(tokens, device="cuda").repeat(batch, 1), engine.inv_freq, engine.dtype)
    operands = dict(x=kernels.b200_embedding(engine.embed, ids), layers=engine.layers, keys=engine.state.keys,
                    values=engine.state.values, cosine=cosine, sine=sine, positions=engine.positions,
                    block_table=engine.state.block_table if engine.paged else None)
    operands.update(changed)
    with pytest.raises(ValueError):
        kernels.b200_qwen2_prompt_layers(**operands, q_heads=cfg.num_heads, scale=engine.scale, epsilon=cfg.rms_norm_eps)


def test_operands_are_checked_before_any_launch():
    config = qwen2.Qwen2Config(hidden_size=128, intermediate_size=256, num_layers=2, num_heads=2, num_kv_heads=2,
                               vocab_size=100)
    weights = qwen2.make_weights(config, seed=1, dtype=torch.bfloat16, device="cuda", reproducible=False)
    ids = torch.zeros(2, 5, dtype=torch.int64, device="cuda")
    engine = Qwen2Engine(config, weights, batch=2, capacity=32)
    for name in ("input_norm", "qkv_w", "qkv_b", "o_w", "post_norm", "gate_up_w", "down_w"):
        on_host = [engine.layers[0], dict(engine.layers[1], **{name: engine.layers[1][name].cpu()})]
        _refused(engine, ids, layers=on_host)
        _refused(engine, ids, layers=[engine.layers[0], dict(engine.layers[1], **{name: engine.layers[1][name][:-1]})])
    _refused(engine, ids, keys=engine.state.keys[:1])
    _refused(engine, ids, values=engine.state.values[:1])
    _refused(engine, ids, layers=engine.layers[:1])
    _refused(engine, ids, positions=engine.positions.int())
    _refused(engine, ids, positions=torch.zeros(4, dtype=torch.int64, device="cuda")[::2])
    _refused(engine, ids, x=kernels.b200_embedding(engine.embed, ids)[0])
    paged = Qwen2Engine(config, weights, batch=2, capacity=256, kv_layout="paged")
    table = paged.state.block_table
    for wrong in (table.long(), table[:1], table[0], table.cpu(), table.repeat(1, 2)[:, ::2]):
        _refused(paged, ids, block_table=wrong)
