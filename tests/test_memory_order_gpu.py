"""Kernels whose operands are written while they are already resident, or reused while the tensor core may still read."""

import pytest
import torch

import llm_compiler_b200 as b200
from llm_compiler_b200 import hybrid_kernels as hk
from llm_compiler_b200 import _lib, kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [64, 128])
def test_prompt_attention_whose_reference_maximum_stays(size):
    """Scores within 8 of the first tile's maximum (log2 domain): no tile moves O, so that the stores of P follow the wait for
    the product before directly, 17 times a group. Many heads, so that SMs run different query blocks side by side."""

    g = torch.Generator(device="cuda").manual_seed(size)
    tokens, heads, kv_heads = 2100, 14, 2
    q, k, v = (torch.randn(1, h, tokens, size, generator=g, device="cuda").bfloat16() for h in (heads, kv_heads, kv_heads))
    first = b200.b200_prefill_attention(q, k, v, None, scale=size ** -0.5, causal=True)
    for _ in range(20):
        assert torch.equal(b200.b200_prefill_attention(q, k, v, None, scale=size ** -0.5, causal=True), first)
    kernels.runtime().check_status()
    seen = torch.ones(tokens, tokens, dtype=torch.bool, device="cuda").tril()
    for head in (0, 6, 13):
        scores = (q[0, head].double() @ k[0, head // 7].double().T * size ** -0.5).masked_fill(~seen, -torch.inf)
        weights, values = torch.softmax(scores, -1), v[0, head // 7].double()
        exact = weights @ values
        # probabilities and results are rounded to bf16 once each: 8 significant bits, so by 2^-8 of the value at most
        # (2^-9 just below a power of two); fp32 sums and exponentials err far less
        bound = 1.01 * 2.0 ** -8 * (weights @ values.abs() + exact.abs()) + 1e-6
        assert ((first[0, head].double() - exact).abs() <= bound).all()


def projection(x, w, out):
    """b200_linear into a buffer of the caller's."""

    code = _lib.load().b200_linear(x.data_ptr(), w.data_ptr(), None, None, out.data_ptr(), x.shape[0], x.shape[1],
                                   w.shape[0], x.shape[1], _lib.BF16, _lib.EPILOGUE_NONE, None, 0,
                                   kernels.runtime().status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert code == 0


@pytest.mark.parametrize("rows", [1, 16, 64])
def test_tokens_chosen_behind_a_projection_in_flight(rows):
    """The cluster form is resident while the projection writes the logits: what the buffer held before is never chosen."""

    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 896, generator=g, device="cuda").bfloat16()
    w = torch.randn(151936, 896, generator=g, device="cuda").bfloat16()
    logits = torch.empty(rows, 151936, dtype=torch.bfloat16, device="cuda")
    projection(x, w, logits)
    want = kernels.b200_argmax(logits)
    chosen = torch.empty_like(want)
    for turn in range(20):
        logits.fill_(0)
        logits[:, turn * 7901 % 151936] = 3e4
        torch.cuda.synchronize()
        with kernels.launch_mode(programmatic=True, constant_weights=True):
            projection(x, w, logits)
            kernels.b200_argmax(logits, chosen)
        assert torch.equal(chosen, want)
    kernels.runtime().check_status()


# 16-row and 64-row tiles, CTAs with an SM each (long rings) and without
@pytest.mark.parametrize("rows,heads,k,n", [(1, 16, 512, 128), (16, 14, 256, 192), (32, 16, 512, 128), (64, 40, 128, 512)])
def test_per_head_products_behind_a_projection_in_flight(rows, heads, k, n):
    """W comes ahead of the dependency wait, x does not: what the buffer of x held before is never multiplied."""

    g = torch.Generator(device="cuda").manual_seed(rows)
    rows_in = torch.randn(rows, 896, generator=g, device="cuda").bfloat16()
    w_in = torch.randn(heads * k, 896, generator=g, device="cuda").bfloat16()
    w = torch.randn(heads, n, k, generator=g, device="cuda").bfloat16()
    x = torch.empty(rows, heads, k, dtype=torch.bfloat16, device="cuda")
    projection(rows_in, w_in, x)
    want = hk.head_linear(x, w)
    for _ in range(20):
        x.fill_(float("nan"))
        torch.cuda.synchronize()
        with kernels.launch_mode(programmatic=True, constant_weights=True):
            projection(rows_in, w_in, x)
            y = hk.head_linear(x, w)
        assert torch.equal(y, want)
    kernels.runtime().check_status()
