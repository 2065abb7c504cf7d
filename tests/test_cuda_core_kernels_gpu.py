"""The CUDA-core kernels (fp32, fp16 without 16-byte rows, head sizes 16 / 32 / 256) at the edges of their tiles, splits
and vector loads, against 64-bit products.

Tolerances: a sum of K products in fp32 whose longest chain of additions is `chain` errs by at most chain x 2^-24 of the
summands' absolute sum; attention adds the exponentials (4 ulp of fp32) and one quotient; a 16-bit result is rounded
once (three times in a SwiGLU)."""

import math

import pytest
import torch

import llm_compiler_b200 as b200
from llm_compiler_b200 import kernels

pytestmark = pytest.mark.gpu

ULP = {torch.float32: 2.0 ** -24, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def unaligned(tensor):
    """The same values one element behind a 16-byte boundary."""
    storage = torch.empty(tensor.numel() + 8, dtype=tensor.dtype, device=tensor.device)
    view = storage[1:1 + tensor.numel()].view(tensor.shape)
    view.copy_(tensor)
    return view


# the streaming kernel's row tiles (8, up to 40 rows), K splits and shortest K for many columns, the tiled kernel's 64 x 64 x 16 tiles, with and
# without a cluster over K, vector and scalar loads
@pytest.mark.parametrize("epilogue", ["none", "residual", "swiglu"])
@pytest.mark.parametrize("m,k,n", [(1, 4, 2), (1, 896, 896), (4, 4864, 896), (8, 260, 130), (9, 1028, 6), (16, 520, 9728), (4, 3588, 34),
                                   (40, 4864, 900), (41, 4864, 900), (17, 380, 9728), (17, 384, 9728), (40, 132, 9728),
                                   (17, 896, 1152), (64, 7, 66), (65, 4864, 130), (200, 270, 62), (300, 4864, 896)])
def test_linear_fp32(m, k, n, epilogue):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x, w = (torch.randn(*s, generator=g, device="cuda") for s in ((m, k), (n, k)))
    w *= k ** -0.5
    bias = torch.randn(n, generator=g, device="cuda")
    residual = torch.randn(m, n, generator=g, device="cuda") if epilogue == "residual" else None
    y = x.double() @ w.double().T + bias.double()
    bound = (k / 16 + 40) * ULP[torch.float32] * (x.double().abs() @ w.double().abs().T) + 4 * ULP[torch.float32] * y.abs()
    if epilogue == "residual":
        y, bound = y + residual, bound + 2 * ULP[torch.float32] * (y + residual).abs()
    if epilogue == "swiglu":
        gate, up = y[:, 0::2], y[:, 1::2]
        # |d silu / d gate| <= 1.1; the exponential and the quotient add 8 ulp of the result
        bound = 1.1 * bound[:, 0::2] * up.abs() + (gate * torch.sigmoid(gate)).abs() * bound[:, 1::2]
        y = gate * torch.sigmoid(gate) * up
        bound = bound + 8 * ULP[torch.float32] * y.abs()
    for source in (x, unaligned(x)):
        out = b200.b200_linear(source, w, bias, residual=residual, epilogue=epilogue)
        assert ((out.double() - y).abs() <= bound + 1e-30).all()


def attention(q, k, v, visible, mask, scale):
    """q [H, D], k [C, G, D] -> [H, D] over the first `visible` keys, in 64 bits."""
    heads, groups = q.shape[0], k.shape[1]
    scores = torch.einsum("gnd,cgd->gnc", q.double().view(groups, -1, q.shape[1]), k[:visible].double()) * scale
    if mask is not None:
        scores = scores + mask[:visible].double()
    return torch.einsum("gnc,cgd->gnd", torch.softmax(scores, -1), v[:visible].double()).reshape(heads, -1)


def sum_error(d, scale, q, k, longest):
    """Relative error of a sum of probabilities times values: that of a score, absolutely, and of the exponential, in a
    probability and in the denominator; then a sum over keys. Of finite operands."""
    score = (d + 2) * ULP[torch.float32] * scale * q.double().norm(dim=-1).max() * k.double().norm(dim=-1).max()
    return 2 * score + (longest + 16) * ULP[torch.float32]


def attention_bound(dtype, d, scale, q, k, v, longest):
    return (sum_error(d, scale, q, k, longest) + 2 * ULP[dtype]) * v.double().abs().max()


def decode_limits(dtype, scale, q, k, v, n, mask, expected):
    """Of every element: the sums' error on the absolute values, one rounding, half a step of fp16's subnormals. A result
    that is 1 % off in one head, or lacks a part of the context, is outside."""
    size = attention(q, k, v.abs(), n, mask, scale)
    return sum_error(q.shape[1], scale, q, k[:n], n) * size + 1.01 * ULP[dtype] * expected.abs() + 2.0 ** -25


@pytest.mark.parametrize("dtype,d,groups", [(torch.float32, 64, 7), (torch.float32, 128, 9), (torch.float16, 64, 1),
                                            (torch.float16, 128, 8), (torch.bfloat16, 16, 2), (torch.float16, 32, 16),
                                            (torch.float32, 256, 3), (torch.bfloat16, 256, 8)])
def test_decode_attention(dtype, d, groups):
    g = torch.Generator(device="cuda").manual_seed(d + groups)
    lengths, capacity, kv_heads, scale = [1, 63, 64, 65, 0, 700, 511], 701, 2, d ** -0.5
    batch = len(lengths)
    q = torch.randn(batch, kv_heads * groups, 1, d, generator=g, device="cuda").to(dtype)
    k, v = (torch.randn(batch, capacity, kv_heads, d, generator=g, device="cuda").to(dtype) for _ in range(2))
    for b, n in enumerate(lengths):
        k[b, n:], v[b, n:] = torch.nan, torch.inf
    masks = [None, torch.zeros(batch, 1, 1, capacity, device="cuda")]
    masks[1][:, :, :, 3::7] = -torch.inf
    masks[1][5] = torch.finfo(torch.float32).min  # every key masked alike: they count alike
    for mask in masks:
        for kept in (k, unaligned(k)):
            out = b200.b200_decode_attention(q, kept, v, torch.tensor(lengths, device="cuda"), mask, scale=scale)
            for b, n in enumerate(lengths):
                actual = out[b, :, 0].double()
                if n == 0:
                    assert actual.isnan().all()
                    continue
                row, own = None if mask is None else mask[b, 0, 0], q[b, :, 0]
                if b == 5 and row is not None:  # what the lowest value leaves of the scores: nothing
                    row, own = torch.zeros_like(row), torch.zeros_like(own)
                expected = attention(own, k[b], v[b], n, row, scale)
                assert ((actual - expected).abs() <= decode_limits(dtype, scale, own, k[b], v[b], n, row, expected)).all()
    kernels.runtime().check_status()


@pytest.mark.parametrize("dtype,d", [(torch.float32, 64), (torch.float32, 128), (torch.bfloat16, 16),
                                     (torch.float16, 32), (torch.float32, 256), (torch.bfloat16, 256)])
@pytest.mark.parametrize("t", [1, 16, 32, 33, 63, 65, 200])
def test_prefill_attention(t, dtype, d):
    g = torch.Generator(device="cuda").manual_seed(d + t)
    batch, heads, kv_heads, scale = 2, 4, 2, d ** -0.5
    q = torch.randn(batch, t, heads, d, generator=g, device="cuda").to(dtype).transpose(1, 2)
    k, v = (torch.randn(batch, kv_heads, t, d, generator=g, device="cuda").to(dtype) for _ in range(2))
    mask = torch.where(torch.rand(batch, 1, t, t, generator=g, device="cuda") < 0.3, -torch.inf, 0.5)
    mask[:, :, t // 2] = -torch.inf
    bound = attention_bound(dtype, d, scale, q, k, v, t)
    causal = torch.full((t, t), -torch.inf, device="cuda").triu(1).double()
    for own in (None, mask):
        bias = causal if own is None else own.double()
        scores = torch.einsum("bgntd,bgsd->bgnts", q.double().reshape(batch, kv_heads, -1, t, d), k.double()) * scale
        weights = torch.softmax(scores + (bias if own is None else bias[:, :, None]), -1)
        expected = torch.einsum("bgnts,bgsd->bgntd", weights, v.double()).reshape(batch, heads, t, d)
        for kept in (k, unaligned(k)):
            out = b200.b200_prefill_attention(q, kept, v, own, scale=scale, causal=own is None).double()
            assert torch.equal(out.isnan(), expected.isnan())
            assert (out - expected).nan_to_num().abs().max() <= bound


def test_prefill_attention_fp32_does_not_read_values_that_a_row_does_not_see():
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v = (torch.randn(1, 2, 100, 64, generator=g, device="cuda") for _ in range(3))
    v[0, 1, 70], k[0, 0, 90] = float("inf"), float("nan")
    out = b200.b200_prefill_attention(q, k, v, None, scale=0.125, causal=True)
    assert out[0, 1, :70].isfinite().all() and not out[0, 1, 70:].isfinite().any()
    assert out[0, 0, :90].isfinite().all()
