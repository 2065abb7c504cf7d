"""The RMS norm inside the projection behind it (a few fp32 rows), against 64-bit products.

Tolerance of a normed projection: a sum of K products in fp32, whose longest chain of additions has `chain` terms, errs
by at most chain x 2^-24 of the summands' absolute sum; the product with the norm's weight, the mean of the squares, its
root and the product with it add 8 roundings."""

import pytest
import torch

from llm_compiler_b200 import kernels

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -24


# one CTA and a cluster along K, ragged K, columns and rows, row tiles of 4 and 8, the most rows
@pytest.mark.parametrize("epilogue", ["none", "swiglu"])
@pytest.mark.parametrize("m,k,n", [(1, 4, 2), (1, 896, 1152), (4, 896, 9728), (4, 4864, 900), (5, 132, 34), (8, 3584, 514),
                                   (9, 1028, 6), (40, 4864, 66)])
def test_norm_in_the_projection(m, k, n, epilogue):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = 3.0 * torch.randn(m, k, generator=g, device="cuda")
    w = torch.randn(n, k, generator=g, device="cuda") * k ** -0.5
    norm = torch.rand(k, generator=g, device="cuda") + 0.5
    bias = torch.randn(n, generator=g, device="cuda")
    wide = torch.full((m, k + 8), float("nan"), device="cuda")
    wide[:, :k] = x
    h = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * norm.double()
    y = h @ w.double().T + bias.double()
    bound = (k / 16 + 48) * ULP * (h.abs() @ w.double().abs().T) + 4 * ULP * y.abs()
    if epilogue == "swiglu":
        gate, up = y[:, 0::2], y[:, 1::2]
        # |d silu / d gate| <= 1.1; the exponential and the quotient add 8 ulp of the result
        silu = gate * torch.sigmoid(gate)
        bound = 1.1 * bound[:, 0::2] * up.abs() + silu.abs() * bound[:, 1::2]
        y = silu * up
        bound = bound + 8 * ULP * y.abs()
    for source in (x, wide[:, :k]):
        out = kernels.b200_rms_norm_linear(source, norm, w, bias, epsilon=1e-6, epilogue=epilogue)
        assert ((out.double() - y).abs() <= bound + 1e-30).all()


def test_norm_in_the_projection_leaves_other_calls_alone():
    x, w, norm = (torch.randn(*s, device="cuda") for s in ((41, 896), (64, 896), (896,)))
    assert kernels.b200_rms_norm_linear(x, norm, w, epsilon=1e-6) is None  # too many rows
    assert kernels.b200_rms_norm_linear(x[:4, 1:893], norm[:892], w[:, :892].contiguous(), epsilon=1e-6) is None  # no 16-byte rows
    assert kernels.b200_rms_norm_linear(x[:4].bfloat16(), norm.bfloat16(), w.bfloat16(), epsilon=1e-6) is None
