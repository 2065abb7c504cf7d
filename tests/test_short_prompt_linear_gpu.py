"""Projections of short prompts against the 64-bit product at the lines of the dispatch: too few tiles for the persistent
kernel, and the row counts around it.

Bound of an element: K 2^-23 sum |x w| for fp32 sums in any order, and half an ulp (at most 2^-8 of a bf16 value, 2^-11
of an fp16 value) for every rounding: one, or two in front of a residual."""

import pytest
import torch

import llm_compiler_b200 as b200
from llm_compiler_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("k,n", [(896, 1152), (4864, 896), (896, 260), (72, 64), (896, 258)])
@pytest.mark.parametrize("m", [65, 77, 128, 129, 500, 1023, 1024, 1030, 2048])
def test_linear(m, k, n, dtype):
    g = torch.Generator().manual_seed(m + k + n)
    x = torch.randn(m, k, generator=g).to(dtype).cuda()
    w = (torch.randn(n, k, generator=g) * k ** -0.5).to(dtype).cuda()
    bias, residual = torch.randn(n, generator=g).to(dtype).cuda(), torch.randn(m, n, generator=g).to(dtype).cuda()
    half = 1.01 * 2.0 ** (-8 if dtype == torch.bfloat16 else -11)  # (second order terms)
    exact = x.double() @ w.double().T
    sums = k * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T) + 2.0 ** -24  # (an fp16 subnormal)
    for b, r in ((None, None), (bias, None), (bias, residual), (None, residual)):
        inner = exact if b is None else exact + b.double()
        total = inner if r is None else inner + r.double()
        bound = sums + 2.0 ** -22 * (inner.abs() + total.abs()) + half * (total.abs() + 2 * sums)
        if r is not None:
            bound = bound + half * (inner.abs() + sums)
        out = b200.b200_linear(x, w, b, residual=r, epilogue="none" if r is None else "residual")
        assert ((out.double() - total).abs() <= bound).all()
        assert torch.equal(out, b200.b200_linear(x, w, b, residual=r, epilogue="none" if r is None else "residual"))
    # rows of a wider matrix
    wide = torch.randn(m, k + 8, generator=g).to(dtype).cuda()
    strided = b200.b200_linear(wide[:, 8:], w)
    exact = wide[:, 8:].double() @ w.double().T
    sums = k * 2.0 ** -23 * (wide[:, 8:].double().abs() @ w.double().abs().T) + 2.0 ** -24
    assert ((strided.double() - exact).abs() <= sums + half * (exact.abs() + sums)).all()
    kernels.runtime().check_status()
