"""16-bit projections of up to 8 rows (csrc/linear_rows.cu) against the 64-bit product, in every form a decode step has.

The bound of an element is what fp32 sums in any order may be off, K 2^-23 sum |x w|, plus half an ulp of the result
type for every rounding of the result: at most 2^-8 of it for bf16 with its 8 significant bits, 2^-11 for fp16 with 11
(two roundings where a sum is rounded in front of a residual).
"""

import pytest
import torch

import llm_compiler_b200 as b200
from llm_compiler_b200 import kernels

pytestmark = pytest.mark.gpu

# K: one lane's piece, less than a chunk of 32, ends inside a chunk, one ring, several rings, a cluster along K;
# N: a part of a column tile, tiles and a remainder, more tiles than the GPU holds at once
SIZES = [(1, 8, 4), (3, 40, 20), (8, 896, 1152), (5, 904, 260), (8, 4864, 896), (2, 3592, 4612), (7, 18944, 64),
         (4, 896, 15000)]


def _operands(m, k, n, dtype):
    g = torch.Generator().manual_seed(m * 31 + k * 7 + n)
    wide = torch.randn(m, k + 24, generator=g).to(dtype).cuda()  # rows of a wider matrix
    w = (torch.randn(n, k, generator=g) * k ** -0.5).to(dtype).cuda()
    return wide[:, 8:8 + k], w, torch.randn(m, n, generator=g).to(dtype).cuda(), torch.randn(n, generator=g).to(dtype).cuda()


def _product(x, w):
    exact = x.double() @ w.double().T
    return exact, w.shape[1] * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)


def _half_ulp(dtype):
    return 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11


def _check(actual, exact, bound):
    assert ((actual.double() - exact).abs() <= bound).all()


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,k,n", SIZES)
def test_linear(m, k, n, dtype, early):
    x, w, residual, bias = _operands(m, k, n, dtype)
    half, (exact, sums) = _half_ulp(dtype), _product(x, w)
    half *= 1.01  # (second order terms)
    with kernels.launch_mode(programmatic=early, constant_weights=early):
        plain = b200.b200_linear(x, w)
        biased = b200.b200_linear(x, w, bias)
        added = b200.b200_linear(x, w, residual=residual, epilogue="residual")
        gated = b200.b200_linear(x, w, epilogue="swiglu")
    tiny = 2.0 ** -24  # an fp16 subnormal is off by up to 2^-25
    _check(plain, exact, sums + half * (exact.abs() + sums) + tiny)
    shifted = exact + bias.double()
    _check(biased, shifted, sums + half * (shifted.abs() + 2 * sums) + 2.0 ** -23 * shifted.abs() + tiny)
    total = exact + residual.double()
    _check(added, total, sums + half * (exact.abs() + total.abs() + 2 * sums) + 2.0 ** -23 * total.abs() + 2 * tiny)
    gate, up = exact[:, 0::2], exact[:, 1::2]
    silu = gate * torch.sigmoid(gate)
    # gate, up, silu and the product are rounded; the slope of silu is at most 1.1
    off_gate = 1.1 * (sums[:, 0::2] + half * gate.abs()) + half * silu.abs() + 2.0 ** -20 * silu.abs() + 2 * tiny
    off_up = sums[:, 1::2] + half * up.abs() + tiny
    bound = off_gate * up.abs() + silu.abs() * off_up + off_gate * off_up
    _check(gated, silu * up, bound + half * ((silu * up).abs() + bound) + tiny)
    kernels.runtime().check_status()


@pytest.mark.parametrize("m,k,n", SIZES)
def test_forms_of_the_decode_chain(m, k, n):
    x, w, residual, _ = _operands(m, k, n, torch.bfloat16)
    half, (exact, sums) = 1.01 * _half_ulp(torch.bfloat16), _product(x, w)
    partials, squares = kernels.b200_linear_partial(x, w, row_squares=True)
    assert squares.shape == partials.shape[:2]
    _check(partials.sum(0), exact, sums)
    exact_squares = x.double().square().sum(-1)
    _check(squares.sum(0), exact_squares, k * 2.0 ** -23 * exact_squares)
    total = exact + residual.double()
    out = kernels.b200_linear_splitk_residual(x, w, residual)
    _check(out, total, sums + half * (exact.abs() + total.abs() + 2 * sums))
    scale = torch.rsqrt(exact_squares / k + 1e-6)[:, None]
    normed = exact * scale
    for given in (None, squares):
        _check(kernels.b200_linear_rms_input(x, w, epsilon=1e-6, row_squares=given), normed,
               1.01 * sums * scale + (half + k * 2.0 ** -23) * normed.abs())
    kernels.runtime().check_status()


# the sizes above whose rows take few blocks, the projections of a Qwen2-0.5B layer, longer K, more
# column tiles than the GPU holds at once, and one matrix over the limit
CHAIN = [(1, 896, 1152), (8, 896, 896), (3, 4864, 896), (5, 904, 1092), (2, 3584, 2308), (7, 3584, 2800), (4, 18944, 512),
         (6, 896, 9728), (2, 264, 30000), (8, 72, 2500), (1, 896, 12000),
         (8, 3072, 3072), (8, 3072, 3076)]  # (on both sides of the largest matrix)


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("m,k,n", CHAIN)
def test_a_row_is_the_same_bit_for_bit_in_a_larger_batch(m, k, n, early):
    """16 rows run on the tcgen05 kernels; the same rows in a batch of up to 8 give the same bits in every form."""
    x, w, residual, bias = _operands(16, k, n, torch.bfloat16)
    few = slice(0, m)
    with kernels.launch_mode(programmatic=early, constant_weights=early):
        many = kernels.b200_linear_partial(x, w, row_squares=True)
        mine = kernels.b200_linear_partial(x[few], w, row_squares=True)
        assert torch.equal(mine[0], many[0][:, few]) and torch.equal(mine[1], many[1][:, few])
        assert torch.equal(kernels.b200_linear_partial(x[few], w), many[0][:, few])
        assert torch.equal(kernels.b200_linear_splitk_residual(x[few], w, residual[few]),
                           kernels.b200_linear_splitk_residual(x, w, residual)[few])
        out, squares = kernels.b200_linear_splitk_residual(x, w, residual, row_squares=True)
        out_few, squares_few = kernels.b200_linear_splitk_residual(x[few], w, residual[few], row_squares=True)
        assert torch.equal(out_few, out[few])
        assert (squares is None) == (squares_few is None)
        if squares is not None:
            assert torch.equal(squares_few, squares[:, few])
        given = torch.rand((112, 16), device="cuda") + 0.1
        for epilogue in ("none", "swiglu"):
            assert torch.equal(kernels.b200_linear(x[few], w, epilogue=epilogue), kernels.b200_linear(x, w, epilogue=epilogue)[few])
            for parts in (None, given):
                assert torch.equal(
                    kernels.b200_linear_rms_input(x[few], w, epsilon=1e-6, epilogue=epilogue,
                                                  row_squares=None if parts is None else parts[:, few].contiguous()),
                    kernels.b200_linear_rms_input(x, w, epsilon=1e-6, epilogue=epilogue, row_squares=parts)[few])
        assert torch.equal(kernels.b200_linear(x[few], w, bias), kernels.b200_linear(x, w, bias)[few])
    kernels.runtime().check_status()
