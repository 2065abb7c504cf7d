"""Projections of 65 rows and more in tiles of 64 or 128 rows and 32, 64 or 128 columns, on both sides of the lines between
the tiles and between short rings and long ones (148 tiles), K in fewer blocks than a ring has stages and in more: a tile's
sums do not depend on its size or its ring, so every row and column equals that of a call on the other side of a line bit
for bit."""

import pytest
import torch

from llm_compiler_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("epilogue", ["none", "residual", "swiglu"])
# tiles: 2 x 74 and 2 x 75 of 64 columns; 1 x 148 and 1 x 149 of 64; 5 x 28 and 5 x 30 of 128; ragged rows and columns;
# 64-row tiles: 3 x 49 of 32 columns and 3 x 50; 2 x 74 of 64 columns and 2 x 75
@pytest.mark.parametrize("m,k,n,fewer", [(130, 896, 4800, 4736), (77, 64, 9500, 9470), (128, 456, 9536, 9472),
                                         (515, 1032, 3840, 3584), (600, 8, 3840, 3520),
                                         (130, 1096, 1600, 1568), (65, 328, 4800, 4736), (129, 4864, 912, 896)])
def test_sums_do_not_depend_on_the_ring(m, k, n, fewer, epilogue, dtype):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x, w = ((torch.randn(*s, generator=g, device="cuda") * k ** -0.25).to(dtype) for s in ((m, k), (n, k)))
    bias = torch.randn(n, generator=g, device="cuda").to(dtype)
    residual = torch.randn(m, n, generator=g, device="cuda").to(dtype) if epilogue == "residual" else None
    full = kernels.b200_linear(x, w, bias, residual=residual, epilogue=epilogue)
    part = kernels.b200_linear(x, w[:fewer], bias[:fewer], epilogue=epilogue,
                               residual=None if residual is None else residual[:, :fewer].contiguous())
    assert torch.equal(full[:, :part.shape[1]], part)
    if epilogue == "none":
        exact = x.double() @ w.double().T + bias.double()
        # one rounding of the result, and sums in fp32 in one chain of K / 16 products
        bound = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * exact.abs() + \
            (k / 16 + 8) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T) + 1e-6
        assert ((full.double() - exact).abs() <= bound).all()


# K blocks a slice (64 rows: 6 or 4 stages up to 7 blocks, 12 or 8 from 8 on): 7, 8 (one of them ragged), 12, 15, 15 in one slice
@pytest.mark.parametrize("k,n", [(448, 18944), (4096, 1024), (4040, 1016), (3584, 3584), (8200, 2048), (904, 18944)])
@pytest.mark.parametrize("m", [9, 64])
def test_partial_sums_do_not_depend_on_the_ring(m, k, n):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = (torch.randn(65, k, generator=g, device="cuda") * k ** -0.25).bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.25).bfloat16()
    taller = kernels.b200_linear_partial(x, w)  # 128-row tiles, short rings
    few = kernels.b200_linear_partial(x[:m], w)
    assert few.shape[0] == taller.shape[0] and torch.equal(few, taller[:, :m])
    # fp32 sums in one chain of products a slice, the slices added in 64 bits
    exact = x[:m].double() @ w.double().T
    bound = (k / 16 + 8) * 2.0 ** -23 * (x[:m].double().abs() @ w.double().abs().T) + 1e-6
    assert ((few.double().sum(0) - exact).abs() <= bound).all()


# CTAs: 152 against 148 of 8 blocks; 160 against 145 of 13; 158 against 148 of 23
@pytest.mark.parametrize("k,n,fewer", [(960, 4864, 4736), (4096, 4096, 3712), (2880, 10032, 9472)])
def test_partial_sums_of_more_ctas_than_sms_are_no_second_wave(k, n, fewer):
    """A few more columns take a few more CTAs, which short rings hold beside the others: the time grows by the columns (8 % at
    most here) and what two CTAs on an SM take from one another (0.94, 1.15 and 1.23 of the time in all), where long rings, one
    CTA an SM, add a wave (1.53, 1.50 and 1.45)."""

    def microseconds(columns):
        weights = [(torch.randn(columns, k, device="cuda") * k ** -0.5).bfloat16() for _ in range(2 + 300_000_000 // (2 * k * n))]
        x = torch.randn(48, k, device="cuda").bfloat16()
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream), kernels.launch_mode(programmatic=True, constant_weights=True):
            kernels.b200_linear_partial(x, weights[0])
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                for w in weights:
                    kernels.b200_linear_partial(x, w)
        graph.replay()
        best = float("inf")
        for _ in range(10):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            graph.replay()
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end))
        return best * 1e3 / len(weights)

    few, more = microseconds(fewer), microseconds(n)
    print(f"{fewer}: {few:.2f} us, {n}: {more:.2f} us")
    assert more <= 1.35 * few
