"""fp16 projections and prompt attention on the tensor cores, against the CUDA-core kernels that the same calls take
when a base address is not a multiple of 16 bytes, and against the oracle.

Tolerance: either kernel sums exact fp16 products in fp32 (order: K x 2^-24 of the summands, below a thousandth of what
follows) and rounds a result to 11 bits; a SwiGLU rounds three factors, attention one quotient. 4 x 2^-11 of the
largest result covers the worst of them."""

import math

import pytest
import torch

from oracle import serve_ops
import llm_compiler_b200 as b200
from llm_compiler_b200 import _lib, kernels

pytestmark = pytest.mark.gpu

BOUND = 4 * 2.0 ** -11


def unaligned(tensor):
    """The same values one element behind a 16-byte boundary."""
    storage = torch.empty(tensor.numel() + 8, dtype=tensor.dtype, device=tensor.device)
    view = storage[1:1 + tensor.numel()].view(tensor.shape)
    view.copy_(tensor)
    assert view.data_ptr() % 16
    return view


def close(actual, expected):
    actual, expected = actual.float().cpu(), expected.float().cpu()
    assert torch.equal(torch.isnan(actual), torch.isnan(expected))
    assert torch.equal(actual.isinf(), expected.isinf())
    actual, expected = (t[expected.isfinite()] for t in (actual, expected))
    if expected.numel():
        assert (actual - expected).abs().max().item() <= BOUND * expected.abs().max().item()


# around the row tiles (16 / 32 / 64 warp-level, 64, 128), the persistent kernel's first size, few and many columns,
# remainders of the 64-wide K blocks
@pytest.mark.parametrize("epilogue", ["none", "bias", "residual", "swiglu"])
@pytest.mark.parametrize("m,k,n", [(1, 8, 16), (1, 896, 896), (16, 72, 130), (17, 896, 9728), (64, 136, 2400),
                                   (65, 896, 1152), (128, 4864, 896), (129, 72, 264), (1023, 200, 896),
                                   (1024, 896, 1152), (1100, 72, 904)])
def test_linear(m, k, n, epilogue):
    g = torch.Generator().manual_seed(m + k + n)
    x, w = torch.randn(m, k, generator=g).half().cuda(), (0.1 * torch.randn(n, k, generator=g)).half().cuda()
    bias = torch.randn(n, generator=g).half().cuda() if epilogue in ("bias", "swiglu") else None
    residual = torch.randn(m, n, generator=g).half().cuda() if epilogue == "residual" else None
    options = dict(residual=residual, epilogue="none" if epilogue == "bias" else epilogue)
    close(b200.b200_linear(x, w, bias, **options), b200.b200_linear(unaligned(x), w, bias, **options))
    kernels.runtime().check_status()


def test_linear_overflow_stays_in_its_row_and_column():
    x, w = torch.full((70, 64), 100.0).half().cuda(), torch.full((136, 64), 1.0).half().cuda()
    x[3] = 60000.0  # the sum overflows fp16
    x[5, 7] = float("inf")
    w[9, 0] = float("nan")
    close(b200.b200_linear(x, w), b200.b200_linear(unaligned(x), w))


@pytest.mark.parametrize("m", [8, 16, 70, 1100])  # streamed rows, warp-level, tcgen05, the persistent kernel
def test_swiglu_of_every_gate_is_that_of_the_cuda_cores_bit_for_bit(m):
    gates = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.float16)
    for part in gates.view(-1, 4096):
        bias = torch.stack([part, torch.full_like(part, 1.5)], dim=1).flatten().cuda()
        x, w = torch.zeros(m, 64).half().cuda(), torch.zeros(8192, 64).half().cuda()
        tensor_cores, cuda_cores = (b200.b200_linear(rows, w, bias, epilogue="swiglu") for rows in (x, unaligned(x)))
        assert torch.equal(tensor_cores.isnan(), cuda_cores.isnan())
        assert torch.equal(tensor_cores.nan_to_num(nan=0.0, posinf=7e4, neginf=-7e4),
                           cuda_cores.nan_to_num(nan=0.0, posinf=7e4, neginf=-7e4))


# Probabilities far below the row's largest count alike in P V and in the denominator: one key 2^-octaves above all others
# (whose value is zero), so that the result is the others' sum. Its error: the score's and the exponential's (2^-22
# together), 2 t 2^-24 of the sums, one fp16 rounding.
@pytest.mark.parametrize("octaves", [14, 20, 25, 30])
@pytest.mark.parametrize("t,d", [(130, 64), (515, 128), (4096, 64), (4096, 128)])
def test_prefill_attention_of_a_long_tail(t, d, octaves):
    q, k, v = (torch.zeros(1, 2, t, d) for _ in range(3))
    v[:] = 300.0 + torch.randn(1, 2, t, d, generator=torch.Generator().manual_seed(octaves))
    v[:, :, 0], q[..., 0], k[:, :, 0, 0] = 0.0, 1.0, octaves * 0.6931
    q, k, v = q.half().cuda(), k.half().cuda(), v.half().cuda()
    scale = 1.0
    largest = math.exp(-k[0, 0, 0, 0].double().item())  # of the others, against the first key's
    others = torch.arange(t, device="cuda").double()[None, None, :, None]
    expected = v.double().cumsum(2) * largest / (1 + others * largest)
    out = b200.b200_prefill_attention(q, k, v, None, scale=scale, causal=True).double()
    bound = (2.0 ** -20 + 2 * t * 2.0 ** -24 + 2.0 ** -11) * expected.abs() + 2.0 ** -25  # (half a subnormal's step)
    assert ((out - expected).abs() <= bound).all()


@pytest.mark.parametrize("mode", ["fast", "pytorch_compatible"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("t", [1, 8, 9, 15, 64, 65, 130])
def test_prefill_attention(t, d, mode):
    g = torch.Generator().manual_seed(t + d)
    batch, heads, kv_heads = 2, 6, 2
    q = torch.randn(batch, t, heads, d, generator=g).half().cuda().transpose(1, 2)
    k, v = (torch.randn(batch, kv_heads, t, d, generator=g).half().cuda() for _ in range(2))
    lowest = torch.zeros(batch, 1, t, t)
    lowest[:, :, :, t // 2:] = torch.finfo(torch.float32).min  # soft mask of the lowest value: some rows see only it
    lowest[1, :, t // 3] = torch.finfo(torch.float32).min
    hidden = torch.zeros(1, 1, t, t).expand(batch, 1, t, t).clone()
    hidden[:, :, t // 2] = -torch.inf  # a row that sees nothing is NaN
    options = dict(scale=d ** -0.5, numerical_mode=mode)
    for mask in (None, lowest.cuda(), hidden.cuda(), serve_ops.causal_mask(batch, t).half().cuda()):
        kept = unaligned(q.transpose(1, 2)).transpose(1, 2)
        close(b200.b200_prefill_attention(q, k, v, mask, causal=mask is None, **options),
              b200.b200_prefill_attention(kept, k, v, mask, causal=mask is None, **options))
    expected = serve_ops.prefill_attention(q.cpu(), k.cpu(), v.cpu(), serve_ops.causal_mask(batch, t),
                                           groups=heads // kv_heads, scale=d ** -0.5)
    close(b200.b200_prefill_attention(q, k, v, None, causal=True, **options), expected)


def test_prefill_attention_does_not_read_values_that_a_row_does_not_see():
    g = torch.Generator().manual_seed(4)
    q, k, v = (torch.randn(1, 2, 100, 64, generator=g).half().cuda() for _ in range(3))
    v[0, 1, 70] = float("inf")
    k[0, 0, 90] = float("nan")
    out = b200.b200_prefill_attention(q, k, v, None, scale=0.125, causal=True)
    assert out[0, 1, :70].isfinite().all() and not out[0, 1, 70:].isfinite().any()
    assert out[0, 0, :90].isfinite().all() and out[0, 0, 90:].isnan().all()


# A C caller's output may start on any element. (The warp-level kernel stores pairs, the others up to 16 bytes at once.)
@pytest.mark.parametrize("variant", [None, "mma.sync"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m,k,n", [(1, 896, 896), (8, 72, 130), (16, 72, 130), (33, 136, 64), (64, 136, 2400), (70, 72, 258),
                                   (1100, 72, 904)])
def test_linear_output_on_an_odd_element(m, k, n, dtype, variant):
    g = torch.Generator().manual_seed(m + n)
    x, w, bias = (torch.randn(*s, generator=g).to(dtype).cuda() for s in ((m, k), (n, k), (n,)))
    library, code = _lib.load(), {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}[dtype]
    for epilogue, columns in ((_lib.EPILOGUE_NONE, n), (_lib.EPILOGUE_RESIDUAL, n), (_lib.EPILOGUE_SWIGLU, n // 2)):
        residual = torch.randn(m, n, generator=g).to(dtype).cuda()
        workspace = torch.zeros(library.b200_linear_workspace_bytes(m, k, n, code, epilogue), dtype=torch.uint8, device="cuda")
        results = []
        for offset in (0, 1):
            storage = torch.full((m * columns + 2,), 77.0, dtype=dtype, device="cuda")
            output = storage[offset:offset + m * columns]
            with kernels.kernel_variants(linear=variant):
                assert library.b200_linear(x.data_ptr(), w.data_ptr(), bias.data_ptr(), residual.data_ptr(),
                                           output.data_ptr(), m, k, n, k, code, epilogue, workspace.data_ptr(),
                                           workspace.numel(), kernels.runtime().status.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream) == 0
            assert (storage[:offset] == 77.0).all() and (storage[offset + m * columns:] == 77.0).all()
            results.append(output.clone())
        assert torch.equal(*results)
    kernels.runtime().check_status()


def test_linear_on_several_streams_at_once():
    """Sizes that split K through a workspace: every stream, and every captured graph, has its own."""

    g = torch.Generator().manual_seed(5)
    x = [torch.randn(48, 4864, generator=g).half().cuda() for _ in range(3)]
    w = (0.02 * torch.randn(896, 4864, generator=g)).half().cuda()
    expected = [b200.b200_linear(rows, w) for rows in x]
    assert kernels.linear_workspace_bytes(48, 4864, 896, torch.float16) > 0
    torch.cuda.synchronize()
    streams, graphs, outputs = [torch.cuda.Stream() for _ in x], [], []
    for rows, stream in zip(x, streams):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            outputs.append([b200.b200_linear(rows, w) for _ in range(20)])
        graphs.append(graph)
    for _ in range(5):
        for graph, stream in zip(graphs, streams):
            with torch.cuda.stream(stream):
                graph.replay()
        eager = []
        for rows, stream in zip(x, streams):
            with torch.cuda.stream(stream):
                eager.append([b200.b200_linear(rows, w) for _ in range(20)])
        torch.cuda.synchronize()
        for results in (*zip(outputs, expected), *zip(eager, expected)):
            assert all(torch.equal(result, results[1]) for result in results[0])
    rt = kernels.runtime()
    addresses = []
    for stream in streams:
        with torch.cuda.stream(stream):
            addresses.append(rt.own_workspace("linear", 64).data_ptr())
            assert rt.own_workspace("linear", 64).data_ptr() == addresses[-1]
    assert len(set(addresses)) == len(streams)
    torch.cuda.synchronize()
