"""The per-head products of latent attention on the tensor cores: rows and columns around a tile, K in fewer 64-wide blocks
than a ring has stages, as many and more, CTAs that have an SM each and CTAs that do not, W ahead of the dependency wait."""

import pytest
import torch

from llm_compiler_b200 import hybrid_kernels as hk
from llm_compiler_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("m,heads,k,n", [(1, 16, 512, 128), (16, 16, 128, 512), (17, 14, 64, 256), (32, 16, 512, 128),
                                         (64, 3, 520, 72), (65, 2, 1096, 136), (5, 40, 200, 328), (70, 20, 584, 256)])
def test_head_linear(m, heads, k, n, early):
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    x = torch.randn(m, heads, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(heads, n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    exact = torch.einsum("mhk,hnk->mhn", x.double(), w.double())
    # one rounding of the result, and fp32 sums in one chain of K / 16 products
    bound = 2.0 ** -8 * exact.abs() + (k / 16 + 8) * 2.0 ** -23 * torch.einsum("mhk,hnk->mhn", x.double().abs(), w.double().abs())
    torch.cuda.synchronize()
    with kernels.launch_mode(programmatic=early, constant_weights=early):
        y = hk.head_linear(x, w)
    assert ((y.double() - exact).abs() <= bound + 1e-6).all()
