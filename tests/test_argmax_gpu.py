"""Greedy tokens: rows shared by a cluster and rows of one CTA, against the first of a row's largest logits."""

import pytest
import torch

from llm_compiler_b200 import kernels

pytestmark = pytest.mark.gpu


# rows of one cluster and of one CTA each; fewer elements than threads, ragged ends, rows off a 16-byte boundary
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,vocab", [(1, 1), (1, 7), (3, 1000), (2, 8192), (1, 32767), (64, 32768), (5, 151936), (96, 1025), (97, 1025)])
def test_argmax(rows, vocab, dtype):
    g = torch.Generator(device="cuda").manual_seed(vocab)
    wide = torch.randint(-3, 3, (rows, vocab + 9), generator=g, device="cuda").to(dtype)  # (many ties)
    wide[:, vocab:] = 9.0
    wide[0, vocab - 1] = 5.0
    for logits in (wide[:, :vocab], wide[:, :vocab].contiguous()):
        first = (logits == logits.max(-1, keepdim=True).values).to(torch.int8).argmax(-1)  # (the first of equals)
        assert torch.equal(kernels.b200_argmax(logits), first)
    wide[rows - 1, :vocab] = float("-inf")
    assert int(kernels.b200_argmax(wide[:, :vocab])[rows - 1]) == 0


# both sides of the lines between rows shared by a cluster and rows of one CTA: 80 rows (32-bit elements 96), 16 KB a row
@pytest.mark.parametrize("dtype,rows,vocab", [(torch.bfloat16, 80, 8192), (torch.bfloat16, 81, 8192), (torch.bfloat16, 80, 8191),
                                              (torch.float16, 80, 8193), (torch.float32, 96, 4096), (torch.float32, 97, 4096),
                                              (torch.float32, 96, 4095)])
@pytest.mark.parametrize("programmatic", [False, True])
def test_argmax_on_both_sides_of_its_lines(dtype, rows, vocab, programmatic):
    g = torch.Generator(device="cuda").manual_seed(vocab)
    logits = torch.randint(-3, 3, (rows, vocab), generator=g, device="cuda").to(dtype)  # (many ties)
    logits[0, vocab - 1] = 5.0
    logits[rows - 1] = float("-inf")
    first = (logits == logits.max(-1, keepdim=True).values).to(torch.int8).argmax(-1)  # (the first of equals)
    torch.cuda.synchronize()
    with kernels.launch_mode(programmatic=programmatic):
        assert torch.equal(kernels.b200_argmax(logits), first)
