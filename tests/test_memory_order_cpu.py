"""Orderings between threads, grids and the tensor core that no run can be relied on to show: read off the kernels' source."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "llm-compiler_b200" / "csrc"


def test_probabilities_in_tensor_memory_are_stored_behind_the_product_before():
    """Prompt attention keeps one buffer of P a group. The product that read it is behind the wait on o_done, but only a
    fence orders a thread's next access to tensor memory behind a wait: it belongs between the wait and the stores on every
    path, not only where O is moved as well."""

    source = (CSRC / "prefill_attention_tcgen05.cu").read_text()
    wait = re.search(r"mbarrier_wait_ready_first\(smem_u32\(&o_done\[g\]\), \(j - 1\) & 1", source)
    move = source.index("if (ok && raise)", wait.end())
    store = source.index("tmem_store_32x16(p_taddr", move)
    assert wait.end() < move < store
    assert re.search(r'if \(ok\) asm volatile\("tcgen05\.fence::after_thread_sync;"', source[wait.end():move])


def test_kernels_that_wait_on_the_device_promise_nothing_about_their_operands():
    """A kernel of a programmatic launch is resident while the kernel before it still writes. __restrict__ on a read-only
    operand would promise that it does not change for as long as the kernel runs, and let loads move ahead of the wait."""

    for path in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]:
        for kernel in re.split(r"__global__", path.read_text())[1:]:
            parameters, _, body = kernel.partition("{")
            if "grid_dependency_wait" in body:
                assert "__restrict__" not in parameters, f"{path.name}: {parameters.strip()}"


def test_operands_that_a_kernel_in_flight_may_write_are_read_as_such():
    """__ldg reads through a path that takes its data as constant while the kernel runs. In the projections that wait on the
    device that holds for no operand (the tiled fp32 product, which does not, keeps it)."""

    for name, kernel in (("linear_tcgen05.cu", "add_bias"), ("linear.cu", "linear_rows_kernel("), ("linear_rows.cu", "")):
        source = (CSRC / name).read_text()
        body = source[source.index(kernel):]
        end = re.search(r"\n}\n", body).end() if kernel else len(body)
        assert "__ldg" not in body[:end], name
