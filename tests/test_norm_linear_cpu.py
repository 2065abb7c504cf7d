"""Where the RMS norm goes inside the fp32 projection behind it: a host-side rule on sizes, asked without a device."""

import pytest

from llm_compiler_b200 import kernels


# The norm costs registers and arithmetic in every CTA and saves a launch: it goes inside where both forms take one wave of
# CTAs, or two (not of 4 rows with full rings), on both sides of each line.
@pytest.mark.parametrize("m,k,n,pays", [
    (4, 896, 1152, True), (4, 896, 9728, True),    # a decode step of Qwen2-0.5B: one wave, two waves with and without
    (1, 2048, 3552, True), (1, 2048, 3560, False),  # 4 rows, full rings: 444 and 445 CTAs, three an SM
    (4, 896, 11840, True), (4, 896, 11848, False),  # 4 rows, half rings: 1480 and 1481 CTAs, five an SM
    (8, 256, 3552, True), (8, 256, 3560, False),   # 8 rows: 445 CTAs are a second wave with the norm only
    (8, 256, 4744, True),                          # ... and 593 in either form
    (32, 2560, 440, True), (32, 2560, 454, False),  # clusters of two
    (41, 896, 64, False), (0, 896, 64, False),     # rows that are not streamed, no rows
    (40, 2560, 23436, False), (9, 512, 23918, False), (1, 4096, 14648, False)])
def test_where_the_norm_pays_inside(m, k, n, pays):
    assert kernels.rms_norm_linear_pays(m, k, n) is pays
