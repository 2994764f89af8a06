"""The exact blocks of the FP64 digit products: over one block the FP32 sums of the levels that matter hold every
integer, for the largest digits in every place, whatever the order of the additions."""

import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "sphericalfourierbesseldecompositions.jl_gb300", "csrc")


def _constant(path, name):
    return int(re.search(rf"constexpr int {name} = (\d+);", open(os.path.join(CSRC, path)).read()).group(1))


# the leading digit of a 55-bit integer, and of a folded ring sum of 56 bits
@pytest.mark.parametrize("path,block,lead", [("digit64.cuh", "SBK", 128), ("ring64_tc.cu", "SBR", 256)])
def test_levels_of_a_block_are_exact(path, block, lead):
    K = _constant(path, block) * _constant("digit64.cuh", "KC")
    assert _constant("digit64.cuh", "ND") == 7
    for v in range(7):
        largest = K * (lead * 128 + v * 128 * 128)           # v + 1 products, one with the leading data digit
        unit = 2.0 ** (-14 - 8 * v)                            # of the scales
        steps = K // 16 * (v + 1)                              # accumulations into the level
        lost = 0.0 if largest <= 1 << 24 else steps * float(np.spacing(np.float32(largest))) * unit
        assert v >= 6 or lost == 0.0, (v, largest)
        assert lost < 2.0 ** -54
