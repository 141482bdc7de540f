"""GPU test that ff_error_sums and ff_error_sums_noalloc return the same sums bit
for bit (include/fishfry.h: the same fixed order), from one block's partials to
all of them, and that the arrays the library keeps for them are what the header
says."""
import os
import re

import numpy as np
import pytest

from test_zz_no_alloc import noalloc_sums


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(1, 1, 1), (5, 13, 63), (64, 48, 40), (160, 160, 150), (1, 1, 75841)])
def test_both_entry_points_return_the_same_sums(torch_cuda, ff, n, precision):
    torch = torch_cuda
    dt = torch.float64 if precision == 0 else torch.float32
    phi = torch.from_numpy(np.random.default_rng(3).standard_normal(n)).to(dt).cuda().reshape(-1)
    modes = [(1, 2, 3, 0.25, 0.5)]
    for m in ([], modes):
        for p in (None, phi):
            assert noalloc_sums(ff, n, p, m, precision) == list(ff.error_sums(n, p, m, precision))


def test_sizes_in_the_header(ff):
    """The sizes of the library's device arrays, from the source's constants."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = open(os.path.join(root, "fishfry_b200", "csrc", "ff_field.cu")).read()
    blocks = int(re.search(r"kSumBlocks = (\d+)", src).group(1))
    slots = int(re.search(r"kSumSlots = (\d+)", src).group(1))
    assert re.search(r"kSumSlotDoubles = 3 \* kSumBlocks \+ 3;", src)
    assert re.search(r"g_sum_slots\[kSumSlots\]\[kSumSlotDoubles\];", src)
    assert re.search(r"g_noalloc_partials\[kSumSlotDoubles\];", src)
    slot = 8 * (3 * blocks + 3)
    text = open(os.path.join(root, "include", "fishfry.h")).read()
    assert "(%d KB per GPU" % round(slots * slot / 1000) in text
    assert "(%d KB per GPU" % round(slot / 1000) in text
