"""The call path's host side, without a GPU."""
import pytest
import torch

import flamia_blackwell_attention_b200 as F
from flamia_blackwell_attention_b200 import _op


@pytest.mark.parametrize("side", [0, 511, 2 ** 30, 2 ** 31 - 2, 2 ** 31 - 1, 2 ** 33 + 5])
def test_window_sides_reach_the_kernels_whole(side):
    """A side of any size means at least as many keys there: the numbers handed to the launches never wrap, and leave room for the
    positions (below 2^30) that the kernels add to them."""
    q = torch.empty(1, 256, 2, 64, dtype=torch.bfloat16, device="meta")
    facts = _op._plan_facts(F.resolve_fp8(q, q, q, window_size=(side, side)))
    for name in ("window_left_p1", "window_right_p1"):
        assert min(side, 256) < facts[name] <= 2 ** 30 + 1
