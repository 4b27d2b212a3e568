"""The call path's host side, without a GPU."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

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


def test_torch_function_modes_see_the_op():
    calls = []

    class Mode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            calls.append(str(func))
            return func(*args, **(kwargs or {}))
    with FakeTensorMode():
        q = torch.empty(1, 256, 2, 128, dtype=torch.bfloat16, device="cuda")
        with Mode():
            F.flash_attn_fp8(q, q, q)
            F.flash_attn_fp4(q, q, q)
    assert "lowbit_attn.fp8" in calls and "lowbit_attn.fp4" in calls
