"""GPU: forms of a call (masks, layouts, document tables, transforms around it) against the same call in its plain form."""
import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu


def _step(fn, q, k, v, do, **kw):
    """(out, dq, dk, dv) of one call; deterministic, so that two calls on the same values compare bit for bit."""
    q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
    out = fn(q, k, v, deterministic=True, **kw)
    return (out.detach(), *torch.autograd.grad(out, (q, k, v), do))


@pytest.mark.parametrize("s", [256, 1000])             # whole tiles; batch rows run as documents
@pytest.mark.parametrize("window,same", [((2 ** 31 - 2, 2 ** 31 - 2), (None, None)), ((2 ** 31 - 2, 100), (None, 100)),
                                         ((100, 2 ** 31 - 2), (100, None)), ((2 ** 33 + 5, 2 ** 31 - 1), (None, None))])
def test_window_longer_than_any_sequence(s, window, same):
    import flamia_blackwell_attention_b200 as F
    x = [t.cuda() for t in attention_inputs(2, s, 2, 1, 64, seed=11)]
    for a, b in zip(_step(F.flash_attn_fp8, *x, window_size=window), _step(F.flash_attn_fp8, *x, window_size=same)):
        assert torch.equal(a, b)
