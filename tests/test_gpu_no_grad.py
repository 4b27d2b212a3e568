"""Calls without gradients return the bytes of the same call with them (O and LSE), through the public entry points."""
import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,sq,sk,h,hk,d,kw", [
    (1, 128, 128, 1, 1, 128, dict(causal=True)),
    (2, 640, 640, 2, 1, 128, dict(causal=True)),                 # the last block without a second stage
    (1, 384, 1152, 3, 1, 128, dict()),
    (1, 128, 8192, 1, 1, 128, dict(causal=True)),                # few items of many key tiles
    (1, 2049, 2049, 2, 1, 96, dict(causal=True)),
    (1, 896, 896, 2, 2, 64, dict(causal=True)),
    (2, 512, 512, 2, 1, 64, dict()),
    (2, 1000, 1000, 2, 1, 64, dict()),                           # rows that are no whole tiles
    (1, 385, 385, 2, 2, 80, dict(causal=True)),
    (1, 640, 640, 2, 2, 128, dict(causal=True, softcap=20.0)),
    (1, 896, 896, 2, 1, 128, dict(causal=True, window_size=(300, 0))),
    (1, 896, 896, 2, 1, 128, dict(causal=True, fp4=True)),
    (2, 640, 640, 2, 2, 128, dict(fp4=True)),
])
def test_the_bytes_of_the_call_with_gradients(b, sq, sk, h, hk, d, kw):
    import flamia_blackwell_attention_b200 as F
    kw = dict(kw)
    fn = F.flash_attn_fp4 if kw.pop("fp4", False) else F.flash_attn_fp8
    q, k, v, _ = attention_inputs(b, max(sq, sk), h, hk, d, seed=21)
    q, k, v = q[:, :sq].contiguous().cuda(), k[:, :sk].contiguous().cuda(), v[:, :sk].contiguous().cuda()
    with torch.no_grad():
        o, lse = fn(q, k, v, return_lse=True, **kw)
        alone = fn(q, k, v, **kw)
    og, lseg = fn(*(t.detach().clone().requires_grad_(True) for t in (q, k, v)), return_lse=True, **kw)
    assert F.check_status() == 0
    assert torch.equal(o, og) and torch.equal(lse, lseg) and torch.equal(alone, o)
