"""Forwards of few items run on blocks of 128 query rows: the bytes of the same rows in a call of many items (blocks of 256)."""
import pytest
import torch

from inputs import attention_inputs
from launches import launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,sk,h,hk,d,dtype,kw", [
    (128, 128, 1, 1, 128, "bfloat16", dict(causal=True)),                          # (one block of either size)
    (129, 129, 2, 1, 64, "float16", dict(causal=True)),                            # one row in the second block
    (256, 1152, 4, 2, 128, "bfloat16", dict(causal=True)),                         # bottom-right aligned
    (640, 256, 2, 2, 128, "bfloat16", dict(causal=True)),                          # leading rows without a key
    (300, 300, 2, 2, 80, "bfloat16", dict()),
    (2049, 2049, 2, 1, 128, "bfloat16", dict(causal=True)),
    (1024, 1024, 3, 1, 128, "bfloat16", dict(causal=True, window_size=(200, 0))),  # the stages of a block of 256 start at one key tile
    (900, 900, 2, 2, 64, "bfloat16", dict(window_size=(130, 70))),
    (640, 640, 2, 1, 128, "bfloat16", dict(causal=True, softcap=20.0)),
    (640, 640, 2, 1, 128, "bfloat16", dict(causal=True, used=500)),
    (896, 896, 2, 1, 128, "bfloat16", dict(causal=True, fp4=True)),
    (384, 1280, 2, 2, 128, "float16", dict(fp4=True)),
    (768, 768, 4, 2, 128, "bfloat16", dict(causal=True, token=True)),
])
@pytest.mark.parametrize("grad", [False, True])
def test_bytes_of_a_call_of_many_items(s, sk, h, hk, d, dtype, kw, grad):
    import flamia_blackwell_attention_b200 as F
    kw = dict(kw)
    fn, used = F.flash_attn_fp4 if kw.pop("fp4", False) else F.flash_attn_fp8, kw.pop("used", None)
    if kw.pop("token", False):
        kw["options"] = F.FP8AttnOptions(operand_scaling="token_local", ds_dq_rowlocal="all")
    q, k, v, _ = (t.to(getattr(torch, dtype)) for t in attention_inputs(1, max(s, sk), h, hk, d, seed=31))
    x = [t.contiguous().cuda() for t in (q[:, :s], k[:, :sk], v[:, :sk])]

    def call(b):
        more = dict(kw, seqused_k=torch.full((b,), used, dtype=torch.int32, device="cuda")) if used else kw
        q, k, v = (t.repeat(b, 1, 1, 1).requires_grad_(grad) for t in x)
        with torch.set_grad_enabled(grad):
            return fn(q, k, v, return_lse=True, **more)
    many = torch.cuda.get_device_properties(0).multi_processor_count // (2 * ((s + 255) // 256 * h)) + 1
    (o, lse), (om, lsem) = call(1), call(many)
    assert F.check_status() == 0
    for i in (0, many - 1):
        assert torch.equal(om[i], o[0]) and torch.equal(lsem[i], lse[0])


def test_which_calls_run_on_blocks_of_128(tmp_path):
    import flamia_blackwell_attention_b200 as F
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for s, h in ((640, 1), (256, sms // 2), (256, sms // 2 + 1)):
        q, k, v = (torch.zeros(1, s, n, 64, dtype=torch.bfloat16, device="cuda") for n in (h, 1, 1))
        with torch.no_grad():
            grids = [g[0] for n, g, _ in launches(lambda: F.flash_attn_fp8(q, k, v, causal=True), tmp_path) if "fwd_kernel" in n]
        assert grids == [(s + 127) // 128 * h if 2 * ((s + 255) // 256) * h <= sms else h]
