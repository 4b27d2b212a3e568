"""Per-key tables of the token-local forward: the narrow ones against float ones, bit for bit."""
import math

import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sq,sk,h,hk,d,causal", [
    (128, 128, 1, 1, 128, True),         # one tile
    (384, 384, 4, 2, 128, True),         # an odd number of tiles, a half block of rows at the end
    (256, 640, 3, 1, 128, False),
    (256, 384, 2, 2, 64, True),
])
def test_narrow_tables_change_nothing(sq, sk, h, hk, d, causal):
    import flamia_blackwell_attention_b200 as F
    from flamia_blackwell_attention_b200 import kernels as K
    s = max(sq, sk)
    q, k, v, _ = (t.cuda() for t in attention_inputs(2, s, h, hk, d, seed=41))
    q, k, v = q[:, :sq].contiguous(), k[:, :sk].contiguous(), v[:, :sk].contiguous()
    v[:, ::3] *= 2.0 ** 40               # factors far from 1, and a token whose factor is the smallest there is
    v[:, 5] *= 2.0 ** -100
    k[:, 7] = 0.0
    ops = [K.quantize_fp8_blocks(t, token_local_exponents=True) for t in (q, k, v)]
    want, _, st = K.attn_fwd(*ops, causal=causal, softmax_scale=1.0 / math.sqrt(d), token_local=True)
    opts = F.FP8AttnOptions(operand_scaling="token_local", ds_dq_rowlocal="all")
    with torch.no_grad():
        got = F.flash_attn_fp8(q, k, v, causal=causal, options=opts)
    assert K.read_status(st) == 0
    assert torch.equal(got, want)
