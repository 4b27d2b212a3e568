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
    v[:, ::3] *= 2.0 ** 40               # factors far from 1,
    v[:, 5] = 1.75 * 2.0 ** -118         # a token whose factor is the smallest there is
    k[:, 7] = 0.0                        # and one without any (its factor is 1)
    ops = [K.quantize_fp8_blocks(t, token_local_exponents=True) for t in (q, k, v)]
    assert float(ops[2]["token_factors"].min()) == 2.0 ** -126 and float(ops[1]["token_factors"][:, :, 7].min()) == 1.0
    want, want_lse, st = K.attn_fwd(*ops, causal=causal, softmax_scale=1.0 / math.sqrt(d), token_local=True)
    opts = F.FP8AttnOptions(operand_scaling="token_local", ds_dq_rowlocal="all")
    with torch.no_grad():
        got, lse = F.flash_attn_fp8(q, k, v, causal=causal, options=opts, return_lse=True)
    assert K.read_status(st) == 0
    assert torch.isfinite(got).all() and torch.equal(got, want) and torch.equal(lse, want_lse)


def test_narrow_tables_hold_what_the_float_ones_do():
    """Every exponent that a token factor can take, in f_K and f_V, against fl_token_aux."""
    from flamia_blackwell_attention_b200 import _lib as L, kernels as K
    e = torch.arange(-126, 127, dtype=torch.float32)
    fk, fv = torch.exp2(e).cuda(), torch.exp2(e.roll(100)).cuda()
    n = e.numel()
    kv, rcp = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int16, device="cuda")
    L.check(L.load().fl_token_tables(L.ptr(fk), L.ptr(fv), n, L.ptr(kv), L.ptr(rcp), K._stream()), "fl_token_tables")
    lg, inv = K.token_aux(fv)
    halves = kv.view(torch.bfloat16).float().view(n, 2)          # lower half first
    assert torch.equal(halves[:, 1], fk) and torch.equal(halves[:, 0], lg) and torch.equal(rcp.view(torch.bfloat16).float(), inv)
