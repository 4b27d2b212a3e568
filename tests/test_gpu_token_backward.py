"""Token-local backward on D that comes divided by the token's factor, against the one on D as it is: the factors are powers of two, so
the two give the same bits (but for products below 2^-126, which these inputs do not have)."""
import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,sq,sk,h,hk,kw", [
    (1, 128, 128, 1, 1, dict(causal=True)),
    (2, 384, 384, 2, 1, dict(causal=True)),
    (1, 256, 640, 4, 2, dict(causal=False)),
    (1, 640, 256, 1, 1, dict(causal=True)),                  # leading rows without a key
    (1, 512, 512, 2, 2, dict(causal=True, window=(130, 0))),
])
def test_divided_d(b, sq, sk, h, hk, kw):
    from flamia_blackwell_attention_b200 import kernels as K
    q, k, v, g = attention_inputs(b, max(sq, sk), h, hk, 128, seed=31)
    g = g * torch.exp2(torch.arange(max(sq, sk)) % 23 - 11.0)[None, :, None, None].to(g.dtype)       # factors far apart
    g[:, 5] = 0                                                                          # a token without one
    q, g, k, v = (t.cuda() for t in (q[:, :sq], g[:, :sq], k[:, :sk], v[:, :sk]))
    qq, kq, vq = (K.quantize_fp8_blocks(t, token_local_exponents=True, output_tile_stats=True) for t in (q, k, v))
    kw = dict(kw, softmax_scale=128 ** -0.5, token_local=True)
    out, lse, st = K.attn_fwd(qq, kq, vq, **kw)
    assert K.read_status(st) == 0
    pre = torch.exp2(torch.arange(b * sq, device="cuda") % 5 - 14.0)     # a pre-scale per row of dQ (the other variant), far from overflow
    for rows in (None, pre):
        got = []
        for fold in (False, True):
            acc = torch.empty(b, h, 128, sq, dtype=torch.float16, device="cuda")
            gq = K.quantize_fp8_blocks(g, compute_d_with_output=out, shifted_log2_lse_from=lse, log2_lse_shift=8.0, d_multiplier=-2.0 ** -8,
                                       zero_accumulator=acc, output_tile_stats=True, token_local_exponents=True, d_per_factor=fold)
            ks, _ = K.dq_prescale(gq["tile_stats"], vq["tile_stats"], kq["tile_stats"])
            dk, dv, st = K.attn_bwd(qq, kq, vq, gq, lse_log2=gq["lse_log2"], d_rows=gq["D"], dq_acc=acc, dq_scale=ks, dq_rowlocal=True,
                                    dq_scale_rows=rows, d_per_factor=fold, **kw)
            assert K.read_status(st) == 0 and torch.isfinite(dk.float()).all() and torch.isfinite(dv.float()).all()
            got.append((dk, dv, acc.double(), gq))
        (dk0, dv0, x, g0), (dk1, dv1, y, g1) = got
        assert torch.equal(g0["D"], g1["D"] * g1["token_factors"])
        assert torch.equal(dk0, dk1) and torch.equal(dv0, dv1)
        # (up to five partial sums in any order: each rounds the f16 accumulator once, by 2^-11 of what it holds)
        assert float((x - y).norm()) <= 5 * 2.0 ** -11 * float(x.norm()) + 1e-6


def test_refused():
    """The flag goes with token factors."""
    from flamia_blackwell_attention_b200 import kernels as K
    x = torch.randn(1, 128, 1, 128, device="cuda").bfloat16()
    with pytest.raises(RuntimeError):
        K.quantize_fp8_blocks(x, d_per_factor=True)
