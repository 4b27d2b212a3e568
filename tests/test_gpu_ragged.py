"""Batch rows that are no whole tiles, as batch rows: against the same rows as packed documents, bit for bit."""
import warnings

import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,h,hk,d,dtype,kw", [
    (1, 1, 1, 1, 128, "bfloat16", dict(causal=True)),
    (3, 127, 2, 1, 64, "float16", dict(causal=False)),
    (2, 129, 4, 2, 128, "bfloat16", dict(causal=True)),             # one row in the last tile
    (2, 257, 2, 2, 96, "bfloat16", dict(causal=True)),              # and in the last block of 256
    (2, 383, 2, 1, 80, "float16", dict(causal=False)),
    (2, 640 + 31, 3, 1, 64, "bfloat16", dict(causal=True, window_size=(200, 0))),
    (2, 500, 2, 2, 128, "bfloat16", dict(causal=False, window_size=(60, 130))),
    (2, 300, 2, 1, 128, "bfloat16", dict(causal=True, softcap=20.0)),
    (2, 300, 2, 1, 128, "float16", dict(causal=True, deterministic=True)),
])
def test_batch_rows_equal_documents(b, s, h, hk, d, dtype, kw):
    """dQ to the rounding of its f16 sums, which come in arrival order with a pre-scale per batch row instead of one (the bound of
    test_gpu_full_size.py for the same)."""
    import flamia_blackwell_attention_b200 as F
    x = [t.to(getattr(torch, dtype)).cuda() for t in attention_inputs(b, s, h, hk, d, seed=21)]

    def step(q, k, v, g, **more):
        q, k, v = (t.detach().clone().requires_grad_(True) for t in (q, k, v))
        out, lse = F.flash_attn_fp8(q, k, v, return_lse=True, **kw, **more)
        return (out.detach(), lse, *torch.autograd.grad(out, (q, k, v), g))
    o, lse, dq, dk, dv = step(*x)
    cu = torch.arange(0, b * s + 1, s, dtype=torch.int32, device="cuda")
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        po, plse, pdq, pdk, pdv = step(*(t.flatten(0, 1) for t in x), cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=s, max_seqlen_k=s)
    assert torch.equal(lse, plse.view(h, b, s).transpose(0, 1))
    for got, want in ((o, po), (dk, pdk), (dv, pdv)):
        assert torch.equal(got, want.view(got.shape))
    assert float((dq.float() - pdq.view(dq.shape).float()).norm()) <= 8e-3 * float(pdq.float().norm())
    assert F.check_status() == 0


@pytest.mark.parametrize("b,h,s", [(1, 1, 200), (1, 1, 1), (1, 2, 200), (2, 1, 130)])
def test_returned_lse_is_the_callers_own(b, h, s):
    """What a caller writes into the returned LSE reaches no gradient, and the tensor holds no more memory than its rows."""
    import flamia_blackwell_attention_b200 as F
    q, k, v, g = (t.cuda() for t in attention_inputs(b, s, h, h, 64, seed=22))
    for t in (q, k, v):
        t.requires_grad_(True)
    out, lse = F.flash_attn_fp8(q, k, v, causal=True, return_lse=True)
    assert lse.shape == (b, h, s) and lse.untyped_storage().nbytes() == 4 * b * h * s
    want = torch.autograd.grad(out, (q, k, v), g, retain_graph=True)
    lse.fill_(7.0)
    got = torch.autograd.grad(out, (q, k, v), g)
    assert all(torch.equal(x, y) for x, y in zip(got[1:], want[1:]))
    assert float((got[0].float() - want[0].float()).norm()) <= 8e-3 * float(want[0].float().norm())     # (the order of dQ's f16 sums)


@pytest.mark.parametrize("s,d", [(8, 64), (3, 128)])
def test_more_batch_rows_than_a_grid_has_in_y_and_z(s, d):
    """65540 batch rows of two kinds: every row has the bytes of its kind in a call of two rows (dQ to the order of its f16 sums, of which a
    row of up to 128 keys has one)."""
    import flamia_blackwell_attention_b200 as F
    b = 65540
    two = [t.cuda() for t in attention_inputs(2, s, 1, 1, d, seed=23)]

    def step(x):
        q, k, v = (t.requires_grad_(True) for t in x[:3])
        out = F.flash_attn_fp8(q, k, v, causal=True)
        return out.detach(), *torch.autograd.grad(out, (q, k, v), x[3])
    many = step([t.repeat(b // 2, 1, 1, 1) for t in two])
    assert F.check_status() == 0
    for got, want in zip(many, step(two)):
        assert torch.equal(got.view(b // 2, 2, s, 1, d), want.view(1, 2, s, 1, d).expand(b // 2, -1, -1, -1, -1))


@pytest.mark.parametrize("rows", [3, 250, 1 << 20, -7])
@pytest.mark.parametrize("d", [64, 128])
def test_rows_of_the_c_entries_are_read_with_their_flag(rows, d, monkeypatch):
    """src_rows and out_rows hold anything where neither slot tables nor FL_Q_ROWS / FL_A_ROWS ask for them."""
    from flamia_blackwell_attention_b200 import _lib as L
    from test_gpu_bwd import run_step
    x = attention_inputs(1, 256, 2, 1, d, seed=24)
    want = run_step(*x, True)

    class Quant(L.QuantArgs):
        def __init__(self):
            super().__init__(src_rows=rows)

    class Attn(L.AttnArgs):
        def __init__(self):
            super().__init__(out_rows=rows)
    monkeypatch.setattr(L, "QuantArgs", Quant)
    monkeypatch.setattr(L, "AttnArgs", Attn)
    for got, w in zip(run_step(*x, True), want):
        assert torch.equal(got, w)
