"""Split schedules: the forward whose items are cut into pieces, against the CPU oracle and against whole items."""
import pytest
import torch

from inputs import attention_inputs
from oracle import attention_oracle as A

pytestmark = pytest.mark.gpu


def schedule(tiles, share):
    """A schedule that hands `share` positions (key tiles; an item has at least one) to each CTA, wherever that cuts."""
    from flamia_blackwell_attention_b200 import _lib as L
    at, left = [0], share
    for item, n in enumerate(tiles):
        t = 0
        while n - t > left:
            t += left
            at.append(item << L.SPLIT_TILE_BITS | t)
            left = share
        left -= max(n - t, 1)
        if left <= 0 and item + 1 < len(tiles):
            at.append((item + 1) << L.SPLIT_TILE_BITS)
            left = share
    s = L.Split(parts=len(at))
    for i, v in enumerate(at + [len(tiles) << L.SPLIT_TILE_BITS]):
        s.at[i] = v
    assert 2 <= s.parts <= L.SPLIT_MAX
    return s


def fwd_tiles(b, sq, sk, h, causal):
    """Key tiles of the forward's items, in the kernel's order of items."""
    def n(blk):
        return max(0, (min(sk, min(sq, blk * 256 + 256) + sk - sq) if causal else sk) + 127) // 128
    blocks = range((sq + 255) // 256)
    return [n(x) for x in reversed(blocks) for _ in range(b * h)] if causal else [n(x) for _ in range(b * h) for x in blocks]


def operands(q, k, v, fp4=False):
    from flamia_blackwell_attention_b200 import kernels as K
    kw = dict(also_make_nvfp4_copy=True, hadamard_rotation_scope="nvfp4_copy") if fp4 else {}
    return [K.quantize_fp8_blocks(t.cuda(), **(kw if i < 2 else {})) for i, t in enumerate((q, k, v))]


# b, s_q, s_k, h, h_kv, d, causal, form
FWD = [
    (1, 256, 1024, 1, 1, 128, False, {}),
    (1, 1024, 1024, 2, 1, 128, True, {}),
    (2, 384, 384, 4, 2, 128, True, {}),                       # the last block without a second stage
    (1, 256, 640, 2, 1, 128, True, {}),                       # bottom-right aligned
    (1, 640, 256, 2, 2, 128, True, {}),                       # leading rows, and whole items, without a key
    (1, 1152, 1152, 2, 2, 64, True, {}),
    (2, 512, 512, 2, 2, 64, False, {}),
    (2, 640, 640, 2, 1, 128, False, dict(window=(None, 200))),
    (3, 256, 768, 2, 1, 128, False, dict(used=[768, 130, 1])),    # pieces past a row's last valid key
    (1, 768, 768, 2, 2, 128, True, dict(softcap=20.0)),
    (1, 896, 896, 2, 1, 128, True, dict(fp4=True)),
    (2, 512, 640, 2, 2, 128, False, dict(fp4=True, group=True)),
    (1, 896, 896, 2, 1, 128, True, dict(group=True)),
]


@pytest.mark.parametrize("share", [1, 3, 7])
@pytest.mark.parametrize("b,sq,sk,h,hk,d,causal,form", FWD)
def test_forward_in_pieces(b, sq, sk, h, hk, d, causal, form, share):
    """Every piece frames a row's P-hat as the whole item does (N(0, 1) operands: the first tile's maximum is refreshed by no later one), so
    the rounded terms are the same but for one exponential in four, by polynomials up to 7.5e-5 apart (codes of P-hat are about a
    twelfth apart: of 1e5 codes some fifteen fall on another value, 1e-3 of O's norm). O differs by that, f32 sums in another order and the last bit
    of bfloat16 (2^-9): below 2^-8; the LSE by a few units of 2^-20 of logarithms up to about 10."""
    from flamia_blackwell_attention_b200 import _lib as L, kernels as K
    q, k, v, _ = attention_inputs(b, max(sq, sk), h, hk, d, seed=11)
    q, k, v = q[:, :sq], k[:, :sk], v[:, :sk]
    form = dict(form)
    fp4, group, used = (form.get(n) for n in ("fp4", "group", "used"))
    kw = dict(causal=causal, softmax_scale=d ** -0.5, mode=L.FL_MODE_FP4 if fp4 else L.FL_MODE_FP8, window=form.get("window"),
              p_group=bool(group), seqused_k=torch.tensor(used, dtype=torch.int32).cuda() if used else None, softcap=form.get("softcap", 0.0))
    ops = operands(q, k, v, fp4)
    tiles = fwd_tiles(b, sq, sk, h, causal)
    if "window" in form:          # only a right side: an item ends where its last row does
        tiles = [min(n, (min(640, 256 * (i % 3) + 256) + 200 + 127) // 128) for i, n in enumerate(tiles)]
    if sum(max(t, 1) for t in tiles) / share > 150:
        pytest.skip("more shares than CTAs")
    o1, l1, s1 = K.attn_fwd(*ops, **kw)
    o2, l2, s2 = K.attn_fwd(*ops, split=schedule(tiles, share), **kw)
    o3, l3, _ = K.attn_fwd(*ops, split=schedule(tiles, share), **kw)
    assert K.read_status(s1) == 0 and K.read_status(s2) == 0
    assert torch.equal(o2, o3) and torch.equal(l2, l3)
    vis = torch.isfinite(l1)
    assert torch.equal(vis, torch.isfinite(l2))
    assert float((l1[vis] - l2[vis]).abs().max()) < 1e-4
    assert A.accuracy(o2.float().cpu(), o1.float().cpu())["rel_l2"] < 2.0 ** -8
    assert float(o2[~vis.permute(0, 2, 1)].abs().max() if (~vis).any() else 0.0) == 0.0


@pytest.mark.parametrize("sq,sk,h,hk,d,causal", [(256, 2048, 2, 1, 128, False), (1024, 1024, 2, 2, 128, True), (512, 1024, 2, 1, 64, True)])
def test_forward_in_pieces_vs_oracle(sq, sk, h, hk, d, causal):
    from flamia_blackwell_attention_b200 import kernels as K
    q, k, v, _ = attention_inputs(1, max(sq, sk), h, hk, d, seed=12)
    q, k, v = q[:, :sq], k[:, :sk], v[:, :sk]
    out, lse, st = K.attn_fwd(*operands(q, k, v), causal=causal, softmax_scale=d ** -0.5, split=schedule(fwd_tiles(1, sq, sk, h, causal), 2))
    ro, rl, *_ = A.qdq_attention(q, k, v, causal=causal)
    assert K.read_status(st) == 0
    assert A.accuracy(out.float().cpu(), ro)["rel_l2"] < 3.2e-2
    assert float((lse.cpu() - rl).abs().max()) < 2e-3


@pytest.mark.parametrize("entry,sq,sk,h,hk,d,dtype,kw", [
    ("fp8", 128, 8192, 1, 1, 128, "bfloat16", {}),
    ("fp8", 2048, 2048, 2, 1, 96, "float16", {}),
    ("fp8", 2048, 4096, 1, 1, 32, "bfloat16", dict(causal=False)),
    ("fp4", 2048, 4096, 2, 1, 128, "bfloat16", {}),
])
def test_public_call_in_pieces(entry, sq, sk, h, hk, d, dtype, kw, tmp_path):
    """The call takes the split schedule on its own."""
    import flamia_blackwell_attention_b200 as F
    from launches import launches
    q, k, v, _ = (t.to(getattr(torch, dtype)) for t in attention_inputs(1, max(sq, sk), h, hk, d, seed=13))
    q, k, v = q[:, :sq].contiguous(), k[:, :sk].contiguous(), v[:, :sk].contiguous()
    causal = kw.get("causal", True)
    fn = F.flash_attn_fp4 if entry == "fp4" else F.flash_attn_fp8
    x = [t.cuda() for t in (q, k, v)]
    with torch.no_grad():
        names = [n for n, _, _ in launches(lambda: fn(*x, causal=causal), tmp_path)]
        out, lse = fn(*x, causal=causal, return_lse=True)
    assert any("fwd_merge" in n for n in names), names
    if d == 128:        # against the same quantised operands (rotated by default), as in test_gpu_fwd.py
        ro, rl, *_ = A.qdq_attention(q, k, v, causal=causal, fp4_qk=entry == "fp4", rotate_qk=True)
        assert A.accuracy(out.float().cpu(), ro)["rel_l2"] < 3.2e-2
        assert float((lse.cpu() - rl).abs().max()) < 2e-3
    else:               # (padded head dims: against fp32 attention, as in test_gpu_api.py)
        assert A.accuracy(out.float().cpu(), A.attention_fp32(q.float(), k.float(), v.float(), None, causal)[0])["rel_l2"] < 8e-2
