"""Quantiser launches of more tiles than three rounds, whose warps past a document's end write zeros and do nothing else, against launches
that treat every row alike; and the forward's form for short documents against its other ones: bit for bit."""
import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu


def _slots(lens):
    """(slot_src, slot_rows, rows of the aligned buffer) of documents back to back, and two empty slots."""
    src, rows, at = [], [], 0
    for n in lens:
        for r in range(0, n, 128):
            src.append(at + r)
            rows.append(min(128, n - r))
        at += n
    src, rows = src + [-1, -1], rows + [0, 0]
    return torch.tensor(src, dtype=torch.int32).cuda(), torch.tensor(rows, dtype=torch.int32).cuda(), 128 * len(src)


def _same(a, b, names):
    for n in names:
        assert torch.equal(a[n].view(torch.uint8), b[n].view(torch.uint8)), n


LENS = [1, 8, 9, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 300] * 30      # edges of warps and tiles


@pytest.mark.parametrize("d,rotate,nvfp4,dtype", [(128, True, False, "bfloat16"), (128, True, True, "float16"), (128, False, True, "bfloat16"),
                                                  (64, False, False, "float16"), (128, False, False, "bfloat16")])
def test_rows_kernel(d, rotate, nvfp4, dtype):
    from flamia_blackwell_attention_b200 import kernels as K
    x = attention_inputs(1, sum(LENS), 4, 1, d, seed=61)[0][0].to(getattr(torch, dtype)).cuda()
    kw = dict(packed_slots=_slots(LENS), output_tile_stats=True, also_make_nvfp4_copy=nvfp4, apply_hadamard_rotation=rotate,
              hadamard_rotation_scope="nvfp4_copy" if nvfp4 else "all")
    many, plain = K.quantize_fp8_blocks(x, **kw), K.quantize_fp8_blocks(x, legacy_kernel=True, **kw)
    _same(many, plain, ("codes", "fac", "e", "tile_stats") + (("x4", "sf4_raw") if nvfp4 else ()))


@pytest.mark.parametrize("d,o_packed", [(128, True), (64, True), (128, False)])
def test_prologue(d, o_packed):
    """Heads for more than three rounds (either form of the prologue; two heads: of one of them) against a head at a time."""
    from flamia_blackwell_attention_b200 import kernels as K
    lens = LENS[:192]
    slots = _slots(lens)
    h, s = 6, slots[2]
    x, o = (t[0].cuda() for t in attention_inputs(1, sum(lens), h, h, d, seed=62)[:2])
    if not o_packed:
        o = torch.randn(1, s, h, d, device="cuda").to(x.dtype)
    lse = torch.randn(1, h, s, device="cuda")

    def run(heads):
        acc = torch.full((1, heads.stop - heads.start, s, d), 7.0, dtype=torch.float16, device="cuda")
        got = K.quantize_fp8_blocks(x[:, heads].contiguous(), packed_slots=slots, compute_d_with_output=o[..., heads, :].contiguous(),
                                    shifted_log2_lse_from=lse[:, heads].contiguous(), log2_lse_shift=8.0, d_multiplier=-2.0 ** -8, zero_accumulator=acc,
                                    output_tile_stats=True)
        assert not acc.any()
        return got
    for n in (2, 5, h):          # (five: the form of two steps)
        many = run(slice(0, n))
        for i in range(n):
            one = run(slice(i, i + 1))
            assert torch.equal(many["codes"][:, :, i].view(torch.uint8), one["codes"][:, :, 0].view(torch.uint8))
            _same({k: many[k][:, i].contiguous() for k in ("fac", "D", "lse_log2", "tile_stats")},
                  {k: one[k][:, 0].contiguous() for k in ("fac", "D", "lse_log2", "tile_stats")}, ("fac", "D", "lse_log2", "tile_stats"))


@pytest.mark.parametrize("lens", [[1, 127, 128, 129, 2, 256, 64, 130, 3], [40] * 30 + [128, 384], [190, 193] * 4])
@pytest.mark.parametrize("entry,d,kw", [("fp8", 128, dict(causal=True)), ("fp8", 64, dict()), ("fp8", 80, dict(causal=True, softcap=20.0)),
                                        ("fp8", 128, dict(causal=True, window_size=(60, 0))), ("fp4", 128, dict(causal=True)), ("fp4", 128, dict())])
def test_forward(lens, entry, d, kw):
    """Documents of fewer than 192 rows on average, against the same documents with a long one behind them that lifts the average."""
    import flamia_blackwell_attention_b200 as F
    fn = F.flash_attn_fp4 if entry == "fp4" else F.flash_attn_fp8
    long = lens + [192 * (len(lens) + 1)]
    x = [t[0].cuda() for t in attention_inputs(1, sum(long), 4, 2, d, seed=63)[:3]]
    (o, lse), (ol, lsel) = _forward(fn, x, lens, **kw), _forward(fn, x, long, **kw)
    assert F.check_status() == 0
    n = sum(lens)
    assert torch.equal(o, ol[:n]) and torch.equal(lse, lsel[:, :n])


def _forward(fn, x, lens, **kw):
    import flamia_blackwell_attention_b200 as F
    maps = F.DocMaps.from_cu_seqlens(torch.tensor([0] + lens, dtype=torch.int32).cumsum(0, dtype=torch.int32)).to("cuda")
    with torch.no_grad():
        return fn(*(t[:sum(lens)] for t in x), doc_maps=maps, return_lse=True, **kw)


def test_which_documents_are_short(tmp_path):
    import flamia_blackwell_attention_b200 as F
    from launches import launches
    x = [torch.zeros(400, 1, 128, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
    for lens, form in (([191, 192], ", 2>"), ([191, 193], ", 1>")):
        names = [n for n, _, _ in launches(lambda: _forward(F.flash_attn_fp8, x, lens), tmp_path) if "fwd_kernel" in n]
        assert len(names) == 1 and form in names[0], names
