"""The backward prologue's launch (quantised dO, D, shifted LSE, zeroed accumulator): its forms against each other and against the plain
quantiser, bit for bit."""
import pytest
import torch

from launches import launches

pytestmark = pytest.mark.gpu


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def _inputs(b, s, h, d, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(b, s, h, d, generator=gen, device="cuda")
    x *= torch.exp2(torch.randint(-12, 12, (b, s, h, 1), generator=gen, device="cuda").float())     # rows, blocks and tiles of other exponents
    x[:, 5::97] = 0.0
    o = torch.randn(b, s, h, d, generator=gen, device="cuda")
    lse = torch.randn(b, h, s, generator=gen, device="cuda")
    lse[:, :, 3::101] = -float("inf")
    return x.bfloat16(), o.bfloat16(), lse


def _prologue(x, o, lse, s=None, **kw):
    from flamia_blackwell_attention_b200 import kernels as K
    b, h, d = (1 if x.dim() == 3 else x.shape[0]), x.shape[-2], x.shape[-1]
    acc = torch.full((b, h, s or x.shape[1], d), 7.0, dtype=torch.float16, device="cuda")
    got = K.quantize_fp8_blocks(x, compute_d_with_output=o, shifted_log2_lse_from=lse, log2_lse_shift=8.0, d_multiplier=-2.0 ** -8,
                                zero_accumulator=acc, **kw)
    assert not acc.any()
    return got


def _threads(fn, tmp_path):
    return [block for name, _, block in launches(fn, tmp_path) if "quant_blocks" in name]


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("rounds,extra,threads", [
    (0, 1, 512), (0, 16, 512), (1, 0, 512),        # no more than a tile an SM: nothing would cover a tile taken in two steps
    (1, 1, 256), (2, 0, 256),
    (2, 1, 512), (3, 0, 512), (3, 1, 256), (4, 0, 256),
    (4, 1, 256), (5, 0, 512), (6, 0, 256),         # five rounds: the last one has a tile an SM again
])
def test_launch_shape(d, rounds, extra, threads, tmp_path):
    x, o, lse = _inputs(1, 128 * (rounds * _sms() + extra), 1, d)
    assert _threads(lambda: _prologue(x, o, lse), tmp_path) == [(threads, 1, 1)]


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("tiles", [1, 160, 1000])
def test_channel_major_copy_takes_a_tile_at_once(tiles, d, tmp_path):
    from flamia_blackwell_attention_b200 import kernels as K
    x, o, lse = _inputs(1, 128 * tiles, 1, d)
    got = []
    assert _threads(lambda: got.append(_prologue(x, o, lse, make_channel_major_copy=True)), tmp_path) == [(512, 1, 1)]
    _equal(got[0], K.quantize_fp8_blocks(x, make_channel_major_copy=True), ("codes", "codes_t", "fac"), "plain")


def _equal(got, want, keys, what):
    for k in keys:
        a, b = (t[k].contiguous().view(torch.uint8) for t in (got, want))
        assert torch.equal(a, b), (what, k, int((a != b).sum()))


TABLES = ("codes", "e", "fac", "sf_tok_raw", "sf_dim_raw", "tile_stats")


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("token_local", [False, True])
@pytest.mark.parametrize("tiles", [1, 29, 61])       # of 3 x 5 heads: 915 are four rounds of two blocks an SM (two steps), 435 three of one
def test_every_output_equals_the_plain_launch(tiles, token_local, d):
    from flamia_blackwell_attention_b200 import kernels as K
    b, s, h = 3, 128 * tiles, 5
    x, o, lse = _inputs(b, s, h, d)
    stats = [torch.zeros(b, s, device="cuda") for _ in range(2)]
    kw = dict(output_sf_atoms=True, output_tile_stats=True, token_local_exponents=token_local)
    got = _prologue(x, o, lse, row_stat=("sumsq", stats[0]), **kw)
    want = K.quantize_fp8_blocks(x, legacy_kernel=True, row_stat=("sumsq", stats[1]), **kw)
    _equal(got, want, TABLES + (("token_factors",) if token_local else ()), "plain")
    assert torch.equal(*stats)
    for i in range(b):                                # D and the LSE: a batch row alone is a launch of another grid, here of one step
        _equal({k: got[k][i:i + 1] for k in ("D", "lse_log2")}, _prologue(x[i:i + 1], o[i:i + 1], lse[i:i + 1], **kw), ("D", "lse_log2"), i)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("last", [1, 65])             # the last document's second half box starts past the source, or one row before its end
@pytest.mark.parametrize("slots,o_packed", [(7, True), (61, True), (183, True), (183, False)])      # of 5 heads: 35, 305 (one step), 915 tiles (two)
def test_packed_rows_equal_the_aligned_buffer(slots, o_packed, last, d):
    lens = [[1, 63, 64, 0, 65, 127, 128][i % 7] for i in range(slots - 1)] + [last]
    h, s, total = 5, 128 * slots, sum(lens)
    first = [sum(lens[:i]) for i in range(slots)]
    src = torch.tensor([f if n else -1 for f, n in zip(first, lens)], dtype=torch.int32, device="cuda")
    rows = torch.tensor(lens, dtype=torch.int32, device="cuda")
    at = torch.tensor([128 * i + r for i, n in enumerate(lens) for r in range(n)], device="cuda")
    x, o, lse = _inputs(1, s, h, d, seed=1)
    xp, op = x[0, :total].contiguous(), o[0, :total].contiguous()
    xa, oa = torch.zeros_like(x), torch.zeros_like(o)
    xa[0, at], oa[0, at] = xp, op
    stats = [torch.zeros(1, s, device="cuda") for _ in range(2)]
    kw = dict(output_sf_atoms=True, output_tile_stats=True)
    got = _prologue(xp, op if o_packed else oa, lse, s=s, packed_slots=(src, rows, s), row_stat=("sumsq", stats[0]), **kw)
    want = _prologue(xa, oa, lse, row_stat=("sumsq", stats[1]), **kw)
    _equal(got, want, TABLES + ("D", "lse_log2"), "aligned")
    assert torch.equal(*stats)
