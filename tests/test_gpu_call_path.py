"""GPU: the launches of a whole call against the single-operand kernels: the one-launch Q / K / V quantiser (batched, packed rows,
head dims read with zero columns), the document tables and the LSE's way back, bit for bit."""
import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu

LENS = [300, 1, 128, 77, 515, 127, 129]


def _state(entry, q, k, v, docs, **kw):
    """(out, lse, state) of the registered op under the plan of these arguments, with gradients in the plan."""
    import flamia_blackwell_attention_b200 as F
    from flamia_blackwell_attention_b200 import _op
    q, k, v = (t.clone().requires_grad_(True) for t in (q, k, v))
    plan = (F.resolve_fp8 if entry == "fp8" else F.resolve_fp4)(q, k, v, causal=True, **kw)
    pid = _op.register_plan(plan)
    return getattr(torch.ops.lowbit_attn, entry)(q.detach(), k.detach(), v.detach(), docs, pid, 0)


@pytest.mark.parametrize("entry,d,dtype", [("fp8", 128, "bfloat16"), ("fp4", 128, "float16"), ("fp8", 64, "bfloat16"), ("fp8", 96, "float16"),
                                           ("fp8", 80, "bfloat16"), ("fp8", 32, "bfloat16")])
@pytest.mark.parametrize("form", ["batched", "packed"])
def test_one_launch_quantiser_equals_single_launches(entry, d, dtype, form):
    from flamia_blackwell_attention_b200 import kernels as K
    h, hk, dt = 3, 1, getattr(torch, dtype)
    dp = d if d in (64, 128) else (64 if d < 64 else 128)
    rot = dict(apply_hadamard_rotation=d == 128, hadamard_rotation_scope="nvfp4_copy" if entry == "fp4" else "all",
               also_make_nvfp4_copy=entry == "fp4")
    if form == "batched":
        q, k, v, _ = (t.to(dt).cuda() for t in attention_inputs(2, 384, h, hk, d, seed=3))
        _, _, st = _state(entry, q, k, v, [])
        slots, base = None, 0
    else:
        q, k, v, _ = (t[0].to(dt).cuda() for t in attention_inputs(1, sum(LENS), h, hk, d, seed=3))
        cu = torch.tensor([0] + list(torch.tensor(LENS).cumsum(0)), dtype=torch.int32, device="cuda")
        _, _, st = _state(entry, q, k, v, [cu, cu], cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(LENS), max_seqlen_k=max(LENS))
        slots, base = (st[-4], st[-3], st[-5].numel()), 1
    pad = lambda t: torch.nn.functional.pad(t, (0, dp - d))      # noqa: E731
    want = [K.quantize_fp8_blocks(pad(t), legacy_kernel=True, packed_slots=slots, output_tile_stats=i > 0, **(rot if i < 2 else {}))
            for i, t in enumerate((q, k, v))]
    for i, w in enumerate(want):
        assert torch.equal(st[base + 2 * i].view(torch.uint8), w["codes"].view(torch.uint8)), i
        assert torch.equal(st[base + 2 * i + 1], w["fac"]), i
    assert torch.equal(st[base + 7], want[1]["tile_stats"]) and torch.equal(st[base + 8], want[2]["tile_stats"])
    if d == dp and slots is None:                        # the wrapper of the same launch
        for w, got in zip(want, K.quantize_qkv(q, k, v, output_tile_stats=True, **rot)):
            assert w.keys() == got.keys() and all(torch.equal(w[n].view(torch.uint8), got[n].view(torch.uint8)) for n in w)
    if entry == "fp4":
        for i in range(2):
            assert torch.equal(st[base + 9 + 2 * i], want[i]["x4"]) and torch.equal(st[base + 10 + 2 * i], want[i]["sf4_raw"])


@pytest.mark.parametrize("lens", [LENS, [5], [128] * 3, [1] * 700, [2049, 3]])
def test_document_tables_in_one_launch(lens):
    """fl_doc_tables against the host construction, and the call's LSE rows in the caller's order."""
    from flamia_blackwell_attention_b200._routes import Docs
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    total = int(cu[-1])
    ref = Docs(cu, cu[1:] - cu[:-1], total, False)
    q, k, v, _ = (t[0].cuda() for t in attention_inputs(1, total, 2, 1, 64, seed=4))
    c = cu.cuda()
    _, lse, st = _state("fp8", q, k, v, [c, c], cu_seqlens_q=c, cu_seqlens_k=c, max_seqlen_q=max(lens), max_seqlen_k=max(lens), return_lse=True)
    for name, t in zip(("start", "len", "row_map", "slot_src", "slot_rows"), st[-7:-2]):
        assert torch.equal(t.cpu(), getattr(ref, name)), name
    rows = ref.row_map.cuda().long()
    assert torch.equal(lse[:, rows[rows >= 0]], st[0][0][:, rows >= 0])


@pytest.mark.parametrize("b,s,h", [(1, 1, 1), (3, 127, 2), (5, 128, 1), (2, 300, 3), (40, 129, 1)])
def test_documents_of_one_length(b, s, h):
    """The forms for hosts that run batch rows as documents: fl_doc_tables without boundaries, fl_unpack_lse into (b, h, s)."""
    from flamia_blackwell_attention_b200 import _lib as L
    total, capacity = b * s, b * ((s + 127) // 128 * 128)
    stream = torch.cuda.current_stream().cuda_stream

    def tables(cu):
        t = [torch.full((n,), 7, dtype=torch.int32, device="cuda") for n in (b, b, capacity, capacity // 128, capacity // 128)]
        L.check(L.load().fl_doc_tables(L.ptr(cu), b, s if cu is None else 0, total, capacity, *(L.ptr(x) for x in t), stream), "fl_doc_tables")
        return t
    got, want = tables(None), tables(torch.arange(0, total + 1, s, dtype=torch.int32, device="cuda"))
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    lse, out = torch.randn(h, capacity, device="cuda"), torch.empty(b, h, s, device="cuda")
    L.check(L.load().fl_unpack_lse(L.ptr(lse), L.ptr(got[3]), L.ptr(got[4]), capacity, h, s, total, L.ptr(out), stream), "fl_unpack_lse")
    assert torch.equal(out, lse.view(h, b, -1)[..., :s].transpose(0, 1))


@pytest.mark.parametrize("b,h,hk,nt,causal", [(1, 1, 1, 1, False), (3, 5, 5, 7, False), (2, 16, 4, 40, False), (2, 3, 1, 9, True)])
def test_dq_prescale_of_many_tiles(b, h, hk, nt, causal):
    """The pre-scale table against the maxima taken directly (the bound's arithmetic itself is pinned elsewhere)."""
    from flamia_blackwell_attention_b200 import kernels as K
    g = torch.Generator().manual_seed(5)
    do, v, k = (torch.rand(b, n, nt, 2, generator=g).cuda() * 100 for n in (h, hk, hk))
    ks, ps = K.dq_prescale(do, v, k, causal_local=causal)
    for t in range(nt):
        q_sl, k_sl = (slice(t, t + 1), slice(0, t + 1)) if causal else (slice(0, nt), slice(0, nt))
        bound = 8.0 * do[:, :, q_sl, 1].amax((1, 2)).sqrt() * v[:, :, k_sl, 1].amax((1, 2)).sqrt() * k[:, :, k_sl, 0].amax((1, 2))
        want = torch.exp2(torch.floor(torch.log2(65504.0 / bound)))
        assert torch.equal(ks[:, t], want) and torch.equal(ps[:, t], 1.0 / want)


@pytest.mark.parametrize("lens,kw", [(LENS, {}), ([1] * 1100 + [700], {}), ([5000, 3, 1300], dict(window_size=(400, 0))),
                                     ([640, 128, 256], dict(deterministic=True))])
def test_work_list_changes_nothing(lens, kw):
    """Documents through fl_doc_work's lists (several chunks of its scan, equal costs, a window, document order) against the kernel's
    own walk over the document table: O, LSE, dK and dV bit for bit (with an ordered dQ its accumulator, too), every pair exactly
    once, in document order or longest first."""
    from flamia_blackwell_attention_b200 import kernels as K
    h, hk, d = 3, 1, 128
    total = sum(lens)
    q, k, v, _ = (t[0].cuda() for t in attention_inputs(1, total, h, hk, d, seed=6))
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    out, _, st = _state("fp8", q, k, v, [cu, cu], cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(lens), max_seqlen_k=max(lens), **kw)
    start, length, row_map, slot_src, slot_rows, work = st[-7:-1]
    n_f, n_b = work[:2].tolist()
    tiles = row_map.numel() // 128
    pairs = work[4:4 + 8 * tiles].view(2, tiles, 4)
    for part, rows, n in ((pairs[0], 256, n_f), (pairs[1], 128, n_b)):
        got = sorted((s, m, b) for s, m, b, _ in part[:n].tolist())
        assert got == sorted((s, m, b) for s, m in zip(start.tolist(), length.tolist()) for b in range((m + rows - 1) // rows))
    ops = [dict(codes=st[1 + 2 * i].view(torch.uint8), fac=st[2 + 2 * i]) for i in range(3)]
    want, lse, _ = K.attn_fwd(*ops, causal=True, softmax_scale=d ** -0.5, window=kw.get("window_size"),
                              packed_out=(slot_src, slot_rows, total), doc_start=start, doc_len=length)
    live = row_map >= 0
    assert torch.equal(out, want[0]) and torch.equal(st[0][0][:, live], lse[0][:, live])
    # the order of the lists: as the documents lie (the ordered dQ waits for entries before it), or no block before a longer one
    left = kw["window_size"][0] if "window_size" in kw else max(lens)
    for part, rows, n in ((pairs[0], 256, n_f), (pairs[1], 128, n_b)):
        raw = [tuple(e[:3]) for e in part[:n].tolist()]
        if kw.get("deterministic"):
            assert raw == sorted((s, m, b) for s, m, b in raw)
            continue
        cost = []
        for _, m, b in raw:
            if rows == 256:      # key tiles of both halves of the block, from the window's first key on
                lo = max(0, b * 256 - left) // 128 * 128
                cost.append(sum((min(m, b * 256 + i + 128) - lo + 127) // 128 for i in (0, 128) if b * 256 + i < m))
            else:                # query tiles from the diagonal to the window's last one
                cost.append(min((m + 127) // 128, (min(m, b * 128 + 128) - 1 + left) // 128 + 1) - b)
        assert cost == sorted(cost, reverse=True)
    # the backward, both ways, from the same operands
    docs = dict(doc_start=start, doc_len=length)
    g = attention_inputs(1, total, h, hk, d, seed=6)[3][0].cuda()
    res = []
    for lists in (None, work):
        acc = torch.empty(1, h, row_map.numel(), d, dtype=torch.float16, device="cuda")
        gq = K.quantize_fp8_blocks(g, packed_slots=(slot_src, slot_rows, row_map.numel()), compute_d_with_output=out, shifted_log2_lse_from=st[0],
                                   log2_lse_shift=8.0, d_multiplier=-2.0 ** -8, zero_accumulator=acc, output_tile_stats=True)
        ks, _ = K.dq_prescale(gq["tile_stats"], st[9], st[8])
        order = torch.zeros(1, h, tiles, 2, dtype=torch.int32, device="cuda") if kw.get("deterministic") else None
        dk, dv, status = K.attn_bwd(*ops, gq, lse_log2=gq["lse_log2"], d_rows=gq["D"], dq_acc=acc, dq_scale=ks, causal=True, softmax_scale=d ** -0.5,
                                    window=kw.get("window_size"), packed_out=(slot_src, slot_rows, total), dq_order=order, work=lists, **docs)
        assert K.read_status(status) == 0
        res.append((dk, dv) + ((acc,) if kw.get("deterministic") else ()))
    for a, b in zip(*res):
        assert torch.equal(a, b)
