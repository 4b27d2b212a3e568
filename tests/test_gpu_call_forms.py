"""GPU: forms of a call (masks, layouts, document tables, transforms around it) against the same call in its plain form."""
import pytest
import torch

from inputs import attention_inputs

pytestmark = pytest.mark.gpu


def _step(fn, q, k, v, do, **kw):
    """(out, dq, dk, dv) of one call; deterministic, so that two calls on the same values compare bit for bit."""
    q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
    out = fn(q, k, v, deterministic=True, **kw)
    return (out.detach(), *torch.autograd.grad(out, (q, k, v), do))


@pytest.mark.parametrize("s", [256, 1000])             # whole tiles; batch rows that are none
@pytest.mark.parametrize("window,same", [((2 ** 31 - 2, 2 ** 31 - 2), (None, None)), ((2 ** 31 - 2, 100), (None, 100)),
                                         ((100, 2 ** 31 - 2), (100, None)), ((2 ** 33 + 5, 2 ** 31 - 1), (None, None))])
def test_window_longer_than_any_sequence(s, window, same):
    import flamia_blackwell_attention_b200 as F
    x = [t.cuda() for t in attention_inputs(2, s, 2, 1, 64, seed=11)]
    for a, b in zip(_step(F.flash_attn_fp8, *x, window_size=window), _step(F.flash_attn_fp8, *x, window_size=same)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("entry,d,opts", [("fp8", 128, {}), ("fp8", 64, {}), ("fp4", 128, {}), ("fp8", 128, dict(ds_dq_rowlocal="all")),
                                          ("fp8", 128, dict(operand_scaling="token_local", ds_dq_rowlocal="all"))])
@pytest.mark.parametrize("s,hk,causal", [(128, 4, False), (256, 4, True), (384, 2, False)])
def test_dk_dv_of_items_with_few_query_tiles(entry, d, opts, s, hk, causal):
    """Every key tile's dK and dV are sums in a fixed order, so they repeat bit for bit; items of one to six query tiles, where an
    item's first and last iteration (whose hand-overs differ) are most of them, and several items a CTA."""
    import flamia_blackwell_attention_b200 as F
    fn = F.flash_attn_fp8 if entry == "fp8" else F.flash_attn_fp4
    kw = dict(options=(F.FP8AttnOptions if entry == "fp8" else F.FP4AttnOptions)(**opts)) if opts else {}
    q, k, v, do = (t.cuda() for t in attention_inputs(128, s, 4, hk, d, seed=12))
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    first = None
    for _ in range(10):
        dk, dv = torch.autograd.grad(fn(q, k, v, causal=causal, **kw), (k, v), do)
        first = first or (dk, dv)
        assert torch.equal(dk, first[0]) and torch.equal(dv, first[1])


@pytest.mark.parametrize("causal", [False, True])
def test_key_tiles_that_no_query_sees(causal):
    """seqused_k far below s_k: most key tiles are items without query tiles, many in a row for each CTA, beside an ordered dQ whose
    reduction is still waiting for its turn. Bit for bit the same again; dense: bit for bit the call on the keys in use alone."""
    import flamia_blackwell_attention_b200 as F
    b, s, used = 2, 4096, 256
    q, k, v, do = (t.cuda() for t in attention_inputs(b, s, 8, 8, 128, seed=13))
    k[:, used:], v[:, used:] = 0, 0                      # (the f16 pre-scale of dQ is sized from all keys)
    su = torch.full((b,), used, dtype=torch.int32, device="cuda")
    first = _step(F.flash_attn_fp8, q, k, v, do, causal=causal, seqused_k=su)
    for x, y in zip(first, _step(F.flash_attn_fp8, q, k, v, do, causal=causal, seqused_k=su)):
        assert torch.equal(x, y)
    assert not first[2][:, used:].any() and not first[3][:, used:].any()
    if not causal:
        out, dq, dk, dv = _step(F.flash_attn_fp8, q, k[:, :used], v[:, :used], do)
        assert torch.equal(out, first[0]) and torch.equal(dq, first[1])
        assert torch.equal(dk, first[2][:, :used]) and torch.equal(dv, first[3][:, :used])


@pytest.mark.parametrize("entry", ["fp8", "fp4"])
def test_documents_of_a_pack_equal_their_own_calls(entry):
    """Several short items per CTA, most of them partly filled (rows stored one by one): O and LSE of every document bit for bit those of
    a call on that document alone, time after time."""
    import flamia_blackwell_attention_b200 as F
    fn = F.flash_attn_fp8 if entry == "fp8" else F.flash_attn_fp4
    lens = [1, 300, 77, 128, 129, 256, 5, 640, 31, 200] * 4
    edges = [0] + list(torch.tensor(lens).cumsum(0))
    q, k, v, _ = (t[0].cuda() for t in attention_inputs(1, sum(lens), 16, 16, 128, seed=14))

    def call(lo, hi, cu):
        cu = torch.tensor(cu, dtype=torch.int32, device="cuda")
        return fn(q[lo:hi], k[lo:hi], v[lo:hi], causal=True, cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=640, max_seqlen_k=640, return_lse=True)
    alone = [call(lo, hi, [0, hi - lo]) for lo, hi in zip(edges[:10], edges[1:11])]
    for _ in range(5):
        out, lse = call(0, edges[-1], edges)
        for i in range(10):
            lo, hi = edges[i], edges[i + 1]
            assert torch.equal(out[lo:hi], alone[i][0]) and torch.equal(lse[:, lo:hi], alone[i][1]), i


@pytest.mark.parametrize("first,last", [(0, 700), (64, 764)])
def test_lse_of_rows_that_no_document_covers(first, last):
    """A token buffer longer than its documents: their LSE rows are those of the exact pack, the others zeros."""
    import flamia_blackwell_attention_b200 as F
    q, k, v, _ = (t[0].cuda() for t in attention_inputs(1, 900, 2, 2, 64, seed=15))
    kw = dict(causal=True, max_seqlen_q=400, max_seqlen_k=400, return_lse=True)
    cu = torch.tensor([first, first + 300, last], dtype=torch.int32, device="cuda")
    own = cu - first
    del [torch.full((2, 900), float("nan"), device="cuda") for _ in range(64)][:]      # (what the allocator hands out next)
    lse = F.flash_attn_fp8(q, k, v, cu_seqlens_q=cu, cu_seqlens_k=cu, **kw)[1]
    want = F.flash_attn_fp8(*(t[first:last] for t in (q, k, v)), cu_seqlens_q=own, cu_seqlens_k=own, **kw)[1]
    assert torch.equal(lse[:, first:last], want)
    assert not lse[:, :first].any() and not lse[:, last:].any()


def test_tables_on_another_device_are_refused():
    """Host tensors (cu_seqlens, seqused_*, maps, k) and tables of another type or size are an error before the first launch."""
    import flamia_blackwell_attention_b200 as F
    from flamia_blackwell_attention_b200 import _op
    q = torch.randn(384, 2, 64, device="cuda", dtype=torch.bfloat16)
    cu, su = torch.tensor([0, 128, 384], dtype=torch.int32), torch.tensor([100, 256], dtype=torch.int32)
    packed = dict(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=256, max_seqlen_k=256)
    aligned = dict(packed, cu_seqlens_q=cu.cuda())
    aligned["cu_seqlens_k"] = aligned["cu_seqlens_q"]
    for kw in (packed, dict(aligned, seqused_q=su, seqused_k=su)):
        with pytest.raises(RuntimeError, match="on q's device"):
            F.flash_attn_fp8(q, q, q, **kw)
    long = su.cuda().repeat(2)
    with pytest.raises(RuntimeError, match="one seqused entry per document"):
        F.flash_attn_fp8(q, q, q, **dict(aligned, seqused_q=long, seqused_k=long))
    q4 = q.view(3, 128, 2, 64)
    with pytest.raises(RuntimeError, match="on q's device"):
        F.flash_attn_fp8(q4, q4, q4, seqused_k=torch.tensor([128, 5, 7], dtype=torch.int32))
    with pytest.raises(RuntimeError, match="must be CUDA tensors"):
        F.flash_attn_fp8(q4, q4.cpu(), q4)
    q8, one = q4.to(torch.float8_e4m3fn), torch.ones(3, 2, device="cuda")
    pre = dict(q_descale=one, k_descale=one, v_descale=one)
    with pytest.raises(ValueError, match="one device"):
        F.flash_attn_fp8(q8, q8, q8.cpu(), **pre)
    with pytest.raises(ValueError, match="codes' device"):
        F.flash_attn_fp8(q8, q8, q8, seqused_k=torch.tensor([128, 5, 7], dtype=torch.int32), **pre)
    maps = F.DocMaps.from_cu_seqlens(cu).to("cuda")
    pid = _op.register_plan(F.resolve_fp8(q, q, q, **packed))
    for bad in (lambda t: t[:4] + [t[4][:-1], t[5]], lambda t: [x.long() for x in t]):
        with pytest.raises(RuntimeError, match="document maps"):
            torch.ops.lowbit_attn.fp8(q, q, q, bad(maps.tensors()), pid, 0)


@pytest.mark.parametrize("d", [16, 48, 80, 96])
@pytest.mark.parametrize("form", ["batched", "ragged", "packed"])
def test_padded_head_dims_at_any_address(d, form):
    """Inputs and an output gradient that start two bytes past an aligned address: bit for bit the aligned call."""
    import flamia_blackwell_attention_b200 as F
    x = [t.cuda() for t in attention_inputs(2, 250 if form == "ragged" else 256, 4, 2, d, seed=16)]
    kw = dict(causal=True)
    if form == "packed":
        cu = torch.tensor([0, 77, 512], dtype=torch.int32, device="cuda")
        x, kw = [t.flatten(0, 1) for t in x], dict(kw, cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=435, max_seqlen_k=435)

    def odd(t):
        y = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape)
        return y.copy_(t)
    for a, b in zip(_step(F.flash_attn_fp8, *map(odd, x), **kw), _step(F.flash_attn_fp8, *x, **kw)):
        assert torch.equal(a, b)


def test_tensor_subclass_goes_through_the_op():
    import flamia_blackwell_attention_b200 as F
    seen = []

    class Sub(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", ""))
            return super().__torch_function__(func, types, args, kwargs or {})
    q, k, v, _ = (t.cuda() for t in attention_inputs(1, 256, 2, 2, 64, seed=17))
    out = F.flash_attn_fp8(q.as_subclass(Sub), k, v, causal=True)
    assert type(out) is Sub and "fp8" in seen
    assert torch.equal(out.as_subclass(torch.Tensor), F.flash_attn_fp8(q, k, v, causal=True))


@pytest.mark.parametrize("form", ["batched", "packed", "aligned", "ragged"])
def test_compiled_autograd(form):
    """A backward traced by compiled autograd, after an eager forward and after a traced one: the eager gradients."""
    import flamia_blackwell_attention_b200 as F
    x, kw = [t.cuda() for t in attention_inputs(2, 250 if form == "ragged" else 256, 2, 2, 128, seed=18)], dict(causal=True)
    if form in ("packed", "aligned"):
        cu = torch.tensor([0, 128, 512], dtype=torch.int32, device="cuda")
        x, kw = [t.flatten(0, 1) for t in x], dict(kw, cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=384, max_seqlen_k=384)
        if form == "aligned":
            su = torch.tensor([100, 384], dtype=torch.int32, device="cuda")
            kw.update(seqused_q=su, seqused_k=su)
    for traced in (False, True):
        torch._dynamo.reset()
        for kw["causal"] in (True, False):               # (the same shapes, another plan: not the first one's trace again)
            fn = lambda q, k, v: F.flash_attn_fp8(q, k, v, deterministic=True, **kw)      # noqa: E731
            q, k, v = (t.detach().requires_grad_(True) for t in x[:3])
            with torch._dynamo.config.patch(compiled_autograd=True):
                out = (torch.compile(fn, backend="aot_eager") if traced else fn)(q, k, v)
                torch.compile(lambda: out.backward(x[3]), backend="aot_eager")()
            for a, b in zip((out.detach(), q.grad, k.grad, v.grad), _step(F.flash_attn_fp8, *x, **kw)):
                assert torch.equal(a, b)


def test_compiled_autograd_with_maps_of_several_sizes():
    """One plan, buffers of other sizes from call to call (what makes a trace take sizes as symbols)."""
    import flamia_blackwell_attention_b200 as F
    x = [t.flatten(0, 1).cuda() for t in attention_inputs(2, 256, 2, 2, 64, seed=20)]
    for size in (512, 640, 896, 1024):
        maps = F.DocMaps.from_cu_seqlens(torch.tensor([0, 128, 512]), padded_size=size).to("cuda")
        q, k, v = (t.detach().requires_grad_(True) for t in x[:3])
        with torch._dynamo.config.patch(compiled_autograd=True):
            out = F.flash_attn_fp8(q, k, v, causal=True, deterministic=True, doc_maps=maps)
            torch.compile(lambda: out.backward(x[3]), backend="aot_eager")()
        for a, b in zip((out.detach(), q.grad, k.grad, v.grad), _step(F.flash_attn_fp8, *x, causal=True, doc_maps=maps)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("form", ["batched", "fp4", "rows", "packed", "maps", "aligned", "seqused", "ragged"])
def test_state_tensors_have_a_storage_each(form):
    """What the op returns shares no memory, with its inputs neither, as its schema says."""
    import flamia_blackwell_attention_b200 as F
    import flamia_blackwell_attention_b200.interface_bwd_fp4 as switches
    from flamia_blackwell_attention_b200 import _op
    entry = "fp4" if form == "fp4" else "fp8"
    packed = form in ("packed", "maps", "aligned")
    x = torch.randn(*((640, 2, 128) if packed else (2, 300 if form == "ragged" else 256, 2, 128)), device="cuda", dtype=torch.bfloat16)
    kw, docs, was = dict(causal=True), [], (switches.DQ_CAUSAL_PRESCALE, switches.DQ_CAUSAL_GRANULARITY)
    if packed:
        cu = torch.tensor([0, 128, 640], dtype=torch.int32, device="cuda")
        kw.update(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=512, max_seqlen_k=512)
        docs = [cu, cu] if form != "maps" else F.DocMaps.from_cu_seqlens(cu.cpu()).to("cuda").tensors()
    if form in ("aligned", "seqused"):
        su = torch.tensor([100, 200], dtype=torch.int32, device="cuda")
        kw.update(seqused_k=su, **(dict(seqused_q=su) if packed else {}))
        docs = docs + [su, su] if packed else [su]
    try:
        if form == "rows":
            switches.DQ_CAUSAL_PRESCALE, switches.DQ_CAUSAL_GRANULARITY = True, "row"
        plan = (F.resolve_fp4 if entry == "fp4" else F.resolve_fp8)(x.requires_grad_(True), x, x, **kw)
    finally:
        switches.DQ_CAUSAL_PRESCALE, switches.DQ_CAUSAL_GRANULARITY = was
    assert plan.bwd.dq_prescale == ("causal_row" if form == "rows" else "row")
    out, lse, state = getattr(torch.ops.lowbit_attn, entry)(x, x, x, docs, _op.register_plan(plan), 0)
    every = [t for t in (out, lse, *state) if t.numel()]
    held = {t.untyped_storage().data_ptr() for t in every}
    assert len(held) == len(every) and not held & {t.untyped_storage().data_ptr() for t in (x, *docs)}


FORMS = ["batched", "fp4", "seqused", "token", "packed", "maps", "aligned", "ragged", "padded"]


def _form(form):
    """(function, (q, k, v, do), keyword arguments) of one call per form of the saved state."""
    import flamia_blackwell_attention_b200 as F
    s, d = 250 if form == "ragged" else 256, 80 if form == "padded" else 128
    x, kw = [t.cuda() for t in attention_inputs(2, s, 2, 2, d, seed=19)], dict(causal=True)
    cu = torch.tensor([0, 128, 512], dtype=torch.int32, device="cuda")
    if form in ("packed", "aligned", "maps"):
        x = [t.flatten(0, 1) for t in x]
        kw.update(dict(doc_maps=F.DocMaps.from_cu_seqlens(cu.cpu()).to("cuda")) if form == "maps" else
                  dict(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=384, max_seqlen_k=384))
    if form == "aligned":
        kw.update(seqused_q=(su := torch.tensor([100, 384], dtype=torch.int32, device="cuda")), seqused_k=su)
    if form == "seqused":
        kw.update(seqused_k=torch.tensor([256, 100], dtype=torch.int32, device="cuda"))
    if form == "token":
        kw.update(options=F.FP8AttnOptions(operand_scaling="token_local", ds_dq_rowlocal="all"))
    else:
        kw.update(deterministic=True)
    return (F.flash_attn_fp4 if form == "fp4" else F.flash_attn_fp8), x, kw


def _same(got, want, form):
    for i, (a, b) in enumerate(zip(got, want)):
        # (without deterministic=True the two key tiles' f16 partial sums of dQ may be added in either order: two roundings of 2^-11)
        assert torch.equal(a, b) or (form == "token" and i == 1 and (a - b).float().norm() <= 2 ** -10 * b.float().norm())


@pytest.mark.parametrize("form", FORMS)
def test_saved_tensors_have_a_storage_each_and_can_be_moved(form):
    fn, x, kw = _form(form)
    q, k, v = (t.detach().requires_grad_(True) for t in x[:3])
    out = fn(q, k, v, **kw)
    want = (out.detach(), *torch.autograd.grad(out, (q, k, v), x[3]))
    held = []

    def pack(t):
        held.append(t.untyped_storage().data_ptr())
        return t.cpu()
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        out = fn(q, k, v, **kw)
    assert len(set(held)) == len(held) >= 4
    _same((out.detach(), *torch.autograd.grad(out, (q, k, v), x[3])), want, form)


@pytest.mark.parametrize("form", ["batched", "packed"])
def test_saved_tensors_left_on_the_host_are_refused(form):
    fn, x, kw = _form(form)
    q, k, v = (t.detach().requires_grad_(True) for t in x[:3])
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t):
        out = fn(q, k, v, **kw)
    with pytest.raises(RuntimeError, match="on dout's device"):
        torch.autograd.grad(out, (q, k, v), x[3])


@pytest.mark.parametrize("form", FORMS)
def test_mode_around_either_pass_sees_the_op(form):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))
    fn, x, kw = _form(form)
    q, k, v = (t.detach().requires_grad_(True) for t in x[:3])
    name, runs = f"lowbit_attn.{'fp4' if form == 'fp4' else 'fp8'}", []
    for around in ((), ("fwd",), ("bwd",), ("fwd", "bwd")):
        seen = []
        with Mode() if "fwd" in around else torch.enable_grad():
            out = fn(q, k, v, **kw)
        with Mode() if "bwd" in around else torch.enable_grad():
            runs.append((out.detach(), *torch.autograd.grad(out, (q, k, v), x[3])))
        assert (f"{name}.default" in seen) == ("fwd" in around) and (f"{name}_bwd.default" in seen) == ("bwd" in around)
        _same(runs[-1], runs[0], form)
