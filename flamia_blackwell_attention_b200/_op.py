"""The attention call as registered torch ops, so that selective activation checkpointing can save it and torch.compile
can trace it. Same op names and schemas as the reference's flash_attn/cute/lowprec/_op.py (:12-16, 428-476):

    lowbit_attn::fp8(Tensor q, Tensor k, Tensor v, Tensor[] docs, int plan, int docs_id) -> (Tensor, Tensor, Tensor[])
    lowbit_attn::fp8_bwd(Tensor dout, Tensor[] state, int entry) -> (Tensor, Tensor, Tensor)          (and ::fp4)

`plan` is a process-local integer handle into an append-only registry of resolved plans; `docs` carries the varlen
tensors (cu_seqlens_q, cu_seqlens_k[, seqused_q, seqused_k]). The saved state is codes + factor tables + O + LSE, not the
bf16 inputs. LSE and the state are non-differentiable; gradients are not materialised for unused outputs.

This module holds the schemas, the fake (meta) implementations and the plan registry; the CUDA and autograd
implementations are native (csrc/host.cpp) and registered when that module is loaded (_lib.host()).
"""
from __future__ import annotations

import threading

import torch

from . import _lib as L
from . import _routes

_REG_LOCK = threading.Lock()
_PLANS: list = []          # handle -> AttnPlan (the native registry holds the same plans at the same handles)
_PLAN_HANDLES: dict = {}   # AttnPlan (by value: plans are frozen) -> handle


def _plan_facts(plan) -> dict:
    """The numbers of a plan that the native launches need (csrc/host.cpp::Plan)."""
    sh, f, bw = plan.shape, plan.fwd, plan.bwd
    win = f.window or (None, None)
    return dict(fp4=plan.entry == "fp4", token_local=f.operand_scaling == "token_local", hadamard=f.qk_hadamard, causal=f.causal,
                need_bwd=bw.kernel != "none", p_group=f.p_hat_frame == "group", seqused_k=f.seqused_k, varlen=sh.varlen,
                aligned=sh.aligned_varlen, ragged=f.ragged_documents, return_lse=f.return_lse, deterministic=bw.deterministic,
                rowlocal=bw.ds_dq_rowlocal == "all", prescale={"row": 0, "causal_tile": 1, "causal_row": 2}[bw.dq_prescale],
                window_left_p1=L.window_p1(win[0]), window_right_p1=L.window_p1(win[1]),
                softcap=f.softcap, softmax_scale=plan.softmax_scale, b=sh.b, s_q=sh.s_q, s_k=sh.s_k, h=sh.h, h_kv=sh.h_kv, d=sh.d,
                tot_q=sh.tot_q, d_call=plan.pad_from or sh.d)


def register_plan(plan) -> int:
    """Handle of a plan. Equal plans share one handle, so the registry grows with the number of DISTINCT plans a
    process resolves, not with the number of calls or of cache evictions."""
    with _REG_LOCK:
        h = _PLAN_HANDLES.get(plan)
        if h is None:
            h = L.host().register_plan(_plan_facts(plan))
            assert h == len(_PLANS)
            _PLANS.append(plan)
            _PLAN_HANDLES[plan] = h
        return h


def _register_entry(plan_id, docs_meta) -> int:
    """Backward entry handle of (plan handle, docs meta = (capacity, aligned) or None)."""
    return L.host().register_entry(plan_id, *((-1, False) if docs_meta is None else docs_meta))


def _fake_fwd(q, k, v, docs, plan, docs_id):
    p = _PLANS[plan]
    sh = p.shape
    is_docs = sh.varlen or p.fwd.ragged_documents
    if sh.aligned_varlen or (is_docs and sh.varlen and p.fwd.return_lse):
        lse_shape = (sh.h, sh.tot_q)
    elif is_docs and not p.fwd.return_lse:
        lse_shape = (0,)
    else:
        lse_shape = (sh.b, sh.h, sh.s_q)
    n_docs = int(docs[0].shape[0]) - 1 if (len(docs) > 0 and not p.fwd.seqused_k) else 0
    spec = _routes.state_spec(p, n_docs, q.dtype, capacity=int(docs[3].numel()) if len(docs) == 6 else None)
    # O / LSE leave as the op's outputs; repacked documents keep the aligned buffer's LSE in the state
    state = [q.new_empty(shape, dtype=dt) for shape, dt in (spec[1:] if (is_docs and not sh.aligned_varlen) else spec[2:])]
    state.append(torch.empty((), dtype=torch.int64))
    return torch.empty_like(q), q.new_empty(lse_shape, dtype=torch.float32), state


def _fake_bwd(dout, state, entry):
    sh, d = _PLANS[L.host().entry(entry)[0]].shape, dout.shape[-1]
    kshape = (sh.tot_k, sh.h_kv, d) if sh.varlen else (sh.b, sh.s_k, sh.h_kv, d)
    return torch.empty_like(dout), dout.new_empty(kshape), dout.new_empty(kshape)


def _define(entry: str):
    name = f"lowbit_attn::{entry}"
    torch.library.define(name, "(Tensor q, Tensor k, Tensor v, Tensor[] docs, int plan, int docs_id) -> "
                               "(Tensor, Tensor, Tensor[])")
    torch.library.define(name + "_bwd", "(Tensor dout, Tensor[] state, int entry) -> (Tensor, Tensor, Tensor)")
    torch.library.register_fake(name)(_fake_fwd)
    torch.library.register_fake(name + "_bwd")(_fake_bwd)


for _e in ("fp8", "fp4"):
    _define(_e)


def op_apply(entry, handle, q, k, v, docs_tensors):
    """Runs the registered op of the entry on a registered plan; returns (out, lse)."""
    # (the native call goes to the dispatcher directly: traced programs, __torch_function__ subclasses and modes need the op itself)
    if torch.compiler.is_compiling() or torch.overrides.has_torch_function((q, k, v)):
        out, lse, _state = getattr(torch.ops.lowbit_attn, entry)(q, k, v, list(docs_tensors), handle, 0)
        return out, lse
    return L.host().run(entry == "fp4", handle, q, k, v, docs_tensors)
