"""Public entry points flash_attn_fp8 / flash_attn_fp4: same signatures, defaults, return values and refusal convention
as the reference's flash_attn/cute/lowprec/api.py (flash_attn_fp4 :169, flash_attn_fp8 :270). Each call resolves one
immutable plan (cached per argument values and tensor metadata) before anything is quantised or launched, then runs the
registered op lowbit_attn::fp8 / ::fp4, whose autograd node carries the plan handle to the backward.
"""
from __future__ import annotations

import threading
import warnings
from dataclasses import dataclass
from typing import Callable, Optional, Tuple

import torch

from . import _lib as L
from . import _op
from . import interface_bwd_fp4 as _switches
from .options import FP4AttnOptions, FP8AttnOptions
from .plan import AttnPlan, _fail, resolve_fp4, resolve_fp8

__all__ = ["flash_attn_fp4", "flash_attn_fp8"]

_REPACK_WARNED = False
REPACK_WARNING = (
    "flash_attn_{entry} got cu_seqlens_q / cu_seqlens_k without seqused_q / seqused_k. No tensor is copied (the kernels "
    "read and write the packed rows in place), but the document tables are rebuilt on the device on every call (one small "
    "launch before the quantiser) and the intermediates take a padded buffer of up to 127 extra rows per document. Build the tables "
    "once with DocMaps.from_cu_seqlens(...) and pass doc_maps=, or lay the documents out at starts that are multiples of "
    "128 and pass the true lengths as seqused_q / seqused_k. (Warned once.)")


@dataclass(frozen=True)
class _Resolved:
    """A resolved plan as the call path uses it."""
    plan: AttnPlan
    handle: int          # of the native plan registry
    plain: bool          # batched, whole tiles, no seqused_k: nothing to check or to convert per call


# Call key -> _Resolved. A plan is a pure function of the argument values and of the tensors' metadata, which is what the key
# holds (a flat tuple: building and hashing frozen dataclasses of the same facts was 40 us of every call). Bounded: the oldest
# entry goes first; a refusal raises and is not remembered.
_CALLS: dict = {}
_CALLS_MAX = 1024
_CALLS_LOCK = threading.Lock()


def _facts(t):
    """What plan resolution may look at in a tensor argument: nothing but metadata."""
    return t.shape, t.dtype, t.requires_grad


def _stand_in(t):
    if not isinstance(t, torch.Tensor):
        return t
    return torch.empty(t.shape, dtype=t.dtype, device="meta", requires_grad=t.requires_grad and t.dtype.is_floating_point)


def _resolve(entry, resolve, q, k, v, kw) -> _Resolved:
    if all(isinstance(t, torch.Tensor) for t in (q, k, v)):     # (otherwise the resolver words the refusal)
        q, k, v = _stand_in(q), _stand_in(k), _stand_in(v)
        kw = {n: _stand_in(x) for n, x in kw.items()}
    plan = resolve(q, k, v, **kw)
    plain = not (plan.shape.varlen or plan.fwd.ragged_documents or plan.fwd.seqused_k)
    return _Resolved(plan, _op.register_plan(plan), plain)


def _resolved(entry, resolve, names, q, k, v, *values) -> _Resolved:
    """The resolved plan of a call; names / values: its keyword arguments in the resolver's names."""
    try:
        # (entry, mode, the module switches the resolver reads, tensor metadata, argument values)
        key = None if torch.compiler.is_compiling() else \
            L.host().call_key(q, k, v, entry, _switches.DQ_CAUSAL_PRESCALE, _switches.DQ_CAUSAL_GRANULARITY, *values)
        if key is None:
            key = (entry, torch.is_grad_enabled(), _switches.DQ_CAUSAL_PRESCALE, _switches.DQ_CAUSAL_GRANULARITY,
                   q.shape, q.dtype, q.requires_grad, k.shape, k.dtype, k.requires_grad, v.shape, v.dtype, v.requires_grad,
                   *[x if not isinstance(x, torch.Tensor) else _facts(x) for x in values])
        hit = _CALLS.get(key)
    except (AttributeError, TypeError):         # not tensors, or an unhashable argument (e.g. a callable object): uncached
        return _resolve(entry, resolve, q, k, v, dict(zip(names, values)))
    if hit is None:
        hit = _resolve(entry, resolve, q, k, v, dict(zip(names, values)))
        with _CALLS_LOCK:
            while len(_CALLS) >= _CALLS_MAX:
                del _CALLS[next(iter(_CALLS))]
            _CALLS[key] = hit
    return hit


def _doc_maps_args(maps, q, cu_q, cu_k, su_q, su_k):
    """doc_maps= stands for the varlen arguments: the plan is resolved as for cu_seqlens = maps.cu."""
    from .docmaps import DocMaps
    if not isinstance(maps, DocMaps):
        _fail("B9", TypeError, f"doc_maps must be a DocMaps; got {type(maps).__name__}")
    if cu_q is not None or cu_k is not None or su_q is not None or su_k is not None:
        _fail("B9", ValueError, "doc_maps carries the documents: do not pass cu_seqlens_* / seqused_* with it")
    if isinstance(q, torch.Tensor) and (q.dim() != 3 or q.shape[0] != maps.total):
        _fail("B9", ValueError, f"doc_maps describes {maps.total} packed rows; q is {tuple(q.shape)}")
    if isinstance(q, torch.Tensor) and q.is_cuda and maps.device != q.device:
        _fail("B9", ValueError, f"doc_maps is on {maps.device}, q on {q.device}: move the maps with .to(device)")
    return maps.cu, maps.cu, maps.max_seqlen, maps.max_seqlen


def _run(call, q, k, v, cu_q, cu_k, su_q, su_k, return_lse, doc_maps=None):
    global _REPACK_WARNED
    plan = call.plan
    if not q.is_cuda:
        raise RuntimeError(f"flash_attn_{plan.entry}: q, k, v must be CUDA tensors (this library has no CPU path)")
    if call.plain:
        out, lse = _op.op_apply(plan.entry, call.handle, q, k, v, ())
        return (out, lse) if return_lse else out
    sh = plan.shape
    if sh.varlen and sh.tot_q != sh.tot_k:
        _fail("B8", NotImplementedError, "packed documents are self-attention documents here: q and k must share "
                                         "cu_seqlens (total_q == total_k)")
    if sh.varlen:
        # the kernels walk ONE document table (built from cu_seqlens_q / seqused_q): the key side must be the same
        # tensor, otherwise a call with different key documents would silently run as self-attention over q's table
        for a, b_, name in ((cu_q, cu_k, "cu_seqlens"), (su_q, su_k, "seqused")):
            if a is None or b_ is None or a is b_:
                continue
            if tuple(a.shape) != tuple(b_.shape) or a.data_ptr() != b_.data_ptr():
                _fail("B8", NotImplementedError, f"packed documents are self-attention documents here: pass the SAME tensor "
                                                 f"as {name}_q and {name}_k (distinct query / key tables are not built)")
    if plan.fwd.ragged_documents and sh.s_q != sh.s_k:
        _fail("B8", NotImplementedError, "lengths that are no multiple of 128 are built for self-attention: s_q must equal s_k; "
                                         f"got {sh.s_q} and {sh.s_k}")
    if sh.varlen and not sh.aligned_varlen and doc_maps is None and not _REPACK_WARNED:
        _REPACK_WARNED = True
        warnings.warn(REPACK_WARNING.format(entry=plan.entry), UserWarning, stacklevel=3)
    if doc_maps is not None:
        docs = tuple(doc_maps.tensors())    # cu, start, len, row_map, slot_src, slot_rows: per call only the work lists are made
    else:
        docs = tuple(t for t in (cu_q, cu_k, su_q, su_k) if t is not None) if sh.varlen else \
            ((su_k.contiguous(),) if plan.fwd.seqused_k else ())
    out, lse = _op.op_apply(plan.entry, call.handle, q, k, v, docs)
    return (out, lse) if return_lse else out


def _is_e4m3(t):
    return isinstance(t, torch.Tensor) and t.dtype is torch.float8_e4m3fn


_COMMON_NAMES = ("softmax_scale", "causal", "window_size", "softcap", "score_mod", "score_mod_bwd", "mask_mod", "cu_seqlens_q",
                 "cu_seqlens_k", "max_seqlen_q", "max_seqlen_k", "seqused_k", "seqused_q", "deterministic", "return_lse")
_FP8_NAMES = _COMMON_NAMES + ("qk_hadamard", "q_quantized", "k_quantized", "q_scale_fused", "options")
_FP4_NAMES = _COMMON_NAMES + ("pv_precision", "backward", "causal_safety", "qk_hadamard", "options")


def flash_attn_fp8(q, k, v, *, softmax_scale: Optional[float] = None, causal: bool = False,
                   window_size: Tuple[Optional[int], Optional[int]] = (None, None), softcap: float = 0.0,
                   score_mod: Optional[Callable] = None, score_mod_bwd: Optional[Callable] = None,
                   mask_mod: Optional[Callable] = None, aux_tensors: Optional[tuple] = None,
                   cu_seqlens_q=None, cu_seqlens_k=None, max_seqlen_q: Optional[int] = None,
                   max_seqlen_k: Optional[int] = None, seqused_k=None, seqused_q=None, deterministic: bool = False,
                   return_lse: bool = False, qk_hadamard: Optional[bool] = None, q_quantized=None, k_quantized=None,
                   q_scale_fused: bool = False, options: Optional[FP8AttnOptions] = None, q_descale=None, k_descale=None,
                   v_descale=None, grad_proxies=None, doc_maps=None):
    """8-bit (MXFP8) attention, forward and backward, on B200.

    q: (b, s, h, d); k, v: (b, s, h_kv, d); bf16 or f16; h % h_kv == 0; d in {64, 128}, or another multiple of 16 below
    128 (run padded with zero columns to the next of 64 / 128). Packed (total, h, d) with
    cu_seqlens_q / cu_seqlens_k (repacked), or with seqused_q / seqused_k as well (aligned, zero-copy: starts multiples of
    128). Returns out (dtype and shape of q); with return_lse=True (out, lse) with lse (b, h, s) float32 in nats,
    non-differentiable ((h, total_q) in the caller's row order on the packed forms). causal is bottom-right aligned.
    E4M3 Q, K, V, dO with one UE8M0 exponent per 32 tokens x the whole head dim; qk_hadamard=None turns the random-sign
    Hadamard rotation of Q / K on at d = 128. Every unserved combination raises with a `.rule` before any launch."""
    if doc_maps is not None:
        cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k = _doc_maps_args(doc_maps, q, cu_seqlens_q, cu_seqlens_k,
                                                                                seqused_q, seqused_k)
    if aux_tensors is not None:
        _fail("B3", NotImplementedError, "aux_tensors belong to score_mod / mask_mod, which this library does not take")
    if q_descale is not None or k_descale is not None or v_descale is not None or grad_proxies is not None or \
            _is_e4m3(q):
        if doc_maps is not None:
            _fail("B7", NotImplementedError, "pre-quantised E4M3 inputs are served on the batched form, not with doc_maps")
        from .prequant_fa3 import flash_attn_fp8_prequant
        return flash_attn_fp8_prequant(resolve_fp8, q, k, v, q_descale, k_descale, v_descale, grad_proxies, dict(
            softmax_scale=softmax_scale, causal=causal, window_size=tuple(window_size), softcap=softcap,
            score_mod=score_mod, score_mod_bwd=score_mod_bwd, mask_mod=mask_mod, cu_seqlens_q=cu_seqlens_q,
            cu_seqlens_k=cu_seqlens_k, max_seqlen_q=max_seqlen_q, max_seqlen_k=max_seqlen_k, seqused_k=seqused_k,
            seqused_q=seqused_q, deterministic=deterministic, return_lse=return_lse, qk_hadamard=qk_hadamard,
            q_quantized=q_quantized, k_quantized=k_quantized, q_scale_fused=q_scale_fused, options=options), return_lse)
    call = _resolved("fp8", resolve_fp8, _FP8_NAMES, q, k, v, softmax_scale, causal, tuple(window_size), softcap, score_mod,
                     score_mod_bwd, mask_mod, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, seqused_k, seqused_q,
                     deterministic, return_lse, qk_hadamard, q_quantized, k_quantized, q_scale_fused, options)
    return _run(call, q, k, v, cu_seqlens_q, cu_seqlens_k, seqused_q, seqused_k, return_lse, doc_maps)


def flash_attn_fp4(q, k, v, *, softmax_scale: Optional[float] = None, causal: bool = False,
                   window_size: Tuple[Optional[int], Optional[int]] = (None, None), softcap: float = 0.0,
                   score_mod: Optional[Callable] = None, score_mod_bwd: Optional[Callable] = None,
                   mask_mod: Optional[Callable] = None, aux_tensors: Optional[tuple] = None,
                   cu_seqlens_q=None, cu_seqlens_k=None, max_seqlen_q: Optional[int] = None,
                   max_seqlen_k: Optional[int] = None, seqused_k=None, seqused_q=None, deterministic: bool = False,
                   return_lse: bool = False, pv_precision: str = "fp8", backward: str = "e4m3",
                   causal_safety: str = "auto", qk_hadamard: Optional[bool] = None,
                   options: Optional[FP4AttnOptions] = None, q_descale=None, k_descale=None, v_descale=None,
                   doc_maps=None):
    """Mixed NVFP4 / FP8 attention, forward and backward, on B200: Q.K^T and its recomputation in the backward on NVFP4
    codes (E2M1, one E4M3 scale per 16 along d); P.V, dP, dV, dK, dQ on E4M3 token blocks. Arguments, shapes and returns
    as flash_attn_fp8; d = 128. With qk_hadamard on (default) the NVFP4 codes are of the rotated rows, the E4M3 copies of
    the rows as given."""
    if doc_maps is not None:
        cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k = _doc_maps_args(doc_maps, q, cu_seqlens_q, cu_seqlens_k,
                                                                                seqused_q, seqused_k)
    if q_descale is not None or k_descale is not None or v_descale is not None or \
            _is_e4m3(q) or _is_e4m3(k) or _is_e4m3(v):
        _fail("B7", TypeError, "flash_attn_fp4 takes bf16 / f16 inputs: pre-quantised E4M3 inputs are a flash_attn_fp8 "
                               "feature of the reference and are not built here")
    if aux_tensors is not None:
        _fail("B3", NotImplementedError, "aux_tensors belong to score_mod / mask_mod, which this library does not take")
    call = _resolved("fp4", resolve_fp4, _FP4_NAMES, q, k, v, softmax_scale, causal, tuple(window_size), softcap, score_mod,
                     score_mod_bwd, mask_mod, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, seqused_k, seqused_q,
                     deterministic, return_lse, pv_precision, backward, causal_safety, qk_hadamard, options)
    return _run(call, q, k, v, cu_seqlens_q, cu_seqlens_k, seqused_q, seqused_k, return_lse, doc_maps)
