"""What surrounds the native call path (csrc/host.cpp): the backward's kernel scalars, the device status word, the document
tables on host tensors, the saved state's specification, and the body of calls on pre-quantised operands (which runs no
quantiser; mirrors the reference's flash_attn/cute/lowprec/_routes.py and prequant_fa3.py).
"""
from __future__ import annotations

import torch

from . import _lib as L
from . import kernels as K

P_SHIFT_LOG2 = 8.0     # the backward recomputes P' = 2^8 P (its E4M3 P-hat then uses the normal range)


def backward_scalars(softmax_scale, dq_boost=1.0):
    """The eight kernel scalars of the reference's 8-bit backward (flash_attn/cute/device_scales.py:734-743, slots 0-7)
    as this library uses them. Block-scaled operands carry their scales with the codes, so every operand descale is 1
    and the scalars are constants: [0] softmax scale of S, [1] dP-sum scale, [2] dS boost 2^-8 (with P' = 2^8 P), [3] dV
    scale 2^-8 (folded into the dV epilogue), [4] dK scale (the dK epilogue), [5] the f16 dQ pre-scale (per query tile on
    the device: fl_dq_prescale; `dq_boost` stands for it here), [6] the D fold multiplier -2^-8 (applied by the dO
    quantiser launch), [7] the dQ postprocess scale softmax_scale / pre-scale."""
    import numpy as np
    f = np.float32
    p_shift = f(2.0 ** P_SHIFT_LOG2)
    sm = f(softmax_scale)
    return (sm, f(1.0), f(1.0) / p_shift, f(1.0) / p_shift, sm, f(dq_boost), -(f(1.0) / p_shift), sm / f(dq_boost))


# --------------------------------------------------------------------------------------------------------------- status
# Every device-side wait of the kernels is bounded; one that runs out writes 0x100 | site into the call's status word and
# the kernel drains, leaving its outputs partly written. Reading the word costs a host synchronisation, so the hot path
# never does it: the device's last word is remembered (natively) for check_status(), and the environment variable
# FLAMIA_B200_CHECK_STATUS=1 makes every forward and backward check it (a debugging mode).
def _device_index(device):
    idx = torch.cuda.current_device() if device is None else torch.device(device).index
    return torch.cuda.current_device() if idx is None else idx


def _status_word(device):
    """The device's status word: one persistent int32 per device, zeroed when it is made and again by check_status()
    after it reported a code (kernels only ever write it when something went wrong), so a call launches no fill kernel.
    A first call made inside a stream capture gets a word of the capture's own."""
    return L.host().status_word(_device_index(device))


def _note_status(status):
    L.host().note_status(status)


def check_status(device=None) -> int:
    """Synchronises `device` (default: the current one) and raises RuntimeError if a flash_attn_fp8 / flash_attn_fp4 call
    there (forward or backward) since the last check gave up a device-side wait or met a bad document table; returns 0
    otherwise. The word is cleared when a code has been reported."""
    return L.host().check_status(_device_index(device))


# --------------------------------------------------------------------------------------------------------------- docs
class Docs:
    """Packed documents laid out at 128-aligned starts of one padded buffer. Built on the device without a host sync:
    the padded capacity is the host-known bound total + 127 * n_docs rounded up to 128. The quantisers read the packed
    rows in place through the slot tables (slot_src / slot_rows: first source row and number of real rows of every
    128-row slot of the buffer); outputs are scattered back through row_map."""

    def __init__(self, cu, lens, total, aligned, capacity=None):
        dev = cu.device
        self.n = int(lens.numel())
        self.len = lens.to(torch.int32).contiguous()
        self.aligned = aligned
        self.slot_src = self.slot_rows = None
        if aligned:
            self.start = cu[:-1].to(torch.int32).contiguous()
            self.capacity = int(total)
            self.row_map = None
            return
        padded = ((self.len + 127) // 128) * 128
        ends = torch.cumsum(padded, 0)
        self.start = (ends - padded).to(torch.int32).contiguous()
        self.capacity = int(capacity) if capacity is not None else ((int(total) + 127 * self.n + 127) // 128) * 128
        rows = torch.arange(self.capacity, device=dev, dtype=torch.int32)
        doc = torch.searchsorted(ends.to(torch.int32), rows, right=True).clamp_(max=self.n - 1)
        off = rows - self.start[doc]
        src = cu[:-1].to(torch.int32)[doc] + off
        live = (off >= 0) & (off < self.len[doc])
        self.row_map = torch.where(live, src, torch.full_like(src, -1)).contiguous()
        first = slice(0, self.capacity, 128)
        self.slot_src = self.row_map[first].contiguous()                     # a slot's first row is real or the slot is empty
        self.slot_rows = torch.where(live[first], (self.len[doc] - off)[first].clamp(max=128),
                                     torch.zeros_like(off[first])).to(torch.int32).contiguous()


def state_spec(plan, n_docs=0, dtype=torch.bfloat16, capacity=None):
    """Shapes and dtypes of the tensors forward() returns as `state`, in order, from the plan alone (n_docs = number of
    documents of a packed call). The fake implementations of the registered ops are built from this, and a GPU test
    checks it against the real state."""
    sh, f = plan.shape, plan.fwd
    fp4 = plan.entry == "fp4"
    tl = f.operand_scaling == "token_local"
    need_bwd = plan.bwd.kernel != "none"
    f8, u8, f32, i32 = torch.float8_e4m3fn, torch.uint8, torch.float32, torch.int32
    docs = sh.varlen
    if docs:
        n, cap = n_docs, sh.tot_q
        if not sh.aligned_varlen:
            cap = capacity if capacity is not None else ((sh.tot_q + 127 * n + 127) // 128) * 128
        b, s_q, s_k = 1, cap, cap
    else:                                   # batch rows of whole tiles
        b, s_q, s_k = sh.b, (sh.s_q + 127) // 128 * 128, (sh.s_k + 127) // 128 * 128
    h, hk, d = sh.h, sh.h_kv, sh.d
    o_rows = sh.tot_q if docs else sh.s_q   # (the caller's)
    spec = [((b, o_rows, h, plan.pad_from or d), dtype), ((b, h, s_q), f32),                   # O, LSE of the kernels
            ((b, s_q, h, d), f8), ((b, h, s_q // 32), f32), ((b, s_k, hk, d), f8), ((b, hk, s_k // 32), f32),
            ((b, s_k, hk, d), f8), ((b, hk, s_k // 32), f32), ((1,), i32)]                     # codes, factors, status
    if need_bwd:      # K / V statistics of the f16 dQ pre-scale: per 128-row tile and head, or per token
        spec += [((b, s_k), f32)] * 2 if plan.bwd.dq_prescale == "causal_row" else [((b, hk, s_k // 128, 2), f32)] * 2
    if fp4:
        spec += [((b, s_q, h, d // 2), u8), ((b, h, s_q // 128, d // 64, 32, 4, 4), u8),
                 ((b, s_k, hk, d // 2), u8), ((b, hk, s_k // 128, d // 64, 32, 4, 4), u8)]
    if tl:
        spec += [((b, h, s_q), f32), ((b, hk, s_k), f32), ((b, hk, s_k), f32)]
    if f.seqused_k:
        spec += [((b,), i32)]
    if docs:
        spec += [((n,), i32), ((n,), i32)] + ([] if sh.aligned_varlen else [((cap,), i32), ((cap // 128,), i32), ((cap // 128,), i32)])
        spec += [((4 + 9 * (cap // 128),), i32)]                  # the kernels' work lists
    return spec


# --------------------------------------------------------------------------------------------------------------- forward
def forward_prequant(plan, q8, k8, v8, descales, seqused_k):
    """Forward on operands that are already E4M3 codes with one float descale per (batch row, kv head): no quantiser runs; the
    descales fill the factor tables, and V's mantissa goes on the output rows. Returns (out, lse, state): state = the tensors
    backward_prequant() needs."""
    from .prequant_fa3 import mantissa
    sh, f = plan.shape, plan.fwd
    qd, kd, vd = descales
    grp = sh.h // sh.h_kv
    need_bwd = plan.bwd.kernel != "none"
    status = _status_word(q8.device)

    def table(dsc, heads_rep, s):
        return dsc.repeat_interleave(heads_rep, dim=1)[:, :, None].expand(sh.b, dsc.shape[1] * heads_rep, s // 32).contiguous()
    qq = dict(codes=q8, fac=table(qd, grp, sh.s_q))
    kq = dict(codes=k8, fac=table(kd, 1, sh.s_k))
    vq = dict(codes=v8, fac=table(vd, 1, sh.s_k))
    out, lse, _ = K.attn_fwd(qq, kq, vq, causal=f.causal, softmax_scale=plan.softmax_scale,
                             out_dtype=torch.float16 if sh.dtype == "float16" else torch.bfloat16, status=status,
                             window=f.window, seqused_k=seqused_k, softcap=f.softcap, o_mult=mantissa(vd))
    state = [out, lse, q8, qq["fac"], k8, kq["fac"], v8, vq["fac"], status]
    if need_bwd:
        state += [K.code_stats(k8, kd), K.code_stats(v8, vd)]
    if seqused_k is not None:
        state += [seqused_k]
    state += [qd, kd]
    _note_status(status)
    return out, lse, state


def backward_prequant(plan, state, dout):
    """dq, dk, dv of a forward_prequant() call. Float descales: the mantissas the block-scaled dK / dQ products left out are
    multiplied in afterwards."""
    from ._op import register_plan
    from .prequant_fa3 import mantissa
    *state, qd, kd = state
    dq_mult = mantissa(kd).repeat_interleave(plan.shape.h // plan.shape.h_kv, dim=1).contiguous()
    return L.host().backward(register_plan(plan), dout, state, mantissa(qd), dq_mult)
