"""Performance cases of the attention calls: what a training or serving program asks of flash_attn_fp8 and flash_attn_fp4,
through those two entry points alone.

    listed()             the named cases        draw(rng)        one more case of the same ranges
    prepare(case, seed)  a program's tensors    run(state)       one pass through the public call
    work(case)           bytes and operations   tolerance(case)  how far correct results may lie apart

A case is a dict of plain values:
    entry      "fp8" (MXFP8) | "fp4" (NVFP4 scores, E4M3 elsewhere)
    pass       "step" (forward and backward, as in training) | "forward" (no gradients, as in serving)
    form       "batch" (b, s, h, d) | "packed" (documents back to back, cu_seqlens) | "maps" (the same with a DocMaps)
    b, sq, sk, h, hk, d, dtype, causal      the call's sizes; packed forms: sq = sk = total tokens, b = 1
    window     left side of a sliding window, 0 = none          softcap    score cap, 0.0 = none
    scaling    "block" (one scale per 32 tokens) | "token" (per-token scales, row-local dS, causal dQ pre-scale)
    ordered    deterministic dQ          lse    return_lse         used    batch rows with seqused_k valid keys
    doc_lo, doc_hi, doc_seed             packed forms: document lengths, log-uniform in [doc_lo, doc_hi]
"""
import math
import random

import numpy as np
import torch

import flamia_blackwell_attention_b200 as F
import flamia_blackwell_attention_b200.interface_bwd_fp4 as switches

_PLAIN = {"entry": "fp8", "pass": "step", "form": "batch", "b": 1, "sq": 128, "sk": 128, "h": 1, "hk": 1, "d": 128,
          "dtype": "bfloat16", "causal": True, "window": 0, "softcap": 0.0, "scaling": "block", "ordered": False,
          "lse": False, "used": False, "doc_lo": 0, "doc_hi": 0, "doc_seed": 0}


def _case(**kw):
    return dict(_PLAIN, **kw)


def listed():
    return [
        # a training step of a small model: every launch and every line of host code shows
        _case(name="step small d64", b=1, sq=512, sk=512, h=4, hk=4, d=64),
        # serving: one short prompt through a grouped-query layer on the mixed route
        _case(name="forward short prompt fp4", entry="fp4", **{"pass": "forward"}, b=1, sq=256, sk=256, h=16, hk=4),
        # training of a model of several billion parameters at 4k context, both routes: the benchmark's own cell
        _case(name="step 4k fp8", b=4, sq=4096, sk=4096, h=16, hk=16),
        _case(name="step 4k fp4", entry="fp4", b=4, sq=4096, sk=4096, h=16, hk=16),
        # an encoder's or a diffusion model's inference: bidirectional, no gradients
        _case(name="forward dense 4k fp8", **{"pass": "forward"}, b=4, sq=4096, sk=4096, h=16, hk=16, causal=False),
        # grouped-query training at 8k with every option that keeps a causal model free of leaks through the scales
        _case(name="step gqa 8k token scales", b=2, sq=8192, sk=8192, h=32, hk=8, scaling="token"),
        # pre-training on documents packed back to back: 16384 tokens, lengths from 128 to 8192
        _case(name="step packed 16k fp8", form="packed", sq=16384, sk=16384, h=16, hk=16, doc_lo=128, doc_hi=8192),
        # fine-tuning on many short samples, the document tables built once in the data loader
        _case(name="step packed maps fp4", entry="fp4", form="maps", sq=6000, sk=6000, h=16, hk=4, doc_lo=16, doc_hi=1024,
              doc_seed=3),
        # a vision encoder in float16: 1000 tokens (no multiple of any tile), head dim 64, bidirectional
        _case(name="step ragged 1000 f16 d64", b=8, sq=1000, sk=1000, h=12, hk=12, d=64, dtype="float16", causal=False),
        # a sliding-window layer with a head dim between the kernels' own
        _case(name="step window 512 d96", b=2, sq=2048, sk=2048, h=16, hk=4, d=96, window=512),
        # long-context training
        _case(name="step 32k fp8", b=1, sq=32768, sk=32768, h=16, hk=16),
        # chunked prefill: 512 new tokens of each of 4 requests against 8192 cached ones, LSE kept for merging
        _case(name="forward chunk of prefill", **{"pass": "forward"}, b=4, sq=512, sk=8192, h=32, hk=8, lse=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng):
    hk = rng.choice((1, 2, 3, 4, 5, 8, 12, 16))
    return hk * rng.choice((1, 1, 2, 4, 7) if hk <= 4 else (1, 1, 2, 4)), hk


def draw(rng):
    """Sizes over the logarithm of their ranges, head counts and options mixed; b fills a token budget drawn the same way."""
    while True:
        kind = rng.choice(("step", "step", "step", "forward", "forward", "packed", "maps", "chunk", "token"))
        h, hk = _heads(rng)
        c = _case(h=h, hk=hk, entry=rng.choice(("fp8", "fp8", "fp4")), causal=rng.random() < 0.7)
        if rng.random() < 0.25:
            c["dtype"] = "float16"
        c["pass"] = "forward" if kind in ("forward", "chunk") or (kind in ("packed", "maps") and rng.random() < 0.3) else "step"
        budget = _log(rng, 1 << 16, 1 << 26)
        if kind == "token":
            c.update(entry="fp8", scaling="token", causal=True)
        if c["entry"] == "fp8" and kind != "token":
            c["d"] = rng.choice((128, 128, 128, 64, 64, 96, 80, 32))
        if kind in ("packed", "maps"):
            lo = _log(rng, 8, 512)
            n = max(lo + 1, min(65536, budget // (h * c["d"])))
            c.update(form=kind, b=1, sq=n, sk=n, doc_lo=lo, doc_hi=lo * rng.choice((2, 16, 64)), doc_seed=rng.randrange(1000))
        else:
            s = _log(rng, 128, 16384)
            whole = c["entry"] == "fp4" or kind in ("chunk", "token") or rng.random() < 0.5
            s = (s + 127) // 128 * 128 if whole else s
            c.update(sq=s, sk=s)
            if kind == "chunk":
                c.update(sk=s * rng.choice((2, 4, 8, 16)), causal=True, lse=rng.random() < 0.5)
            c["b"] = max(1, min(32, budget // (c["sk"] * h * c["d"])))
            extra = rng.random()
            if kind in ("step", "forward"):
                if extra < 0.15 and s > 256:
                    c["window"] = _log(rng, 64, s // 2)
                elif extra < 0.22:
                    c["softcap"] = rng.choice((20.0, 50.0))
                elif extra < 0.29 and s % 128 == 0:
                    c["used"] = True
                elif extra < 0.34 and kind == "step":
                    c["ordered"] = True
        # no drawn case may cost more than the largest listed one
        if work(c)["flops"] < 3e12 and c["b"] * (c["sq"] * h + 2 * c["sk"] * hk) * c["d"] < 1 << 28 and c["sk"] <= 65536:
            return c


# ------------------------------------------------------------------------------------------------------------ the inputs
def _documents(case):
    """Document lengths: log-uniform draws, the last one cut so that they fill the packed rows."""
    rng, left, out = random.Random(case["doc_seed"]), case["sq"], []
    while left > 0:
        out.append(min(left, _log(rng, case["doc_lo"], case["doc_hi"])))
        left -= out[-1]
    return out


def _used(case):
    """Valid keys of each batch row: from half the keys to all of them."""
    rng = random.Random(case["sk"])
    return [rng.randint(case["sk"] // 2, case["sk"]) for _ in range(case["b"])]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt, step = getattr(torch, case["dtype"]), case["pass"] == "step"

    def normal(rows, heads, outliers=False):
        lead = (case["b"], rows) if case["form"] == "batch" else (rows,)
        x = torch.randn(*lead, heads, case["d"], generator=gen, device="cuda", dtype=torch.float32)
        if outliers:       # one channel in a hundred twenty times as large, as in the activations such options are for
            n = heads * case["d"]
            sel = torch.randperm(n, generator=gen, device="cuda")[:max(1, n // 100)]
            x.view(-1, n)[:, sel] *= 20.0
        return x.to(dt)
    tok = case["scaling"] == "token"
    q, k, v = normal(case["sq"], case["h"], tok), normal(case["sk"], case["hk"], tok), normal(case["sk"], case["hk"])
    do = normal(case["sq"], case["h"]) if step else None
    kw = {"causal": case["causal"]}
    if case["window"]:
        kw["window_size"] = (case["window"], 0) if case["causal"] else (case["window"], case["window"])
    if case["softcap"]:
        kw["softcap"] = case["softcap"]
    if case["ordered"]:
        kw["deterministic"] = True
    if case["lse"]:
        kw["return_lse"] = True
    if case["used"]:
        kw["seqused_k"] = torch.tensor(_used(case), dtype=torch.int32, device="cuda")
    if tok:
        kw["options"] = F.FP8AttnOptions(operand_scaling="token_local", ds_dq_rowlocal="all")
    if case["form"] != "batch":
        lens = _documents(case)
        cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32)
        if case["form"] == "maps":
            kw["doc_maps"] = F.DocMaps.from_cu_seqlens(cu).to("cuda")
        else:
            cu = cu.cuda()
            kw.update(cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(lens), max_seqlen_k=max(lens))
    for t in (q, k, v):
        t.requires_grad_(step)
    return {"fn": F.flash_attn_fp4 if case["entry"] == "fp4" else F.flash_attn_fp8, "q": q, "k": k, "v": v, "do": do, "kw": kw,
            "prescale": tok}


def run(state):
    q, k, v, do = state["q"], state["k"], state["v"], state["do"]
    switches.DQ_CAUSAL_PRESCALE = state["prescale"]        # a module switch that such a program sets once
    if do is None:
        with torch.no_grad():
            return state["fn"](q, k, v, **state["kw"])
    out = state["fn"](q, k, v, **state["kw"])
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), do)
    return out.detach(), dq, dk, dv


# ------------------------------------------------------------------------------------------------------------ what it takes
def _pairs(sq, sk, causal, window, used=None):
    """(query, key) pairs that the mask leaves."""
    i = np.arange(sq, dtype=np.int64) + (sk - sq)
    end = np.minimum(i, sk - 1) if causal else np.minimum(i + window, sk - 1) if window else np.full(sq, sk - 1, np.int64)
    if used is not None:
        end = np.minimum(end, used - 1)
    first = np.maximum(i - window, 0) if window else np.zeros(sq, np.int64)
    return int(np.maximum(end - first + 1, 0).sum())


def work(case):
    if case["form"] == "batch":
        used = _used(case) if case["used"] else [None] * case["b"]
        pairs = sum(_pairs(case["sq"], case["sk"], case["causal"], case["window"], u) for u in used) if case["used"] else \
            case["b"] * _pairs(case["sq"], case["sk"], case["causal"], case["window"])
    else:
        pairs = sum(_pairs(n, n, case["causal"], 0) for n in _documents(case))
    q, kv = case["b"] * case["sq"] * case["h"] * case["d"], case["b"] * case["sk"] * case["hk"] * case["d"]
    step = case["pass"] == "step"
    # forward: read Q, K, V, write O; backward: read dO, write dQ, dK, dV; two products forward, five backward
    return {"bytes": 2 * (2 * q + 2 * kv) + (2 * (2 * q + 2 * kv) if step else 0) + (4 * case["b"] * case["sq"] * case["h"] if case["lse"] else 0),
            "flops": (3.5 if step else 1.0) * 4 * case["h"] * case["d"] * pairs}


def tolerance(case):
    """The probabilities and dS pass through E4M3 (three mantissa bits: a value moves by up to 2^-4, 2.7 % root mean square,
    when it is rounded) on the way into their products. Two correct implementations of the same frames differ where a value
    lies at the edge of a rounding interval, in the order of the f16 sums of dQ, and in the last bit of the 16-bit results."""
    return {"rel": 2e-2}
