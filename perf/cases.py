"""The work that users of this package have it do, as a list of measurable cases.

A case is a dict of plain values.  `listed()` holds twelve of them, `draw(rng)` gives more of the same
ranges, `prepare(case, seed)` makes what a program has in hand before the call, `run(state)` is one pass
through the public entry points, `work(case)` what such a pass cannot do without and `tolerance(case)`
how far another correct implementation may be from it.

Lengths are a function of the case alone (its "lens" number seeds them); the seed given to `prepare`
changes the values.  Values are N(0,1) and weights N(0, 1/d), the distributions the benchmark and the
tests use for both operators.
"""
from __future__ import annotations

import math
import random

import torch

import varlenabsorbflashattn_b200 as vb

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}

# dearest work of a listed case (train_long, decode_long), which a drawn one stays under
_MOST_FLOPS = 1.4e13
_MOST_BYTES = 1.7e10


# ------------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------------
def _self(n, lo, hi, H, D, dtype, causal, grad, lens, H_kv=None, check=True):
    """Self-attention over a packed batch of n sequences, lengths log-uniform in [lo, hi]."""
    return dict(op="varlen", kind="self", n=n, q_len=0, lo=lo, hi=hi, cap=0.0, H=H, H_kv=H_kv or H, D=D, dtype=dtype,
                causal=causal, grad=grad, check=check, lens=lens)


def _cross(n, q_len, lo, hi, cap, H, D, dtype, grad, lens, H_kv=None, check=True):
    """q_len queries per segment over its own keys: lengths log-uniform in [lo, hi], a share `cap` of them hi."""
    return dict(op="varlen", kind="cross", n=n, q_len=q_len, lo=lo, hi=hi, cap=cap, H=H, H_kv=H_kv or H, D=D, dtype=dtype,
                causal=False, grad=grad, check=check, lens=lens)


def _absorb(n, q_hi, lo, hi, cap, d_q, d_kv, dtype, grad, lens, check=True):
    """Target attention of n users: 1..q_hi targets each over a history of log-uniform length, H=8, D_H=32."""
    return dict(op="absorb", kind="absorb", n=n, q_hi=q_hi, lo=lo, hi=hi, cap=cap, d_q=d_q, d_kv=d_kv, dtype=dtype,
                grad=grad, check=check, lens=lens)


def listed():
    cases = {
        # the smallest call there is: four sequences of 17 to 255 tokens, H=8, D=64, in the default dtype of torch
        "self_small_fp32": _self(4, 17, 255, 8, 64, "fp32", False, False, 0),
        # one step of a small serving batch: 8 requests decode one token each over caches of up to 4096 keys
        # (the loop has its checks switched off, as it builds cu_seqlens itself)
        "decode_small": _cross(8, 1, 512, 4096, 0.0, 8, 128, "bf16", False, 1, check=False),
        # decode over long caches, 256 requests of 8k to 32k keys (the split-K path at its largest)
        "decode_long": _cross(256, 1, 8192, 32768, 0.0, 8, 128, "bf16", False, 0, check=False),
        # decode with grouped-query heads, a mid-size serving batch of unequal caches
        "decode_gqa": _cross(64, 1, 1024, 16384, 0.0, 32, 128, "bf16", False, 2, H_kv=8, check=False),
        # prefill of a serving batch: fp16, causal, grouped-query heads, forward only
        "prefill_gqa_fp16": _self(16, 128, 8192, 32, 128, "fp16", True, False, 3, H_kv=8),
        # a training step of an ordinary batch: 64 sequences of 1 to 4096 tokens, most of them ragged and short
        "train_causal": _self(64, 1, 4096, 16, 128, "bf16", True, True, 0),
        # a training step of a large batch of long sequences (an eighth of the 1 M-token batch: one GPU's share of it)
        "train_long": _self(65, 128, 8192, 32, 128, "bf16", True, True, 0),
        # training on long user histories: 500 queries per user over up to 102 400 keys, 4 heads of 64
        "train_history": _cross(16, 500, 1, 102400, 0.55, 4, 64, "bf16", True, 0),
        # target attention, one ranking request batch: forward only, checks off
        "absorb_serve": _absorb(32, 16, 8, 2048, 0.0, 256, 256, "bf16", False, 1, check=False),
        # target attention, a training step of 1024 users
        "absorb_train": _absorb(1024, 16, 8, 2048, 0.0, 256, 256, "bf16", True, 0),
        # the same at the production widths: raw features 968 and 216, nearly every history at its cap
        "absorb_prod": _absorb(1137, 10, 8, 2048, 0.97, 968, 216, "bf16", True, 2),
        # a training step in fp32, the default dtype of the operator, on a small batch
        "absorb_fp32": _absorb(64, 16, 8, 2048, 0.0, 256, 256, "fp32", True, 3),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    """One more case of the ranges above, cut down to what the dearest listed case costs."""
    lens = rng.randrange(1 << 20)
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    which = rng.randrange(7)
    if which == 0:  # training or prefill of a packed batch
        D, H = rng.choice((64, 128, 128)), rng.choice((4, 8, 16, 32))
        hi = _logint(rng, 64, 8192)
        c = _self(_logint(rng, 1, 160), _logint(rng, 1, max(1, hi // 4)), hi, H, D, dtype, rng.random() < 0.7, rng.random() < 0.7,
                  lens, H_kv=H // rng.choice((1, 1, 1, 4)))
    elif which == 1:  # the same over a few sequences, where a call is short
        D, H = rng.choice((64, 128)), rng.choice((2, 4, 8, 16))
        hi = _logint(rng, 32, 512)
        c = _self(_logint(rng, 1, 16), _logint(rng, 1, hi), hi, H, D, dtype, rng.random() < 0.5, rng.random() < 0.5, lens)
    elif which == 2:  # decode
        H = rng.choice((8, 16, 32))
        hi = _logint(rng, 512, 32768)
        c = _cross(_logint(rng, 1, 256), rng.choice((1, 1, 1, 2, 4)), _logint(rng, 128, hi), hi, 0.0, H, 128, dtype, False, lens,
                   H_kv=H // rng.choice((1, 1, 4, 8)), check=False)
    elif which == 3:  # queries of a user over a history of their own length
        D, H = rng.choice((64, 64, 128)), rng.choice((2, 4, 8))
        c = _cross(_logint(rng, 2, 32), _logint(rng, 60, 600), 1, _logint(rng, 2048, 102400), rng.choice((0.0, 0.5)), H, D, dtype,
                   rng.random() < 0.7, lens)
    elif which == 4:  # target attention at the benchmark's widths
        c = _absorb(_logint(rng, 8, 4096), rng.randint(1, 18), 8, _logint(rng, 64, 4096), rng.choice((0.0, 0.5)), 256, 256, dtype,
                    rng.random() < 0.6, lens, check=rng.random() < 0.5)
    elif which == 5:  # target attention at raw feature widths
        c = _absorb(_logint(rng, 8, 1400), rng.randint(2, 18), 8, _logint(rng, 256, 2048), rng.choice((0.0, 0.97)),
                    rng.choice((968, 512, 256)), rng.choice((216, 192)), dtype, rng.random() < 0.6, lens, check=rng.random() < 0.5)
    elif rng.random() < 0.5:  # fp32, small batches of either operator
        hi = _logint(rng, 64, 1024)
        c = _self(_logint(rng, 1, 8), _logint(rng, 1, hi), hi, rng.choice((2, 4, 8)), rng.choice((32, 64, 128)), "fp32",
                  rng.random() < 0.5, rng.random() < 0.5, lens)
    else:
        c = _absorb(_logint(rng, 4, 96), rng.randint(1, 16), 8, _logint(rng, 64, 2048), 0.0, 256, rng.choice((256, 216, 128)), "fp32",
                    rng.random() < 0.5, lens)
    while c["n"] > 1:
        w = work(c)
        if w["flops"] <= _MOST_FLOPS and w["bytes"] <= _MOST_BYTES:
            break
        c["n"] = c["n"] * 3 // 4
    return c


# ------------------------------------------------------------------------------------------------
# lengths and work
# ------------------------------------------------------------------------------------------------
def _lengths(c):
    """(query lengths, key lengths) of the case's segments."""
    r = random.Random(c["lens"])
    keys = []
    for _ in range(c["n"]):
        L = _logint(r, c["lo"], c["hi"])
        keys.append(c["hi"] if r.random() < c["cap"] else L)
    if c["kind"] == "self":
        return keys, keys
    if c["kind"] == "cross":
        return [c["q_len"]] * c["n"], keys
    return [r.randint(1, c["q_hi"]) for _ in keys], keys


def work(case):
    ql, kl = _lengths(case)
    Tq, Tk, es = sum(ql), sum(kl), _BYTES[case["dtype"]]
    if case["op"] == "varlen":
        H, H_kv, D = case["H"], case["H_kv"], case["D"]
        cells = sum(L * (L + 1) // 2 for L in ql) if case["causal"] else sum(a * b for a, b in zip(ql, kl))
        io = Tq * H * D + 2 * Tk * H_kv * D          # q, k, v
        n = io + Tq * H * D                          # o
        flops = 4 * H * D * cells
        if case["grad"]:
            n += Tq * H * D + io                     # dO; dq, dk, dv
            flops *= 3.5
        return {"bytes": n * es, "flops": flops}
    H, D_H, d_q, d_kv = 8, 32, case["d_q"], case["d_kv"]
    weights = (d_q + 2 * d_kv) * H * D_H
    io = Tq * d_q + Tk * d_kv + weights
    n = io + Tq * H * D_H
    core = 4 * H * d_kv * sum(a * b for a, b in zip(ql, kl))
    proj = 2 * Tq * H * D_H * (d_q + 2 * d_kv)
    flops = core + proj
    if case["grad"]:
        n += Tq * H * D_H + io
        flops += 2.5 * core + 2 * proj
    return {"bytes": n * es, "flops": flops}


def tolerance(case):
    """Four times the largest errors seen against the same inputs in 64 bits, over the listed cases and drawn ones:
    16-bit types round P, dS, the projections and the outputs to the type (rel 4.5e-3 in bf16 and 5.7e-4 in
    fp16 through the chained weight gradients, single elements of dk up to 0.47 rms in bf16); fp32 sums in
    fp32 (rel 7e-7, max 2.2e-5)."""
    return {"bf16": {"rel": 1.8e-2, "max": 0.95}, "fp16": {"rel": 2.3e-3, "max": 0.1},
            "fp32": {"rel": 3e-6, "max": 1e-4}}[case["dtype"]]


# ------------------------------------------------------------------------------------------------
# inputs and the pass
# ------------------------------------------------------------------------------------------------
def _cu(lens):
    return torch.tensor([0] + lens, dtype=torch.int64).cumsum(0).to(torch.int32).cuda()


def prepare(case, seed):
    ql, kl = _lengths(case)
    Tq, Tk = sum(ql), sum(kl)
    dtype = _DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, std=1.0):
        t = torch.randn(shape, generator=gen, device="cuda", dtype=dtype)
        return t if std == 1.0 else t.mul_(std)

    s = {"op": case["op"], "check": case["check"], "causal": case.get("causal", False), "cu_q": _cu(ql), "cu_k": _cu(kl), "dO": None}
    if case["op"] == "varlen":
        H, H_kv, D = case["H"], case["H_kv"], case["D"]
        s["inputs"] = [randn(Tq, H, D), randn(Tk, H_kv, D), randn(Tk, H_kv, D)]
        d_o = (Tq, H, D)
    else:
        H, D_H, d_q, d_kv = 8, 32, case["d_q"], case["d_kv"]
        s["inputs"] = [randn(Tq, d_q), randn(Tk, d_kv)] + [randn(d, H, D_H, std=d ** -0.5) for d in (d_q, d_kv, d_kv)]
        d_o = (Tq, H, D_H)
    if case["grad"]:
        s["inputs"] = [t.requires_grad_(True) for t in s["inputs"]]
        s["dO"] = randn(*d_o)
    return s


def _forward(s):
    if s["op"] == "varlen":
        vb.set_validate_cu_seqlens(s["check"])
        return vb.packed_varlen_attn(*s["inputs"], cu_seqlens_q=s["cu_q"], cu_seqlens_k=s["cu_k"], causal=s["causal"])
    return vb.packed_target_attn(*s["inputs"], cu_seqlens_q=s["cu_q"], cu_seqlens_k=s["cu_k"], validate=s["check"])


def run(s):
    if s["dO"] is None:
        with torch.no_grad():
            return {"o": _forward(s)}
    o = _forward(s)
    grads = torch.autograd.grad(o, s["inputs"], s["dO"])
    return {"o": o.detach(), "grads": list(grads)}
