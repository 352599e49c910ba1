"""The work that programs have this package do, as cases that can be timed and whose outputs can be compared.

A case is a dict of plain values.  Its "kind" says which public entry point it goes through:

  op      sliding_two_simplicial_attn on device tensors, forward alone ("pass": "fwd") or forward and backward
          through autograd ("fwd_bwd");
  layer   a training pass of SlidingWindowTwoSimplicialMHA under bf16 autocast (fp32 parameters and activations);
  decode  a generation step of the same module in bf16: `new` tokens per sequence against the window caches;
  host    HostPipeline.run on pinned host tensors, forward and backward.

Sizes: b sequences of n rows, hq query and hk key/value heads of d channels, windows w1 and w2.
"""
from __future__ import annotations

import math

import torch

import simplicial_attention_b200 as sa

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def _op(b, n, hq, hk, d, w1, w2, dtype, what):
    return {"kind": "op", "b": b, "n": n, "hq": hq, "hk": hk, "d": d, "w1": w1, "w2": w2, "dtype": dtype, "pass": what}


def _layer(b, n, hq, hk, d, w1, w2):
    return {"kind": "layer", "b": b, "n": n, "hq": hq, "hk": hk, "d": d, "w1": w1, "w2": w2}


def _decode(b, new, hq, hk, d, w1, w2):
    return {"kind": "decode", "b": b, "n": new, "hq": hq, "hk": hk, "d": d, "w1": w1, "w2": w2}


def _host(b, n, hq, hk, d, w1, w2):
    return {"kind": "host", "b": b, "n": n, "hq": hq, "hk": hk, "d": d, "w1": w1, "w2": w2}


def listed():
    return [
        # one sequence generated token by token: the smallest call, all latency
        dict(_decode(1, 1, 8, 4, 64, 512, 32), name="decode_b1"),
        # a serving batch of sequences generated together
        dict(_decode(32, 1, 8, 4, 64, 512, 32), name="decode_b32"),
        # the fp32 correctness configuration (full causal attention: windows as long as the sequence)
        dict(_op(1, 128, 2, 2, 32, 128, 128, "f32", "fwd_bwd"), name="full_causal_f32"),
        # the shape of the reference's own GPU test: a short training pass of few tiles
        dict(_op(2, 128, 4, 4, 64, 64, 32, "bf16", "fwd_bwd"), name="short_bf16"),
        # the forward-only configuration: prefill or evaluation of two sequences
        dict(_op(2, 1024, 8, 8, 64, 512, 32, "bf16", "fwd"), name="prefill_d64"),
        # fp32 training at the usual windows
        dict(_op(1, 1024, 8, 8, 64, 512, 32, "f32", "fwd_bwd"), name="train_f32"),
        # prefill at head dim 128: a prompt of odd length, grouped-query heads
        dict(_op(1, 5001, 16, 4, 128, 512, 32, "bf16", "fwd"), name="prefill_d128"),
        # training on a sequence of odd length with few key/value heads and a long first, short second window
        dict(_op(1, 3001, 8, 2, 64, 1024, 16, "bf16", "fwd_bwd"), name="train_long_window"),
        # one simplicial layer of the 8-layer decoder, forward and backward
        dict(_layer(16, 1024, 8, 4, 64, 512, 32), name="layer_train"),
        # the forward + backward configuration
        dict(_op(4, 4096, 8, 8, 64, 512, 32, "bf16", "fwd_bwd"), name="train_d64"),
        # the same from and to host memory
        dict(_host(4, 4096, 8, 8, 64, 512, 32), name="host_d64"),
        # one GPU's share of the long-sequence configuration: the largest
        dict(_op(1, 16384, 16, 16, 128, 512, 32, "bf16", "fwd_bwd"), name="train_d128"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _heads(rng, most):
    hq = rng.choice([h for h in (1, 2, 3, 4, 6, 8, 12, 16) if h <= most])
    return hq, hq // rng.choice([g for g in (1, 2, 4, 8) if hq % g == 0])


def draw(rng):
    """One more case of the ranges above: windows of 64 ... 1024 and 8 ... 64 rows (or the whole of a short
    sequence), 64 ... 16384 rows, head dims 32 (a small share), 64 and 128."""
    kind = rng.choice(("op", "op", "op", "op", "op", "decode", "decode", "layer", "host"))
    w1, w2 = _log_int(rng, 64, 1024), _log_int(rng, 8, 64)
    if kind == "decode":
        hq, hk = _heads(rng, 16)
        new = 1 if rng.random() < 0.6 else _log_int(rng, 2, 256)
        return _decode(_log_int(rng, 1, 64), new, hq, hk, rng.choice((64, 64, 128)), w1, w2)
    if kind == "layer":
        hq, hk = rng.choice(((8, 8), (8, 4), (8, 2), (4, 4), (4, 1)))
        return _fit(_layer(_log_int(rng, 1, 16), _log_int(rng, 128, 2048), hq, hk, 64, w1, w2), 1.5e12)
    hq, hk = _heads(rng, 16)
    if kind == "host":
        return _fit(_host(_log_int(rng, 1, 8), _log_int(rng, 256, 8192), hq, hk, rng.choice((64, 128)), w1, w2), 3e12)
    dtype, what = rng.choice(("bf16", "bf16", "bf16", "f32")), rng.choice(("fwd", "fwd_bwd"))
    d = rng.choice((32, 64, 64, 64, 128, 128))
    if rng.random() < 0.15:
        n = rng.randint(32, 192)
        return _op(_log_int(rng, 1, 4), n, hq, hk, d, n, n, dtype, what)
    return _fit(_op(_log_int(rng, 1, 8), _log_int(rng, 64, 16384), hq, hk, d, w1, w2, dtype, what),
                7.5e12 if dtype == "bf16" else 5e11)


def _fit(case, most):
    """Fewer sequences, then shorter ones, until a pass takes at most `most` operations."""
    while work(case)["flops"] > most and (case["b"] > 1 or case["n"] > 64):
        if case["b"] > 1:
            case["b"] -= 1
        else:
            case["n"] = max(64, int(case["n"] * 0.8))
    return case


def _pairs(case):
    """Unmasked (j, k) pairs summed over the query rows of one (batch, head)."""
    n, w1, w2 = case["n"], case["w1"], case["w2"]
    if case["kind"] == "decode":                      # every window is full
        return n * w1 * w2
    ramp = min(n, max(w1, w2))
    return sum(min(i + 1, w1) * min(i + 1, w2) for i in range(ramp)) + (n - ramp) * w1 * w2


def work(case):
    """What a pass cannot do without: every input read once, every output written once; 4 d (forward) or 14 d
    (forward and backward) operations per unmasked (row, j, k), plus the layer's two projections."""
    b, n, hq, hk, d, kind = (case[k] for k in ("b", "n", "hq", "hk", "d", "kind"))
    size = 4 if case.get("dtype") == "f32" else 2
    rows_q, rows_k = b * n * hq * d, b * n * hk * d
    pairs = _pairs(case) * b * hq * d
    if kind in ("op", "host"):
        if kind == "op" and case["pass"] == "fwd":
            return {"bytes": size * (2 * rows_q + 4 * rows_k), "flops": 4 * pairs}
        # q, four keys/values, dO in; out and five gradients out
        return {"bytes": size * (4 * rows_q + 8 * rows_k), "flops": 14 * pairs}
    dim = hq * d
    weights = dim * (hq + 4 * hk) * d + hq * d * dim
    if kind == "decode":
        cache = 2 * b * hk * d * (case["w1"] - 1 + case["w2"] - 1)
        return {"bytes": 2 * (weights + 2 * b * n * dim + 2 * cache), "flops": 4 * pairs + 2 * b * n * weights}
    # fp32 parameters and activations: x, dO, out, dx; parameters read, their gradients written
    return {"bytes": 4 * (4 * b * n * dim + 2 * weights), "flops": 14 * pairs + 6 * b * n * weights}


def tolerance(case):
    """fp32: sums of a few thousand 32-bit terms.  bf16: operands, probabilities and results are rounded to 8
    bits.  The gradients of a sequence's first rows see few pairs, where one rounded probability near 1 meets
    |dP - D| ~ sqrt(d): single values there are off by as much as the root mean square of the long rest."""
    if case.get("dtype") == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    forward = case["kind"] == "decode" or case.get("pass") == "fwd"
    return {"rel": 1e-2, "max": 0.3 if forward else 0.95}


def _module(case, dtype, seed):
    torch.manual_seed(seed)
    dim = case["hq"] * case["d"]
    m = sa.SlidingWindowTwoSimplicialMHA(dim=dim, dim_head=case["d"], heads=case["hq"], key_value_heads=case["hk"],
                                         prenorm=True, w1=case["w1"], w2=case["w2"])
    return m.to("cuda", dtype), dim


def prepare(case, seed):
    b, n, hq, hk, d, w1, w2 = (case[k] for k in ("b", "n", "hq", "hk", "d", "w1", "w2"))
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, dtype):
        return torch.randn(shape, generator=gen, device="cuda").to(dtype)

    if case["kind"] == "op":
        dtype = DTYPES[case["dtype"]]
        train = case["pass"] == "fwd_bwd"
        ins = [normal(b, n, hq if x == 0 else hk, d, dtype=dtype).requires_grad_(train) for x in range(5)]
        return {"case": case, "ins": ins, "dout": normal(b, n, hq, d, dtype=dtype) if train else None}
    if case["kind"] == "host":
        shapes = [(b, n, hq, d)] + [(b, n, hk, d)] * 4
        ins = [normal(*s, dtype=torch.bfloat16).cpu().pin_memory() for s in shapes + shapes[:1]]
        outs = [torch.empty(s, dtype=torch.bfloat16).pin_memory() for s in shapes[:1] + shapes]
        return {"case": case, "ins": ins, "outs": outs, "pipe": sa.HostPipeline("cuda", w1=w1, w2=w2)}
    if case["kind"] == "layer":
        m, dim = _module(case, torch.float32, seed)
        x = normal(b, n, dim, dtype=torch.float32).requires_grad_()
        return {"case": case, "module": m, "x": x, "dout": normal(b, n, dim, dtype=torch.bfloat16)}
    m, dim = _module(case, torch.bfloat16, seed)
    with torch.no_grad():       # the prompt: long enough to fill both windows
        prompt = normal(b, max(w1, w2), dim, dtype=torch.bfloat16)
        _, cache = m(prompt, return_cache=True)
    return {"case": case, "module": m, "cache": cache, "x": normal(b, n, dim, dtype=torch.bfloat16)}


def run(state):
    case = state["case"]
    if case["kind"] == "op":
        q, k1, k2, v1, v2 = state["ins"]
        if case["pass"] == "fwd":
            with torch.no_grad():
                return sa.sliding_two_simplicial_attn(q, (k1, k2), (v1, v2), w1=case["w1"], w2=case["w2"])
        for t in state["ins"]:
            t.grad = None
        out = sa.sliding_two_simplicial_attn(q, (k1, k2), (v1, v2), w1=case["w1"], w2=case["w2"])
        out.backward(state["dout"])
        return [out.detach()] + [t.grad for t in state["ins"]]
    if case["kind"] == "host":
        state["pipe"].run(state["ins"], state["outs"])
        return state["outs"]
    if case["kind"] == "layer":
        m, x = state["module"], state["x"]
        x.grad = None
        m.zero_grad(set_to_none=True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = m(x)
        out.backward(state["dout"])
        return [out.detach(), x.grad] + [p.grad for p in m.parameters()]
    with torch.no_grad():
        out, cache = state["module"](state["x"], cache=state["cache"], return_cache=True)
    return out, cache
