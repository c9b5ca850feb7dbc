"""The work a user of this package has it do on one GPU, as cases that can be timed and compared.

Every multi-GPU operator is built from the kernels measured here: the tcgen05 GEMM in its three
operand formats, the attention kernel that serves local, ring and Ulysses use, and the expert
layer.  With one rank a ``CommContext`` has no peers, so a case is one rank's share of the work.

``listed()`` spans the range of each path, ``draw(rng)`` gives another case of the same ranges.
A case is prepared from a seed (inputs, weights, the layer object a program keeps), ``run`` makes
one pass through the public entry points and returns its outputs.
"""
from __future__ import annotations

import math

import torch

from commbench_b200.models.tp_mlp import TPMLP
from commbench_b200.ops.cp import RingAttention, flash_attention
from commbench_b200.ops.gemm import (gemm, gemm_fp8_blockscaled, gemm_fp8_mx,
                                     quantize_blockscaled)
from commbench_b200.ops.moe import MoELayer, router_topk
from commbench_b200.ops.tp_fp8 import MxWeight, quantize_act_mx
from commbench_b200.runtime.context import CommContext

HEAD = 128                       # the attention kernels' head dimension


def listed():
    return [
        # Row-parallel linear of a decode step on one of eight ranks (the GEMM + all-reduce
        # shape M = 16, K = 8192 / 8, N = 8192): the smallest call, launch latency and 17 MB.
        dict(name="gemm_decode", path="gemm", m=16, n=8192, k=1024),
        # A linear layer on a batch that is no multiple of any tile in any dimension.
        dict(name="gemm_ragged", path="gemm", m=777, n=5000, k=3080),
        # One decode step of the tensor-parallel MLP block with one of eight ranks' weights:
        # two weight-bound GEMMs in a row.
        dict(name="mlp_decode", path="mlp", t=48, hidden=8192, inter=3584),
        # The flagship block: the benchmark's prefill step on one rank, the largest case.
        dict(name="mlp_prefill", path="mlp", t=8192, hidden=8192, inter=28672),
        # Column-parallel linear of the same block on one of eight ranks, fp8 operands with one
        # scale per tensor.
        dict(name="gemm_fp8", path="fp8", m=8192, n=3584, k=8192),
        # The same linear with power-of-two 1x128 / 128x128 block scales: quantise the activation,
        # multiply with the kept weight.
        dict(name="linear_fp8_mx", path="mx", m=8192, n=3584, k=8192),
        # Row-parallel linear with fp32 block scales on a ragged batch.
        dict(name="linear_fp8_blockscaled", path="bs", m=3000, n=8192, k=3584),
        # One rank's share of the context-parallel configuration: 16384 tokens, 32 query and 8
        # key/value heads, causal, keys and values written in place in the ring's own slot.
        dict(name="attn_prefill", path="ring", b=1, s=16384, hq=32, hkv=8, causal=True),
        # Chunked prefill: a ragged chunk of queries behind a cached prefix.
        dict(name="attn_chunk", path="attn", b=1, sq=1000, skv=7000, hq=32, hkv=8, causal=True),
        # Decode: one query token per sequence over a cached context of no round length.
        dict(name="attn_decode", path="attn", b=16, sq=1, skv=6001, hq=32, hkv=8, causal=True),
        # The expert layer of the expert-parallel configuration on one rank: 4096 tokens, top-8 over
        # its 32 experts, hidden 7168, intermediate 2048, fp8 dispatch.
        dict(name="moe_prefill", path="moe", t=4096, hidden=7168, inter=2048, experts=32, topk=8,
             per_token=False),
        # The same layer in a decode step: the expert weights are read for a few rows each.
        dict(name="moe_decode", path="moe", t=100, hidden=7168, inter=2048, experts=32, topk=8,
             per_token=False),
    ]


def _log_int(rng, lo, hi, mult=1):
    """An integer of [lo, hi], spread over its logarithm, a multiple of ``mult``."""
    x = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(max(x // mult * mult, lo), hi)


def draw(rng):
    path = rng.choice(["gemm", "gemm", "mlp", "fp8", "mx", "bs", "ring", "attn", "attn", "moe"])
    if path == "gemm":
        return dict(path=path, m=_log_int(rng, 1, 8192), n=_log_int(rng, 512, 16384, 8),
                    k=_log_int(rng, 512, 8192, 8))
    if path == "mlp":
        return dict(path=path, t=_log_int(rng, 1, 8192), hidden=rng.choice([2048, 4096, 8192]),
                    inter=_log_int(rng, 1792, 28672, 8))
    if path == "fp8":
        return dict(path=path, m=_log_int(rng, 16, 8192), n=_log_int(rng, 512, 8192, 8),
                    k=_log_int(rng, 512, 8192, 16))
    if path in ("mx", "bs"):
        return dict(path=path, m=_log_int(rng, 16, 8192), n=_log_int(rng, 512, 8192, 8),
                    k=_log_int(rng, 512, 8192, 128))
    if path == "ring":
        hkv = rng.choice([1, 2, 4, 8])
        return dict(path=path, b=1, s=_log_int(rng, 512, 16384, 256),
                    hq=hkv * rng.choice([1, 2, 4]), hkv=hkv, causal=rng.random() < 0.75)
    if path == "attn":
        hkv = rng.choice([1, 2, 4, 8])
        if rng.random() < 0.5:                       # decode, a few query tokens at most
            return dict(path=path, b=_log_int(rng, 1, 32), sq=rng.choice([1, 1, 1, 2, 4]),
                        skv=_log_int(rng, 256, 16384), hq=hkv * rng.choice([1, 4, 8]), hkv=hkv,
                        causal=True)
        sq = _log_int(rng, 64, 8192)
        return dict(path=path, b=rng.choice([1, 2]), sq=sq, skv=sq + rng.choice([0, 0, 777, 4096]),
                    hq=hkv * rng.choice([1, 4]), hkv=hkv, causal=rng.random() < 0.75)
    return dict(path="moe", t=_log_int(rng, 8, 4096), hidden=rng.choice([2048, 4096, 7168]),
                inter=rng.choice([1024, 2048]), experts=rng.choice([8, 16, 32, 64]),
                topk=rng.choice([2, 4, 8]), per_token=rng.random() < 0.3)


class _State:
    """What a program holds between calls; a context is closed with its state."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        ctx = self.__dict__.get("ctx")
        if ctx is not None:
            ctx.close()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    path = case["path"]

    def randn(*shape, scale=1.0):
        return (torch.randn(*shape, device=dev, generator=g) * scale).bfloat16()

    if path in ("gemm", "fp8", "mx", "bs"):
        m, n, k = case["m"], case["n"], case["k"]
        x, w = randn(m, k), randn(n, k, scale=0.02)
        if path == "gemm":
            return _State(path=path, x=x, w=w)
        if path == "fp8":
            # one scale per tensor, folded into alpha
            sx, sw = x.abs().max().float() / 448.0, w.abs().max().float() / 448.0
            return _State(path=path, x=(x.float() / sx).to(torch.float8_e4m3fn),
                          w=(w.float() / sw).to(torch.float8_e4m3fn), alpha=float(sx * sw))
        if path == "mx":
            return _State(path=path, x=x, w=MxWeight.from_bf16(w))
        wq, ws = quantize_blockscaled(w, 128)
        return _State(path=path, x=x, wq=wq, ws=ws)
    if path == "mlp":
        t = case["t"]
        ctx = CommContext(heap_bytes=2 << 20)
        layer = TPMLP(ctx, case["hidden"], case["inter"], (t + 127) // 128 * 128, seed=seed)
        return _State(path=path, ctx=ctx, layer=layer, x=randn(t, case["hidden"]))
    if path == "ring":
        b, s, hq, hkv = case["b"], case["s"], case["hq"], case["hkv"]
        ctx = CommContext(heap_bytes=4 * b * s * hkv * HEAD + (4 << 20))
        op = RingAttention(ctx, b, s, hq, hkv)
        op.k_local().copy_(randn(b, s, hkv, HEAD))
        op.v_local().copy_(randn(b, s, hkv, HEAD))
        return _State(path=path, ctx=ctx, op=op, q=randn(b, s, hq, HEAD), causal=case["causal"])
    if path == "attn":
        b, hkv = case["b"], case["hkv"]
        return _State(path=path, q=randn(b, case["sq"], case["hq"], HEAD),
                      k=randn(b, case["skv"], hkv, HEAD), v=randn(b, case["skv"], hkv, HEAD),
                      causal=case["causal"], q_offset=case["skv"] - case["sq"])
    t, h, inter, e, k = (case[x] for x in ("t", "hidden", "inter", "experts", "topk"))
    rows = 2 * t * k + e * 128
    ctx = CommContext(heap_bytes=rows * (h + h // 32 + 8) + t * k * h * 2 + (8 << 20))
    layer = MoELayer(ctx, t, h, inter, e, k, seed=seed,
                     dispatch="per_token" if case["per_token"] else "per_pair")
    logits = torch.randn(t, e, device=dev, generator=g)
    return _State(path="moe", ctx=ctx, layer=layer, x=randn(t, h), logits=logits, topk=k)


def run(s):
    if s.path == "gemm":
        return gemm(s.x, s.w)
    if s.path == "mlp":
        return s.layer.forward(s.x)
    if s.path == "fp8":
        return gemm(s.x, s.w, alpha=s.alpha)
    if s.path == "mx":
        q, sf = quantize_act_mx(s.x)
        return gemm_fp8_mx(q, sf, s.w.q, s.w.sf)
    if s.path == "bs":
        q, sc = quantize_blockscaled(s.x, 1)
        return gemm_fp8_blockscaled(q, sc, s.wq, s.ws)
    if s.path == "ring":
        return s.op.forward(s.q, s.op.k_local(), s.op.v_local(), causal=s.causal)
    if s.path == "attn":
        return flash_attention(s.q, s.k, s.v, causal=s.causal, q_offset=s.q_offset)
    idx, w = router_topk(s.logits, s.topk)
    return s.layer.forward(s.x, idx, w)


def work(case):
    path = case["path"]
    if path in ("gemm", "fp8", "mx", "bs"):
        m, n, k = case["m"], case["n"], case["k"]
        xb, wb = {"gemm": (2, 2), "fp8": (1, 1), "mx": (2, 1), "bs": (2, 1)}[path]
        return {"bytes": m * k * xb + n * k * wb + m * n * 2, "flops": 2 * m * n * k}
    if path == "mlp":
        t, h, i = case["t"], case["hidden"], case["inter"]
        return {"bytes": 2 * (2 * t * h + 2 * h * i), "flops": 4 * t * h * i}
    if path in ("ring", "attn"):
        b, hq, hkv = case["b"], case["hq"], case["hkv"]
        sq, skv = (case["s"],) * 2 if path == "ring" else (case["sq"], case["skv"])
        # visible (query, key) pairs: the last query sees every key
        pairs = sq * skv - (sq * (sq - 1) // 2 if case["causal"] else 0)
        return {"bytes": b * (2 * sq * hq * HEAD * 2 + 2 * skv * hkv * HEAD * 2 + sq * hq * 4),
                "flops": 4 * b * hq * HEAD * pairs}
    t, h, i, e, k = (case[x] for x in ("t", "hidden", "inter", "experts", "topk"))
    used = e * (1.0 - (1.0 - k / e) ** t)            # experts that at least one token selects
    return {"bytes": int(t * h * 4 + t * e * 4 + used * 3 * h * i * 2), "flops": 6 * t * k * h * i}


# Largest relative error (2-norm) per path: about four times the distance of the path from the same
# computation in 64 bits on the same operands.  Measured: 1.7e-3 for every GEMM (the rounding of
# the bf16 result), 2.0e-3 to 2.4e-3 for attention (bf16 probabilities as well), 4.5e-3 for the
# expert layer (three bf16 roundings in a row).
_REL = {"gemm": 7e-3, "mlp": 7e-3, "fp8": 7e-3, "mx": 7e-3, "bs": 7e-3, "ring": 9e-3, "attn": 9e-3,
        "moe": 1.8e-2}


def tolerance(case):
    return {"rel": _REL[case["path"]]}


def _q64(x, rows, pow2=False):
    """bf16 [r, K] -> the fp64 values of its e4m3 form with one scale per ``rows`` rows and 128
    columns (fp32 scales amax / 448, rounded up to a power of two with ``pow2``): the quantisation
    is part of the measured call, so the exact result is that of the quantised operands."""
    r, k = x.shape
    pad = (-r) % rows
    f = torch.nn.functional.pad(x.float(), (0, 0, 0, pad)).view((r + pad) // rows, rows, k // 128, 128)
    amax = f.abs().amax(dim=(1, 3), keepdim=True)
    # a tensor divided by a number is multiplied by its reciprocal on a GPU; divide in earnest
    s = torch.where(amax > 0, amax / torch.full_like(amax, 448.0), torch.ones_like(amax))
    if pow2:
        m, e = torch.frexp(s)                        # s = m * 2^e, m in [0.5, 1)
        s = torch.ldexp(torch.ones_like(s), torch.where(m == 0.5, e - 1, e))
    q = (f * (1.0 / s)).to(torch.float8_e4m3fn)
    return (q.double() * s.double()).view(r + pad, k)[:r]


def _attention64(q, k, v, causal, q_offset):
    """(o, lse) of [B, S, H, 128] tensors in 64 bits, one head and 2048 queries at a time."""
    b, sq, hq, d = q.shape
    skv, hkv = k.shape[1], k.shape[2]
    o = torch.empty(b, sq, hq, d, dtype=torch.float64, device=q.device)
    lse = torch.empty(b, hq, sq, dtype=torch.float64, device=q.device)
    cols = torch.arange(skv, device=q.device)
    for bi in range(b):
        for h in range(hq):
            kh, vh = (t[bi, :, h // (hq // hkv)].double() for t in (k, v))
            for r in range(0, sq, 2048):
                s = q[bi, r:r + 2048, h].double() @ kh.t() / math.sqrt(d)
                if causal:
                    rows = torch.arange(r, r + s.shape[0], device=q.device)[:, None] + q_offset
                    s.masked_fill_(cols[None, :] > rows, float("-inf"))
                ls = torch.logsumexp(s, dim=-1)
                lse[bi, h, r:r + 2048] = ls
                o[bi, r:r + 2048, h] = torch.exp(s - ls[:, None]) @ vh
    return o, lse


def exact(case, seed):
    path = case["path"]
    s = prepare(case, seed)
    if path == "gemm":
        return s.x.double() @ s.w.double().t()
    if path == "fp8":
        return s.alpha * (s.x.double() @ s.w.double().t())
    if path in ("mx", "bs"):
        # the weight as prepare() drew it, right after the activation
        dev = s.x.device
        g = torch.Generator(device=dev).manual_seed(seed)
        torch.randn(case["m"], case["k"], device=dev, generator=g)
        w = (torch.randn(case["n"], case["k"], device=dev, generator=g) * 0.02).bfloat16()
        return _q64(s.x, 1, path == "mx") @ _q64(w, 128, path == "mx").t()
    if path == "mlp":
        return (s.x.double() @ s.layer.w1.double().t()) @ s.layer.w2.double().t()
    if path == "ring":
        return _attention64(s.q, s.op.k_local(), s.op.v_local(), s.causal, 0)
    if path == "attn":
        return _attention64(s.q, s.k, s.v, s.causal, s.q_offset)
    w1, w2 = s.layer.weights()
    top, idx = torch.topk(torch.softmax(s.logits.double(), dim=1), s.topk, dim=1)
    weight = top / top.sum(dim=1, keepdim=True)
    x = _q64(s.x, 1)
    y = torch.zeros_like(x)
    inter = case["inter"]
    for e in range(case["experts"]):
        t, k = (idx == e).nonzero(as_tuple=True)
        h = x[t] @ w1[e].double().t()
        o = (torch.nn.functional.silu(h[:, :inter]) * h[:, inter:]) @ w2[e].double().t()
        y.index_add_(0, t, o * weight[t, k][:, None])
    return y
