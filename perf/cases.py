"""The attention and block-mask work whose speed is measured, through the package's public entry points.

A case names one call (``masked_attention_via_map`` forward, or forward and backward, ``flex_attention`` with a
BlockMask, or ``create_block_mask``) and its sizes.  ``listed()`` gives one or two cases of every kind of use,
``draw()`` further ones of the same ranges.
"""
import math

import numpy as np
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import masks as M

F32, BF16 = "float32", "bfloat16"


def _case(api, dtype, B, N, L, Hq, Hkv, d, mask, *, grad, block_size=0, window=0, scaled=False, bf16_out=False):
    """``block_size`` 0: the argument is left out.  ``window``: keys to either side (or behind, for a causal mask) that
    a query sees.  ``scaled``: Q, K, V carry the factor 1/sqrt(d).  ``bf16_out``: the output in bfloat16."""
    return dict(api=api, dtype=dtype, B=B, N=N, L=L, Hq=Hq, Hkv=Hkv, d=d, mask=mask, grad=grad, block_size=block_size,
                window=window, scaled=scaled, bf16_out=bf16_out)


def _blocks(B, H, L, block_size, mask, window=0):
    return dict(api="block_mask", B=B, Hq=H, N=L, L=L, block_size=block_size, mask=mask, window=window)


def listed():
    cases = {
        # the reference's own scale of use: a small float32 model, one layer's training step; all latency
        "f32_causal_tiny": _case("map", F32, 2, 128, 128, 8, 8, 64, "causal", grad=True, block_size=32),
        # float32 training at an ordinary context
        "f32_causal_train": _case("map", F32, 2, 2048, 2048, 16, 16, 64, "causal", grad=True, block_size=128),
        # float32 inference without a mask (an encoder), ragged length, grouped heads
        "f32_encoder_ragged": _case("map", F32, 1, 1500, 1500, 16, 4, 128, "none", grad=False),
        # training on short ragged sequences with a mask written as a plain Python function
        "bf16_lambda_ragged": _case("map", BF16, 2, 1000, 1000, 16, 4, 128, "lambda_window", grad=True, window=256),
        # a few new queries against long cached keys (chunked decoding): the last N positions of L, causal
        "bf16_few_queries": _case("map", BF16, 4, 16, 8192, 32, 8, 128, "tail", grad=False, block_size=128, bf16_out=True),
        # prompt processing: a long causal forward
        "bf16_causal_prefill": _case("map", BF16, 4, 8192, 8192, 32, 32, 128, "causal", grad=False, block_size=128, bf16_out=True),
        # dense causal training step (the benchmark's headline shape)
        "bf16_causal_train": _case("map", BF16, 8, 4096, 4096, 32, 32, 128, "causal", grad=True, block_size=128, scaled=True),
        # sliding-window local attention, training (the benchmark's local shape)
        "bf16_sliding_train": _case("map", BF16, 4, 8192, 8192, 16, 16, 128, "sliding", grad=True, block_size=128, window=256),
        # packed documents, training (the benchmark's packed shape): every row of the batch has its own segments
        "bf16_documents_train": _case("map", BF16, 4, 16384, 16384, 16, 16, 128, "documents", grad=True),
        # one long sequence, training: what each of 8 GPUs holds of 32 heads
        "bf16_long_train": _case("map", BF16, 1, 131072, 131072, 4, 4, 128, "causal", grad=True, block_size=128),
        # flex_attention with a BlockMask kept from step to step, grouped heads of 64
        "flex_bf16_gqa_d64": _case("flex", BF16, 4, 4096, 4096, 32, 8, 64, "causal", grad=True, block_size=128),
        # building the block lists of a long causal mask for every head
        "block_mask_long": _blocks(1, 32, 131072, 128, "causal"),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng, lo, hi):
    """(query heads, kv heads): alike, or in groups of 2, 4 or 8."""
    G = rng.choice((1, 1, 2, 4, 8))
    Hkv = max(1, _spread(rng, lo, hi) // G)
    return Hkv * G, Hkv


def _length(rng, lo, hi):
    """Half of the lengths are whole tiles, half are whatever comes."""
    n = _spread(rng, lo, hi)
    return max(128, n // 128 * 128) if rng.random() < 0.5 else n


def _draw(rng):
    kind = rng.choice(("f32_train", "f32_forward", "ragged", "few_queries", "prefill", "train", "sliding", "documents",
                       "long", "flex", "block_mask"))
    B, d = _spread(rng, 1, 8), rng.choice((64, 128))
    if kind == "f32_train":
        n = _spread(rng, 64, 4096)
        Hq, Hkv = _heads(rng, 4, 16)
        return _case("map", F32, min(B, 4), n, n, Hq, Hkv, rng.choice((32, 64, 64, 128)), "causal", grad=True)
    if kind == "f32_forward":
        n = _spread(rng, 64, 4096)
        Hq, Hkv = _heads(rng, 4, 16)
        return _case("map", F32, min(B, 4), n, n, Hq, Hkv, rng.choice((32, 64, 128, 128)), rng.choice(("none", "causal")), grad=False)
    if kind == "ragged":
        n = _spread(rng, 128, 4096)
        Hq, Hkv = _heads(rng, 8, 32)
        return _case("map", BF16, B, n, n, Hq, Hkv, d, "lambda_window", grad=True, window=_spread(rng, 32, 1024))
    if kind == "few_queries":
        Hq, Hkv = _heads(rng, 8, 64)
        return _case("map", BF16, B, _spread(rng, 1, 127), _spread(rng, 1024, 65536), Hq, Hkv, d, "tail", grad=False, block_size=128,
                     bf16_out=rng.random() < 0.5)
    if kind == "prefill":
        n = _length(rng, 512, 16384)
        Hq, Hkv = _heads(rng, 8, 32)
        return _case("map", BF16, B, n, n, Hq, Hkv, d, "causal", grad=False, bf16_out=rng.random() < 0.5)
    if kind == "train":
        n = _length(rng, 512, 8192)
        Hq, Hkv = _heads(rng, 8, 32)
        return _case("map", BF16, B, n, n, Hq, Hkv, d, "causal", grad=True, scaled=rng.random() < 0.5)
    if kind == "sliding":
        n = _length(rng, 1024, 16384)
        Hq, Hkv = _heads(rng, 8, 16)
        return _case("map", BF16, min(B, 4), n, n, Hq, Hkv, d, "sliding", grad=True, window=_spread(rng, 64, 1024))
    if kind == "documents":
        n = _length(rng, 2048, 16384)
        Hq, Hkv = _heads(rng, 8, 16)
        return _case("map", BF16, min(B, 4), n, n, Hq, Hkv, d, "documents", grad=True)
    if kind == "long":
        n = _length(rng, 32768, 100000)
        H = rng.choice((1, 2, 4))
        return _case("map", BF16, 1, n, n, H, H, d, "causal", grad=True)
    if kind == "flex":
        n = 128 * _spread(rng, 4, 64)
        Hq, Hkv = _heads(rng, 8, 32)
        return _case("flex", BF16, min(B, 4), n, n, Hq, Hkv, d, "causal", grad=rng.random() < 0.5, block_size=128)
    bs = rng.choice((64, 128, 256))
    n = min(_spread(rng, 1024, 131072), 1024 * bs) // bs * bs
    mask = rng.choice(("causal", "sliding"))
    return _blocks(min(B, 4), _spread(rng, 4, 32) if n < 65536 else 8, n, bs, mask, 0 if mask == "causal" else _spread(rng, 64, 4096))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        c = _draw(rng)
        if work(c)["flops"] <= most:
            return c


def _randn(shape, seed, dtype, scale=1.0):
    x = torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
    if scale != 1.0:
        x.mul_(scale)
    return x.to(getattr(torch, dtype))


def _segments(B, L, seed):
    """Packed documents of 256 to 4096 tokens, cut at the end of the row: segment ids [B, L]."""
    rng = np.random.default_rng(seed)
    out = np.zeros((B, L), np.int32)
    for b in range(B):
        lengths = rng.integers(256, 4097, size=L // 256 + 1)
        out[b] = np.repeat(np.arange(lengths.size, dtype=np.int32), lengths)[:L]
    return out


def prepare(case, seed):
    c = case
    if c["api"] == "block_mask":
        # the lists depend on no array; the seed moves the far end of what a query sees (a causal mask reaches back over
        # at least half of the sequence)
        if c["mask"] == "causal":
            mask = M.sliding_window_mask(c["L"] - 1 - seed % 8 * c["L"] // 16, 0)
        else:
            mask = M.sliding_window_mask(c["window"] + seed % 61 * c["block_size"] // 8, c["window"])
        return dict(case=c, mask=mask)
    scale = 1 / math.sqrt(c["d"]) if c["scaled"] else 1.0
    B, N, L, Hq, Hkv, d = (c[k] for k in ("B", "N", "L", "Hq", "Hkv", "d"))
    shapes = [(B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d)]
    if c["api"] == "flex":
        shapes = [(s[0], s[2], s[1], s[3]) for s in shapes]
    qkv = [_randn(s, 8 * seed + i, c["dtype"], scale).requires_grad_(c["grad"]) for i, s in enumerate(shapes)]
    s = dict(case=c, qkv=qkv, dO=_randn(shapes[0], 8 * seed + 3, BF16 if c["bf16_out"] else F32) if c["grad"] else None)
    kw = {}
    if c["api"] == "flex":
        kw["block_mask"] = jm.create_block_mask(M.causal_mask(), 1, 1, N, L, c["block_size"])
        kw["enable_gqa"] = Hq != Hkv
    else:
        if c["block_size"]:
            kw["block_size"] = c["block_size"]
        if c["mask"] == "causal":
            kw["is_causal"] = True
        elif c["mask"] == "lambda_window":
            w = c["window"]
            kw["mask_fn"] = lambda b, h, q, k: (k <= q) & (q - k <= w)
        elif c["mask"] == "tail":
            kw["mask_fn"] = M.sliding_window_mask(L, L - N)
        elif c["mask"] == "sliding":
            kw["mask_fn"] = M.sliding_window_mask(c["window"], c["window"])
            if c["block_size"]:
                kw["window_size"] = (c["window"], c["window"])
        elif c["mask"] == "documents":
            kw["mask_fn"] = M.document_mask(_segments(B, L, seed), causal=True)
    if c["bf16_out"]:
        kw["out_dtype"] = torch.bfloat16
    return dict(s, kw=kw)


def run(state):
    c = state["case"]
    if c["api"] == "block_mask":
        bm = jm.create_block_mask(state["mask"], c["B"], c["Hq"], c["N"], c["L"], c["block_size"])
        return {k: getattr(bm, k) for k in ("kv_num_blocks", "kv_indices", "q_num_blocks", "q_indices", "full_kv_num_blocks",
                                            "full_kv_indices", "full_q_num_blocks", "full_q_indices")}
    call = jm.flex_attention if c["api"] == "flex" else jm.masked_attention_via_map
    O = call(*state["qkv"], **state["kw"])
    if not c["grad"]:
        return O
    return (O.detach(), *torch.autograd.grad(O, state["qkv"], state["dO"]))


def _pairs(c):
    """Allowed (query, key) pairs of one (batch, head)."""
    N, L, w = c["N"], c["L"], c["window"]
    if c["mask"] == "none":
        return N * L
    if c["mask"] == "causal":
        return N * (N + 1) // 2
    if c["mask"] == "tail":
        return N * (L - N) + N * (N + 1) // 2
    q = np.arange(N)
    if c["mask"] == "lambda_window":
        return int((np.minimum(q, w) + 1).sum())
    if c["mask"] == "sliding":
        return int((np.minimum(q + w, L - 1) - np.maximum(q - w, 0) + 1).sum())
    lengths = np.bincount(_segments(1, N, 0)[0]).astype(np.int64)     # one row stands for the others
    return int((lengths * (lengths + 1) // 2).sum())


def work(case):
    c = case
    if c["api"] == "block_mask":
        nq = c["N"] // c["block_size"]
        return {"bytes": 4 * 4 * c["B"] * c["Hq"] * nq * (nq + 1), "flops": 0}
    size, out = (4 if c["dtype"] == F32 else 2), (2 if c["bf16_out"] else 4)
    q, kv = c["B"] * c["N"] * c["Hq"] * c["d"], c["B"] * c["L"] * c["Hkv"] * c["d"]
    nbytes = (q + 2 * kv) * size + q * out
    if c["grad"]:
        nbytes += q * out + (q + 2 * kv) * size
    # Q K^T and P V forward; backward the scores again, dO V^T, and the three gradients
    return {"bytes": nbytes, "flops": 4 * c["d"] * _pairs(c) * c["B"] * c["Hq"] * (3.5 if c["grad"] else 1)}


def tolerance(case):
    if case["api"] == "block_mask":
        return "exact"
    # measured against float64 attention of whole heads of the listed cases, times four.  float32: 2e-7 to 8.5e-7, single
    # values up to 1.7e-5.  bfloat16: 3e-3 (the rounding of the outputs and of P), single values up to 0.11, in the
    # gradients of the longest sequence, whose typical value is small, up to 0.49.
    if case["dtype"] == F32:
        return {"rel": 4e-6, "max": 1e-4}
    return {"rel": 1.2e-2, "max": 0.45 if case["L"] <= 16384 else 0.95}
