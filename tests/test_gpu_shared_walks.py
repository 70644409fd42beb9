"""Backward passes of few CTAs, which share a tile's walk out over the CTAs of a cluster and add their accumulators up through distributed
shared memory: against float64, with the dS tiles handed over and without, at ragged ends, with tiles that nobody visits and parts that
get none.

Bounds (2-norm): bfloat16 gradients carry the rounding of P and dS (2^-9 per value, 2e-3 - 3e-3 on normal inputs) and of the result; float32 2e-6 as in
tests/test_gpu_f32.py."""
import math

import numpy as np
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import attention as A, masks as M

pytestmark = pytest.mark.gpu

SEG = np.repeat(np.arange(40, dtype=np.int32), 47)
CASES = [
    # B, N, L, Hq, Hkv, d, mask                       kv tiles x kv heads x B
    (1, 300, 300, 8, 1, 64, "causal"),                # 3: eight parts of 8 - 24 tiles
    (1, 1000, 1000, 8, 1, 128, "causal"),             # 8
    (2, 700, 1300, 4, 2, 128, "none"),                # 44, the keys' last tile ragged
    (1, 1, 260, 2, 1, 64, "none"),                    # a walk of two tiles: parts without any
    (1, 900, 900, 6, 1, 64, "documents"),
    (1, 130, 1500, 3, 1, 128, "first keys"),          # kv tiles that no query visits
    (1, 1300, 1300, 2, 2, 128, "window"),
]


def _mask(mask, B, N, L):
    q, k = torch.arange(N, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    seg = torch.from_numpy(SEG).cuda()
    return {
        "none": lambda: (dict(), torch.ones(N, L, dtype=torch.bool, device="cuda")),
        "causal": lambda: (dict(is_causal=True), k <= q),
        "documents": lambda: (dict(mask_fn=M.document_mask(SEG[None, :N].repeat(B, 0), causal=True)), (k <= q) & (seg[:N, None] == seg[None, :L])),
        "first keys": lambda: (dict(mask_fn=M.sliding_window_mask(L, 3)), k <= q + 3),
        "window": lambda: (dict(mask_fn=M.sliding_window_mask(200, 90)), (k >= q - 200) & (k <= q + 90)),
    }[mask]()


@pytest.mark.parametrize("scratch", [True, False], ids=["hand-over", "recompute"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,mask", CASES, ids=[f"N{c[1]}_L{c[2]}_H{c[3]}_{c[4]}_d{c[5]}_{c[6]}" for c in CASES])
def test_against_float64(B, N, L, Hq, Hkv, d, mask, dtype, scratch):
    if dtype == torch.float32 and not scratch:
        pytest.skip("float32 has no hand-over")
    g = torch.Generator(device="cuda").manual_seed(N + L)
    q, k, v, do = (torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d), (B, N, Hq, d)))
    kw, allowed = _mask(mask, B, N, L)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    limit = A._scratch_limit
    try:
        if not scratch:
            A.set_backward_scratch_limit(0)
        O = jm.masked_attention_via_map(q, k, v, block_size=N + 1, **kw)
        got = torch.autograd.grad(O, (q, k, v), do.float())
    finally:
        A.set_backward_scratch_limit(limit)
    Q, K, V = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    G = Hq // Hkv
    s = torch.einsum("bnhd,blhd->bhnl", Q, K.repeat_interleave(G, 2)) / math.sqrt(d)
    p = torch.softmax(s.masked_fill(~allowed, float("-inf")), -1).nan_to_num(0.0)
    want = torch.autograd.grad(torch.einsum("bhnl,blhd->bnhd", p, V.repeat_interleave(G, 2)), (Q, K, V), do.double())
    tol = 6e-3 if dtype == torch.bfloat16 else 2e-6
    for name, x, w in zip(("dQ", "dK", "dV"), got, want):
        assert (x.double() - w).norm() <= tol * w.norm(), name
    assert A.device_status() == 0


def test_key_bias():
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn((1, n, h, 64), device="cuda", generator=g).bfloat16() for n, h in ((400, 4), (500, 1), (500, 1), (400, 4)))
    bias = torch.tensor([0.01, -0.02, 0.0, 0.03], device="cuda")
    terms = M.MaskTerms(causal=True, q_offset=100)
    O, lse, ctx = A.attention_forward(q, k, v, terms, need_q_side=True, key_bias=bias)
    got = A.attention_backward(q, k, v, O, lse, do, ctx)
    Q, K, V = (t.double().requires_grad_(True) for t in (q, k, v))
    i, j = torch.arange(400, device="cuda")[:, None] + 100, torch.arange(500, device="cuda")[None]
    s = torch.einsum("bnhd,blhd->bhnl", Q, K.repeat_interleave(4, 2)) / 8 + bias.double()[None, :, None, None] * j
    p = torch.softmax(s.masked_fill(j > i, float("-inf")), -1)
    want = torch.autograd.grad(torch.einsum("bhnl,blhd->bnhd", p, V.repeat_interleave(4, 2)), (Q, K, V), do.double())
    for name, x, w in zip(("dQ", "dK", "dV"), got, want):
        assert (x.double() - w).norm() <= 6e-3 * w.norm(), name
