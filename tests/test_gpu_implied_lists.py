"""Forward passes without block lists (masks of interval terms, whose blocks the kernels know from the indices) against the same passes
over compiled lists: bit for bit, in every kernel that takes them, at edges of tiles and with windows that cut tiles.
And the runs of a few-query call, which meet in the shared memory of a cluster: against float64."""
import ctypes as C
import math

import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat, attention as A, masks as M
from jaxmodules_b200.block_mask import compile_block_lists

pytestmark = pytest.mark.gpu

TERMS = {
    "none": lambda N, L: M.MaskTerms(),
    "causal": lambda N, L: M.MaskTerms(causal=True),
    "tail": lambda N, L: M.MaskTerms(band=(L, max(L - N, 0))),
    "band": lambda N, L: M.MaskTerms(band=(70, 3)),
    "wide band": lambda N, L: M.MaskTerms(causal=True, band=(1500, 0)),
    "window": lambda N, L: M.MaskTerms(window=(100, 1, 2, -(-max(N, L) // 100))),        # its blocks change inside the tiles
    "offset": lambda N, L: M.MaskTerms(causal=True, q_offset=64, k_offset=32),
    "nothing": lambda N, L: M.MaskTerms(causal=True, k_offset=1 << 20),
}
SHAPES = [
    # dtype, B, N, L, Hq, Hkv, d                         kernel
    (torch.bfloat16, 2, 300, 300, 4, 2, 128),            # one CTA per pair of query tiles
    (torch.bfloat16, 1, 513, 900, 2, 2, 64),
    (torch.bfloat16, 2, 16, 1500, 4, 2, 128),            # few queries: runs of keys
    (torch.bfloat16, 1, 128, 300, 2, 1, 64),
    (torch.float32, 2, 300, 300, 4, 2, 64),
    (torch.float32, 1, 129, 700, 2, 1, 128),
    (torch.float32, 1, 5, 9000, 4, 4, 128),              # few queries: planes of listed blocks only
]


def _both(q, k, v, terms, **kw):
    """(O, lse) without lists, and over compiled ones."""
    def lists_fn(tq, tk, q_side):
        dmask = M.to_device_mask(terms, q.shape[1], k.shape[1], q.device)
        return compile_block_lists(dmask, q.shape[0], q.shape[2], q.shape[1], k.shape[1], tq, tk, q.device, q_side=q_side, conservative=True)
    without = A.attention_forward(q, k, v, terms, **kw)
    over = A.attention_forward(q, k, v, terms, lists_fn=lists_fn, **kw)
    return without, over


@pytest.mark.parametrize("mask", TERMS)
@pytest.mark.parametrize("dtype,B,N,L,Hq,Hkv,d", SHAPES, ids=[f"{str(s[0])[6:]}_N{s[2]}_L{s[3]}_d{s[6]}" for s in SHAPES])
def test_against_compiled_lists(dtype, B, N, L, Hq, Hkv, d, mask):
    g = torch.Generator(device="cuda").manual_seed(N + L)
    q, k, v = (torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d)))
    terms = TERMS[mask](N, L)
    without, over = _both(q, k, v, terms)
    spec = M.to_device_mask(terms, N, L, q.device).spec
    implied = nat.host().implies_lists(q, k, v, None, None, nat.BMA_BACKEND_AUTO, C.addressof(spec))
    assert (without[2]["list_tensors"] is None) == bool(implied)
    # few keys per row are left to the persistent kernel, which wants lists
    assert implied or (dtype == torch.bfloat16 and N > 128 and mask in ("band", "window", "tail"))
    assert torch.equal(without[0], over[0]) and torch.equal(without[1], over[1])
    assert A.device_status() == 0


@pytest.mark.parametrize("room", [True, False], ids=["redone", "no planes"])
def test_float32_tiles(monkeypatch, room):
    """The FP32 tile functions walk the same blocks: where results are not finite, and where there is no room for planes.  (Their order of
    blocks differs without lists, so sums do: two evaluations within 2e-6 each of the exact value.)"""
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn((1, 300, 2, 64), device="cuda", generator=g) for _ in range(3))
    if room:
        v[0, 10, 0, 3] = float("inf")
    else:
        monkeypatch.setattr(A, "_F32_PLANES_LIMIT", 0)
    (a, la, _), (b, lb, _) = _both(q, k, v, TERMS["causal"](300, 300))
    assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and torch.isfinite(a).any()
    fin = torch.isfinite(a)
    assert (a[fin].double() - b[fin].double()).norm() <= 4e-6 * b[fin].double().norm() and (la - lb).abs().max() <= 1e-5


@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,N,L,Hq,Hkv,d", [(4, 16, 8192, 32, 8, 128), (8, 1, 4000, 16, 4, 64), (3, 127, 2000, 11, 11, 128), (2, 3, 1100, 5, 1, 64)])
def test_runs_meet_in_a_cluster(B, N, L, Hq, Hkv, d, out):
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d)))
    q[0, 0] *= 8                      # one row whose runs have far apart maxima
    O, lse = jm.masked_attention_via_map(q, k, v, mask_fn=M.sliding_window_mask(L, L - N), block_size=N + 1, out_dtype=out, return_lse=True)
    kk, vv = (t.double().repeat_interleave(Hq // Hkv, 2) for t in (k, v))
    s = torch.einsum("bnhd,blhd->bhnl", q.double(), kk) / math.sqrt(d)
    i, j = torch.arange(N, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    s.masked_fill_(j > i + L - N, float("-inf"))
    want = torch.einsum("bhnl,blhd->bnhd", torch.softmax(s, -1), vv)
    # bfloat16 operands of P V: 2^-9 of each probability, as in every bfloat16 forward pass
    assert (O.double() - want).norm() <= 4e-3 * want.norm() and (lse.double() - torch.logsumexp(s, -1)).abs().max() <= 1e-3
    assert A.device_status() == 0
