"""That the CTAs of a cluster do share walks and runs where the tests of tests/test_gpu_shared_walks.py, tests/test_gpu_f32_shared_rows.py and
tests/test_gpu_implied_lists.py mean them to (bma_cluster_launch_count), and the kernels with a key bias and with results that are not finite
while they share."""
import ctypes as C
import math

import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat, attention as A, masks as M

import test_gpu_f32_shared_rows as rows
import test_gpu_shared_walks as walks

pytestmark = pytest.mark.gpu


def launches(call):
    """(result, launches, sizes of the clusters launched) of a call."""
    lib = nat.lib()
    count = lambda: [lib.bma_launch_count()] + [lib.bma_cluster_launch_count(n) for n in range(2, 9)]
    before = count()
    out = call()
    n, *clusters = (y - x for x, y in zip(before, count()))
    return out, n, [size for size, k in enumerate(clusters, 2) for _ in range(k)]


def _inputs(B, N, L, Hq, Hkv, d, dtype=torch.float32):
    g = torch.Generator(device="cuda").manual_seed(N + L)
    return [torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d), (B, N, Hq, d))]


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,mask", rows.CASES, ids=[f"N{c[1]}_L{c[2]}_H{c[3]}_d{c[5]}_{c[6]}" for c in rows.CASES])
def test_float32_forward(B, N, L, Hq, Hkv, d, mask):
    q, k, v, _ = _inputs(B, N, L, Hq, Hkv, d)
    _, n, clusters = launches(lambda: jm.masked_attention_via_map(q, k, v, mask_fn=rows.MASKS[mask][0], block_size=N + 1))
    last = (N, Hq) == (1500, 16)                        # whole waves of tiles, and the last ones in a launch of their own
    assert len(clusters) == 1 and n == 2 + last         # (the planes are a launch)
    if N == 1:
        assert clusters == [8]                          # a single tile


@pytest.mark.parametrize("scratch", [True, False], ids=["hand-over", "recompute"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,mask", walks.CASES, ids=[f"N{c[1]}_L{c[2]}_H{c[3]}_{c[4]}_d{c[5]}_{c[6]}" for c in walks.CASES])
def test_backward(B, N, L, Hq, Hkv, d, mask, dtype, scratch):
    q, k, v, do = _inputs(B, N, L, Hq, Hkv, d, dtype)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    O = jm.masked_attention_via_map(q, k, v, block_size=N + 1, **walks._mask(mask, B, N, L)[0])
    limit = A._scratch_limit
    try:
        if not scratch:
            A.set_backward_scratch_limit(0)
        _, _, clusters = launches(lambda: torch.autograd.grad(O, (q, k, v), do.float()))
    finally:
        A.set_backward_scratch_limit(limit)
    assert len(clusters) == (2 if dtype == torch.float32 else 1)      # float32: dK / dV and dQ; bfloat16: dK / dV


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,clusters", [(4, 16, 8192, 32, 8, 128, 1), (8, 1, 4000, 16, 4, 64, 1), (3, 127, 2000, 11, 11, 128, 1), (2, 3, 1100, 5, 1, 64, 1),
                                                     (2, 27, 18680, 42, 42, 64, 0)])
def test_few_queries(B, N, L, Hq, Hkv, d, clusters):
    """Up to eight runs meet in a cluster, in one launch, where that makes no more waves; else in the workspace, in two."""
    q, k, v, _ = _inputs(B, N, L, Hq, Hkv, d, torch.bfloat16)
    _, n, sizes = launches(lambda: jm.masked_attention_via_map(q, k, v, block_size=N + 1))
    assert len(sizes) == clusters and n == 2 - clusters
    args, lists = A._make_args(q, k, v), nat.BlockLists(1, 1, 1, -(-L // 128), 128, 128)
    assert nat.lib().bma_attn_fwd_uses_workspace(C.byref(args), C.byref(lists)) == 1 - clusters      # (and none is allocated where it is not)


@pytest.mark.parametrize("dtype,d", [(torch.float32, 64), (torch.float32, 128), (torch.bfloat16, 64), (torch.bfloat16, 128)])
def test_key_bias(dtype, d):
    N, L, H = 300, 500, 4
    q, k, v, do = _inputs(1, N, L, H, 1, d, dtype)
    bias = torch.tensor([0.01, -0.02, 0.0, 0.03], device="cuda")
    terms = M.MaskTerms(causal=True, q_offset=200)
    O, lse, ctx = A.attention_forward(q, k, v, terms, need_q_side=True, key_bias=bias)
    got, _, clusters = launches(lambda: A.attention_backward(q, k, v, O, lse, do, ctx))
    assert len(clusters) == (2 if dtype == torch.float32 else 1)
    Q, K, V = (t.double().requires_grad_(True) for t in (q, k, v))
    i, j = torch.arange(N, device="cuda")[:, None] + 200, torch.arange(L, device="cuda")[None]
    s = torch.einsum("bnhd,blhd->bhnl", Q, K.repeat_interleave(H, 2)) / math.sqrt(d) + bias.double()[None, :, None, None] * j
    p = torch.softmax(s.masked_fill(j > i, float("-inf")), -1)
    want = torch.autograd.grad(torch.einsum("bhnl,blhd->bnhd", p, V.repeat_interleave(H, 2)), (Q, K, V), do.double())
    tol = 6e-3 if dtype == torch.bfloat16 else 2e-6      # (tests/test_gpu_shared_walks.py)
    for name, x, w in zip(("dQ", "dK", "dV"), got, want):
        assert (x.double() - w).norm() <= tol * w.norm(), name


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("operand", ["v", "k", "do"])
@pytest.mark.parametrize("d", [64, 128])
def test_not_finite_while_shared(d, operand, value):
    """One value that is not finite, in the part of a walk that one CTA of a cluster takes: the results of the FP32 tile kernels, as in
    tests/test_gpu_f32_nonfinite.py."""
    q, k, v, do = _inputs(1, 900, 900, 4, 1, d)
    {"v": v, "k": k, "do": do}[operand][0, 700, 0, 3] = value
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))

    def call(backend):
        O = jm.masked_attention_via_map(q, k, v, mask_fn=M.sliding_window_mask(300, 0), backend=backend)
        grads, _, clusters = launches(lambda: torch.autograd.grad(O, (q, k, v), do))
        return [O.detach(), *grads], clusters

    (got, clusters), (want, none) = call(nat.BMA_BACKEND_AUTO), call(nat.BMA_BACKEND_SIMT)
    assert len(clusters) == 2 and none == []
    for name, x, w in zip(("O", "dQ", "dK", "dV"), got, want):
        assert torch.equal(torch.isnan(x), torch.isnan(w)), name
        inf = torch.isinf(w)
        assert torch.equal(torch.isinf(x), inf) and torch.equal(x[inf], w[inf]), name
        fin = torch.isfinite(w)
        assert fin.any() and (x[fin].double() - w[fin].double()).abs().max() <= 2e-5 * max(1.0, float(w[fin].abs().max())), name


def _sizes(dtype, N, H, d, **kw):
    q, k, v, do = _inputs(1, N, N, H, H, d, dtype)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    return launches(lambda: torch.autograd.grad(jm.masked_attention_via_map(q, k, v, **kw), (q, k, v), do.float()))[2]


def test_windows_make_walks_short():
    """512 tiles whose walks a block window keeps to six tiles: no more to share than with a band (the last of the forward's four waves at most)."""
    window = _sizes(torch.float32, 16384, 4, 64, block_size=64, window_size=(256, 256))
    assert window == _sizes(torch.float32, 16384, 4, 64, mask_fn=M.sliding_window_mask(256, 256)) and len(window) <= 1


def test_walks_of_unknown_length():
    """Documents may make walks short: no more CTAs share one than run at once."""
    ids = torch.arange(4096, dtype=torch.int32)[None] // 300
    sizes = _sizes(torch.float32, 4096, 1, 64, mask_fn=M.document_mask(ids.numpy(), causal=True))
    assert len(sizes) == 3 and max(sizes) * 32 <= 148        # (forward, dK / dV and dQ of 32 tiles each)
    ids = torch.arange(1500, dtype=torch.int32)[None] // 128
    q, k, v, _ = _inputs(1, 1500, 1500, 16, 4, 128)
    _, n, clusters = launches(lambda: jm.masked_attention_via_map(q, k, v, mask_fn=M.document_mask(ids.numpy())))
    assert clusters == []                                    # the last tiles have no launch of their own


SCRATCH = {
    "causal": lambda B, N: dict(is_causal=True),
    "documents": lambda B, N: dict(mask_fn=M.document_mask((torch.arange(N, dtype=torch.int32) // 130)[None].repeat(B, 1).numpy(), causal=True)),
    "table": lambda B, N: dict(mask_fn=lambda b, h, q, k: (k <= q) & (q - k < 200) & ((q + k) % 7 != 0)),
    "window": lambda B, N: dict(block_size=50, window_size=(100, 50)),
}


@pytest.mark.parametrize("mask", SCRATCH)
@pytest.mark.parametrize("B,N,Hq,Hkv,d", [(3, 700, 8, 2, 64), (2, 500, 12, 4, 128), (4, 300, 16, 1, 128)])
def test_scratch_does_not_change_the_sums(B, N, Hq, Hkv, d, mask):
    """The CTAs that share a walk are chosen for the whole call: with all dS tiles handed over, in ranges of heads through a small buffer and without
    the hand-over dK and dV are the same bits, and so is dQ where it is read from the same tiles."""
    q, k, v, do = _inputs(B, N, N, Hq, Hkv, d, torch.bfloat16)
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    limit, grads, kernels = A._scratch_limit, [], []
    try:
        for share in ((limit, 1.0), (limit, 0.5), (0, 1.0)):
            A.set_backward_scratch_limit(*share)
            O = jm.masked_attention_via_map(q, k, v, **SCRATCH[mask](B, N))
            g, _, clusters = launches(lambda: torch.autograd.grad(O, (q, k, v), do.float()))
            grads.append(g)
            kernels.append(clusters)
    finally:
        A.set_backward_scratch_limit(limit)
    whole, ranges, recomputed = kernels
    assert len(whole) == 1 and recomputed == whole and len(ranges) > 1 and set(ranges) == set(whole)
    for name, x, y, z in zip(("dQ", "dK", "dV"), *grads):
        assert torch.equal(x, y), name
        assert name == "dQ" or torch.equal(x, z), name
