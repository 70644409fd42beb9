"""Compiled variants and input layouts of the float32 tensor-core kernels and of the split forward (few queries) that the other
tests do not reach: per-head key bias, negative scale, misaligned and expanded tensors, a K / V cache with heads outermost,
a workspace that is too small; and that outputs repeat bit for bit."""
import ctypes as C
import math

import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat
from jaxmodules_b200 import attention as A
from jaxmodules_b200 import masks as M
from jaxmodules_b200.block_mask import compile_block_lists

pytestmark = pytest.mark.gpu


def _randn(*shape, seed=0, dtype=torch.float32):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


def _reference(q, k, v, scale, bias=None, allowed=None):
    """float64 attention of [B, N, Hq, d] with per-head key bias; ``allowed`` bool [N, L]."""
    G = q.shape[2] // k.shape[2]
    q, k, v = q.double(), k.double().repeat_interleave(G, 2), v.double().repeat_interleave(G, 2)
    s = torch.einsum("bnhd,blhd->bhnl", q, k) * scale
    if bias is not None:
        s = s + bias.double()[None, :, None, None] * torch.arange(k.shape[1], device=s.device)
    if allowed is not None:
        s = s.masked_fill(~allowed, float("-inf"))
    return torch.einsum("bhnl,blhd->bnhd", torch.softmax(s, -1), v), torch.logsumexp(s, -1)


# ---- float32 -----------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("d", [17, 32, 64, 128])
def test_f32_key_bias(d):
    """Forward and both backward kernels with another bias for every head of a group.  2-norm bound of every float32 call, with
    a factor of four for the scores: the bias adds up to 300 * 0.05 * 4 = 60 to them, so their float32 rounding is 2^-24 * 60 =
    4e-6 of a probability at the most, where without a bias |s| is about 4."""
    N, Hq, Hkv = 300, 4, 2
    q, k, v, dO = (_randn(2, N, h, d, seed=i) for i, h in enumerate((Hq, Hkv, Hkv, Hq)))
    bias = 0.05 * torch.tensor([1.0, -2.0, 3.0, 4.0], device="cuda")
    O, lse, ctx = A.attention_forward(q, k, v, M.MaskTerms(causal=True), need_q_side=True, key_bias=bias)
    grads = A.attention_backward(q, k, v, O, lse, dO, ctx)
    assert A.device_status() == 0
    leaves = [t.double().requires_grad_(True) for t in (q, k, v)]
    want, _ = _reference(*leaves, 1 / math.sqrt(d), bias, torch.ones(N, N, dtype=torch.bool, device="cuda").tril())
    for name, x, y in zip(("O", "dQ", "dK", "dV"), (O, *grads), (want, *torch.autograd.grad(want, leaves, dO.double()))):
        assert (x.double() - y).norm() <= 8e-6 * y.norm(), name


def _offset_view(t, extra):
    """The same values at an odd element offset, ``extra`` unused values after every row."""
    B, L, H, d = t.shape
    buf = torch.zeros(B * L * H * (d + extra) + 1, device=t.device)
    view = buf[1:].view(B, L, H, d + extra)[..., :d]
    view.copy_(t)
    return view


@pytest.mark.parametrize("d", [30, 64, 100])
@pytest.mark.parametrize("layout", ["odd_base", "odd_stride", "expanded_batch", "expanded_heads"])
def test_f32_layouts(d, layout):
    """Against the same values in plain contiguous tensors: O and dV bit for bit (the planes do not depend on how they were read);
    delta = rowsum(dO * O) is added up in another order for such a dO, and with it dQ and dK (2e-6 each, tests/test_gpu_f32.py)."""
    N, Hq, Hkv = 150, 4, 2
    q, k, v, dO = (_randn(2, N, h, d, seed=i) for i, h in enumerate((Hq, Hkv, Hkv, Hq)))
    if layout == "expanded_batch":
        dO = dO[:1].expand(2, -1, -1, -1)
    elif layout == "expanded_heads":
        dO, k = dO[:, :, :1].expand(-1, -1, Hq, -1), k[:, :, :1].expand(-1, -1, Hkv, -1)
    odd = {"odd_base": 0, "odd_stride": 3}.get(layout)

    def call(change):
        leaves = [change(t).detach().requires_grad_(True) for t in (q, k, v)]
        O = jm.masked_attention_via_map(*leaves, is_causal=True)
        return [O.detach(), *torch.autograd.grad(O, leaves, change(dO))]

    got = call((lambda t: _offset_view(t, odd)) if odd is not None else (lambda t: t))
    want = call(lambda t: t.contiguous())
    assert A.device_status() == 0
    for name, x, y in zip(("O", "dQ", "dK", "dV"), got, want):
        assert torch.equal(x, y) if name in ("O", "dV") else (x - y).norm() <= 4e-6 * y.norm(), name


@pytest.mark.parametrize("d", [64, 128])
def test_f32_repeats(d):
    """The plane products add 64- and 128-column MMAs up in the same accumulator columns, in the order they are issued.  Executed
    in any other order, the first of them (which overwrites) would drop a product: far from the result, and not the same twice."""
    q, k, v, dO = (_randn(2, 1024, 8, d, seed=i) for i in range(4))
    first = None
    for _ in range(40):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        O = jm.masked_attention_via_map(*leaves, is_causal=True)
        out = [O.detach(), *torch.autograd.grad(O, leaves, dO)]
        first = first or out
        assert all(torch.equal(x, y) for x, y in zip(out, first))
    want, _ = _reference(q, k, v, 1 / math.sqrt(d), None, torch.ones(1024, 1024, dtype=torch.bool, device="cuda").tril())
    assert (first[0].double() - want).norm() <= 2e-6 * want.norm()


# ---- few queries, bfloat16 -----------------------------------------------------------------------------------------------------
FEW = [(1, 3, 700, 8, 2, 128), (2, 16, 1500, 8, 2, 64), (1, 30, 400, 4, 4, 128), (1, 128, 300, 2, 2, 64)]   # packed and not


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d", FEW)
@pytest.mark.parametrize("variant", ["bias", "negative_scale", "both"])
def test_few_queries_bias_and_scale(B, N, L, Hq, Hkv, d, variant):
    """The bounds of tests/test_gpu_few_queries.py; the bias of a head moves its weight along the keys."""
    q, k, v = (_randn(B, n, h, d, seed=i, dtype=torch.bfloat16) for i, (n, h) in enumerate(((N, Hq), (L, Hkv), (L, Hkv))))
    scale = (-1 if variant != "bias" else 1) / math.sqrt(d)
    bias = None if variant == "negative_scale" else torch.linspace(-0.04, 0.05, Hq, device="cuda")
    O, lse, _ = A.attention_forward(q, k, v, M.MaskTerms(band=(1 << 20, L - N)), scale=scale, key_bias=bias)
    assert A.device_status() == 0
    i, j = torch.arange(N, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    want, wlse = _reference(q, k, v, scale, bias, j <= i + L - N)
    err = (O.double() - want).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3 and (lse.double() - wlse).abs().max() <= 1e-3


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d", FEW)
def test_few_queries_heads_outermost(B, N, L, Hq, Hkv, d):
    """K and V as a cache [B, H, L, d] seen as [B, L, H, d], and Q as a slice of a fused projection: bit for bit."""
    q, k, v = (_randn(B, n, h, d, seed=i, dtype=torch.bfloat16) for i, (n, h) in enumerate(((N, Hq), (L, Hkv), (L, Hkv))))
    out = lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)
    qkv = torch.cat([q, torch.full_like(q, float("nan"))], dim=2)
    kw = dict(mask_fn=M.sliding_window_mask(L, L - N), block_size=N + 1, out_dtype=torch.bfloat16)
    assert torch.equal(jm.masked_attention_via_map(qkv[:, :, :Hq], out(k), out(v), **kw), jm.masked_attention_via_map(q, k, v, **kw))


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d", FEW)
def test_few_queries_small_workspace(B, N, L, Hq, Hkv, d):
    """``bma_attn_fwd_ws`` with less workspace than it asks for (none, one byte less, misaligned) runs as ``bma_attn_fwd`` does."""
    q, k, v = (_randn(B, n, h, d, seed=i, dtype=torch.bfloat16) for i, (n, h) in enumerate(((N, Hq), (L, Hkv), (L, Hkv))))
    a = A._make_args(q, k, v)
    dmask = M.to_device_mask(M.MaskTerms(), N, L, q.device)
    lists, keep = compile_block_lists(dmask, B, Hq, N, L, 128, 128, q.device, q_side=False, conservative=True)
    lib, st = nat.lib(), torch.cuda.current_stream().cuda_stream
    need = lib.bma_attn_fwd_workspace_bytes(C.byref(a), C.byref(lists))
    ws = torch.empty(max(need, 16) + 16, dtype=torch.uint8, device="cuda")
    results = []
    for ptr, nbytes in ((ws.data_ptr(), need), (None, 0), (ws.data_ptr(), max(need - 1, 0)), (ws.data_ptr() + 8, need)):
        O = torch.empty((B, N, Hq, d), dtype=torch.float32, device="cuda")
        lse = torch.empty((B, Hq, N), dtype=torch.float32, device="cuda")
        a.o, a.lse = A._tensor(O), lse.data_ptr()
        assert lib.bma_attn_fwd_ws(C.byref(a), C.byref(dmask.spec), C.byref(lists), ptr, nbytes, st) == nat.BMA_OK
        results.append((O, lse))
    assert A.device_status() == 0
    want, wlse = _reference(q, k, v, 1 / math.sqrt(d))
    for O, lse in results:
        err = (O.double() - want).abs()
        assert err.max() <= 2e-2 and err.mean() <= 2e-3 and (lse.double() - wlse).abs().max() <= 1e-3
    assert all(torch.equal(results[1][0], r[0]) for r in results[2:])
