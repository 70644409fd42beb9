"""The float32 backward pass that takes delta and writes its block lists in the launch of the planes, against the same pass with
``bma_attn_bwd_preprocess`` before it and compiled lists: bit for bit, for every kind of interval mask, for head dimensions and strides that
the shared launch takes and for those it leaves to the launch of its own."""
import pytest
import torch

from jaxmodules_b200 import attention as A, masks as M
from jaxmodules_b200.block_mask import compile_block_lists

pytestmark = pytest.mark.gpu

TERMS = {
    "none": M.MaskTerms(),
    "causal": M.MaskTerms(causal=True),
    "band": M.MaskTerms(band=(70, 200)),
    "window": M.MaskTerms(window=(128, 1, 2, 6)),
    "window that changes inside tiles": M.MaskTerms(window=(24, 5, 9, 42)),
    "offset": M.MaskTerms(causal=True, q_offset=64, k_offset=32),
    "nothing": M.MaskTerms(causal=True, k_offset=1 << 20),
}


@pytest.mark.parametrize("mask", TERMS)
@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,shift", [(2, 300, 300, 4, 2, 64, 0), (1, 129, 700, 2, 1, 128, 0), (1, 200, 130, 3, 3, 33, 0), (1, 150, 150, 2, 2, 40, 1),
                                                   (1, 5, 9000, 4, 4, 128, 0)])
@pytest.mark.parametrize("cotangent", [torch.float32, torch.bfloat16])
def test_one_launch(B, N, L, Hq, Hkv, d, shift, cotangent, mask):
    g = torch.Generator(device="cuda").manual_seed(N + L)
    q, k, v = (torch.randn(s, device="cuda", generator=g) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d)))
    flat = torch.randn(B * N * Hq * d + shift, device="cuda", generator=g).to(cotangent)
    dO = flat[shift:].view(B, N, Hq, d)          # `shift` values off a 16-byte boundary
    terms = TERMS[mask]
    O, lse, ctx = A.attention_forward(q, k, v, terms, need_q_side=True, out_dtype=cotangent)
    assert ctx["list_tensors"] is None
    got = A.attention_backward(q, k, v, O, lse, dO, ctx)
    lists, keep = compile_block_lists(M.to_device_mask(terms, N, L, q.device), B, Hq, N, L, 128, 128, q.device, q_side=True, conservative=True)
    want = A.attention_backward(q, k, v, O, lse, dO, dict(ctx, lists=lists, list_tensors=keep, lists_have_q_side=True, reuse={}))
    for name, x, y in zip(("dQ", "dK", "dV"), got, want):
        assert torch.equal(x, y), name
    assert A.device_status() == 0
