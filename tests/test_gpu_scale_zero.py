"""A scale of 0: every allowed key weighs the same.  The cut tiles are not done again: the pass runs the kernels of a call with a key bias of 0,
bit for bit, where the FP32 tile functions would sum in another order."""
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import attention as A, masks as M

pytestmark = pytest.mark.gpu

TERMS = {"causal": M.MaskTerms(causal=True), "band": M.MaskTerms(band=(100, 30)), "window": M.MaskTerms(window=(40, 2, 3, 10))}


@pytest.mark.parametrize("mask", TERMS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,d", [(300, 64), (300, 128), (16, 64)])
def test_scale_zero(N, d, dtype, mask):
    L = 400
    g = torch.Generator(device="cuda").manual_seed(N + d)
    q, k, v, do = (torch.randn((1, n, 2, d), device="cuda", generator=g).to(dtype) for n in (N, L, L, N))
    O, lse, ctx = A.attention_forward(q, k, v, TERMS[mask], scale=0.0, need_q_side=True)
    grads = A.attention_backward(q, k, v, O, lse, do.float(), ctx)
    with_bias, lse_bias, _ = A.attention_forward(q, k, v, TERMS[mask], scale=0.0, key_bias=torch.zeros(2, device="cuda"), need_q_side=True)
    assert torch.equal(O, with_bias) and torch.equal(lse, lse_bias)
    i, j = torch.arange(N, device="cuda")[:, None], torch.arange(L, device="cuda")[None]
    start = (i // 40 - 2).clamp(0, 5) * 40
    allowed = {"causal": j <= i, "band": (j >= i - 100) & (j <= i + 30), "window": (j >= start) & (j < start + 200)}[mask]
    p = allowed.double() / allowed.sum(-1, keepdim=True)
    tol = 2e-6 if dtype == torch.float32 else 6e-3      # (as for other scales, tests/test_gpu_f32.py and tests/test_gpu_shared_walks.py)
    want = torch.einsum("nl,blhd->bnhd", p, v.double())
    assert (O.double() - want).norm() <= tol * want.norm()
    assert (lse - allowed.sum(-1).double().log()).abs().max() <= 1e-4
    dv = torch.einsum("nl,bnhd->blhd", p, do.double())
    assert (grads[2].double() - dv).norm() <= tol * dv.norm()
    assert not grads[0].any() and not grads[1].any()     # (dQ and dK carry the scale)
    assert A.device_status() == 0


def test_flex_attention_scale_zero():
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k, v = (torch.randn((1, 2, 200, 64), device="cuda", generator=g) for _ in range(3))
    bm = jm.create_block_mask(M.causal_mask(), 1, 1, 200, 200, 8)
    O = jm.flex_attention(q, k, v, block_mask=bm, scale=0.0)
    O = O[0] if isinstance(O, tuple) else O
    want = v.double().cumsum(2) / torch.arange(1, 201, device="cuda")[:, None]
    assert (O.double() - want).norm() <= 2e-6 * want.norm()
