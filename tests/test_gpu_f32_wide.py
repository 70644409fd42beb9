"""The float32 tensor-core backward for head dimensions 65 - 128 at the edges of its tiles, against the float64 oracle.

Bound as for the narrower heads (tests/test_gpu_f32.py): 2e-6 in the 2-norm, a factor of two above what an FP32 evaluation
shows on such shapes and far below the 2^-17 that a lost low plane would cost."""
import numpy as np
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import attention as A
from jaxmodules_b200 import masks as M
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu

SEG = np.repeat(np.arange(9, dtype=np.int32), 45)[None, :].repeat(2, 0)
CASES = [
    # B, N, L, Hq, Hkv, d, kwargs: one to three 64-wide half tiles around the ring of three boxes, then longer walks
    # (two keys at least: with one, P = 1 and dS = dP - delta is zero but for its rounding, and dQ and dK have no relative error)
    (1, 1, 2, 1, 1, 128, dict(block_size=10)),
    (1, 64, 64, 1, 1, 65, {}),
    (1, 65, 63, 2, 1, 128, dict(block_size=10)),
    (2, 128, 129, 2, 2, 100, dict(block_size=10)),
    (1, 193, 193, 4, 1, 128, dict(is_causal=True)),
    (2, 520, 520, 4, 2, 96, dict(is_causal=True)),
    (1, 320, 320, 2, 2, 128, dict(mask_fn=M.sliding_window_mask(70, 3), block_size=64, window_size=(64, 0))),
    (2, 400, 400, 2, 1, 128, dict(mask_fn=M.document_mask(SEG[:, :400], causal=True))),
    (1, 384, 384, 4, 2, 72, dict(mask_fn=lambda b, h, q, k: (q + k + h) % 3 != 0)),
    (1, 200, 130, 1, 1, 128, dict(mask_fn=M.sliding_window_mask(20, 0), block_size=30)),   # the last queries see no key
    (1, 40, 400, 1, 1, 128, dict(mask_fn=M.sliding_window_mask(400, 0), block_size=41)),   # the last key tiles see no query
]


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,kw", CASES, ids=[f"N{c[1]}_L{c[2]}_d{c[5]}" for c in CASES])
def test_f32_wide_backward(B, N, L, Hq, Hkv, d, kw):
    g = torch.Generator().manual_seed(N * 131 + d)
    Q, K, V, dO = (torch.randn(s, generator=g) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d), (B, N, Hq, d)))
    # inputs and cotangent in other strides than the outputs': heads outermost
    q, k, v = (t.cuda().transpose(1, 2).contiguous().transpose(1, 2).requires_grad_(True) for t in (Q, K, V))
    O = jm.masked_attention_via_map(q, k, v, **kw)
    grads = torch.autograd.grad(O, (q, k, v), dO.cuda())
    assert A.device_status() == 0
    ref = ao.masked_attention_dense(Q.numpy(), K.numpy(), V.numpy(), dO=dO.numpy(), **kw)
    for name, got in zip(("dQ", "dK", "dV"), grads):
        want = torch.from_numpy(np.asarray(ref[name], dtype=np.float64))
        err = (got.cpu().double() - want).norm() / want.norm().clamp(min=1e-3)
        assert err <= 2e-6, (name, float(err))


@pytest.mark.parametrize("d", [72, 128])
def test_f32_wide_key_bias(d):
    """A per-head key bias (ALiBi) through flex_attention's [B, H, L, E] strides, against the FP32 tile kernels: each side
    within 2e-6 of the exact gradients, so 4e-6 between them."""
    from jaxmodules_b200 import _native as nat
    from jaxmodules_b200.flex import flex_attention
    g = torch.Generator().manual_seed(d)
    q, k, v, dO = (torch.randn(2, h, 300, d, generator=g).cuda() for h in (4, 2, 2, 4))
    bm = jm.create_block_mask(M.causal_mask(), 1, 1, 300, 300, 100)
    grads = []
    for backend in (nat.BMA_BACKEND_AUTO, nat.BMA_BACKEND_SIMT):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        O = flex_attention(*leaves, score_mod=lambda s, b, h, i, j: s + 0.05 * (h + 1) * (j - i), block_mask=bm, enable_gqa=True, backend=backend)
        grads.append(torch.autograd.grad(O, leaves, dO))
    assert A.device_status() == 0
    for name, x, y in zip(("dQ", "dK", "dV"), *grads):
        err = (x.double() - y.double()).norm() / y.double().norm()
        assert err <= 4e-6, (name, float(err))
