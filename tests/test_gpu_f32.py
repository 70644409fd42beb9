"""The float32 tensor-core kernels (three bf16 planes per operand) at the edges of their tiles, against the float64 oracle.

Bound: an FP32 evaluation carries the rounding of the scores (2^-24 per term, |s| of a few), of ex2 (2^-22) and of the
sums; the FP32 tile kernels show up to 9e-7 in the 2-norm on these shapes, so 2e-6 leaves both a factor of two and is far
below the 2^-17 that a lost low plane would cost."""
import numpy as np
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import masks as M
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu

SEG = np.repeat(np.arange(9, dtype=np.int32), 45)[None, :].repeat(2, 0)
CASES = [
    # B, N, L, Hq, Hkv, d, kwargs; lengths around the 64- and 128-wide tiles, head dimensions around the padded widths
    (1, 1, 1, 1, 1, 1, {}),
    (1, 63, 64, 2, 1, 64, dict(block_size=10)),
    (1, 65, 65, 2, 2, 63, dict(is_causal=True)),
    (2, 128, 128, 2, 1, 64, dict(is_causal=True)),
    (1, 129, 193, 3, 1, 32, dict(block_size=10)),
    (2, 257, 257, 4, 2, 65, dict(is_causal=True)),
    (1, 320, 320, 2, 2, 128, dict(mask_fn=M.sliding_window_mask(70, 3))),
    (1, 320, 320, 2, 2, 64, dict(mask_fn=M.sliding_window_mask(70, 3), block_size=64, window_size=(64, 0))),
    (2, 400, 400, 2, 1, 48, dict(mask_fn=M.document_mask(SEG[:, :400], causal=True))),
    (1, 384, 384, 4, 2, 64, dict(mask_fn=lambda b, h, q, k: (q + k + h) % 3 != 0)),
    (1, 200, 130, 1, 1, 64, dict(mask_fn=M.sliding_window_mask(20, 0), block_size=30)),   # the last queries see no key
]


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,kw", CASES, ids=[f"N{c[1]}_L{c[2]}_d{c[5]}" for c in CASES])
def test_f32_tensor_core(B, N, L, Hq, Hkv, d, kw):
    g = torch.Generator().manual_seed(N * 131 + d)
    Q, K, V, dO = (torch.randn(s, generator=g) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d), (B, N, Hq, d)))
    q, k, v = (t.cuda().requires_grad_(True) for t in (Q, K, V))
    O, lse = jm.masked_attention_via_map(q, k, v, return_lse=True, **kw)
    grads = torch.autograd.grad(O, (q, k, v), dO.cuda())
    ref = ao.masked_attention_dense(Q.numpy(), K.numpy(), V.numpy(), dO=dO.numpy(), **kw)
    for name, got in zip(("O", "dQ", "dK", "dV"), (O, *grads)):
        want = torch.from_numpy(np.asarray(ref[name], dtype=np.float64))
        err = (got.detach().cpu().double() - want).norm() / want.norm().clamp(min=1e-3)
        assert err <= 2e-6, (name, float(err))
    want = torch.from_numpy(np.asarray(ref["lse"], dtype=np.float64))
    got = lse.cpu().double()
    dead = torch.isinf(want)
    assert torch.equal(torch.isinf(got), dead) and (got - want)[~dead].abs().max() <= 4e-6
