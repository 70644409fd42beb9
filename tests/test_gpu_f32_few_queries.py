"""float32, few queries against many keys: the bf16 planes are made only for the kv blocks that a list names.  Against the FP32
tile kernels, with NaN in the keys and values that no query sees and in the memory the planes are written to."""
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat
from jaxmodules_b200 import attention as A
from jaxmodules_b200 import masks as M

pytestmark = pytest.mark.gpu

MASKS = {
    "window": lambda L: dict(mask_fn=M.sliding_window_mask(100, 300)),
    "table": lambda L: dict(mask_fn=lambda b, h, q, k: (k // 128 == 5 + 3 * b + 7 * h) & (k % 3 != q % 3)),
    "documents": lambda L: dict(mask_fn=M.document_mask(torch.tensor([[2], [7]], dtype=torch.int32).repeat(1, 200),
                                                        (torch.arange(L, dtype=torch.int32) // 1000)[None].repeat(2, 1))),
}


@pytest.mark.parametrize("mask", MASKS)
@pytest.mark.parametrize("N,L,Hq,Hkv,d", [(1, 20000, 4, 2, 64), (130, 20001, 4, 2, 128), (16, 33000, 2, 2, 40)])
def test_unlisted_keys(N, L, Hq, Hkv, d, mask):
    """2e-6 of the exact result on each side in the 2-norm (tests/test_gpu_f32.py)."""
    g = torch.Generator("cuda").manual_seed(N)
    q, k, v, dO = (torch.randn(s, device="cuda", generator=g) for s in ((2, N, Hq, d), (2, L, Hkv, d), (2, L, Hkv, d), (2, N, Hq, d)))
    kw = dict(MASKS[mask](L), block_size=N + 1)
    if mask == "window":                      # keys behind the last window, beyond the 64- and 128-blocks it touches
        k[:, (N + 300) // 128 * 128 + 128:] = float("nan")
        v[:, (N + 300) // 128 * 128 + 128:] = float("nan")

    def call(backend):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        torch.full((1 << 28,), float("nan"), device="cuda")      # (freed at once: the planes are allocated from it)
        O = jm.masked_attention_via_map(*leaves, backend=backend, **kw)
        return [O.detach(), *torch.autograd.grad(O, leaves, dO)]

    got, want = call(nat.BMA_BACKEND_AUTO), call(nat.BMA_BACKEND_SIMT)
    assert A.device_status() == 0
    for name, x, y in zip(("O", "dQ", "dK", "dV"), got, want):
        assert torch.isfinite(x).all(), name
        assert (x.double() - y.double()).norm() <= 4e-6 * y.double().norm().clamp(min=1e-3), name
