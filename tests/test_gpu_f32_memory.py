"""float32 attention where the workspace of the tensor-core kernels is not to be had: the FP32 tile kernels walk the same lists."""
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat, attention as A
from jaxmodules_b200 import masks as M

pytestmark = pytest.mark.gpu


def _inputs(N, L, d):
    g = torch.Generator().manual_seed(N + d)
    return [torch.randn(s, generator=g).cuda() for s in ((2, N, 4, d), (2, L, 2, d), (2, L, 2, d), (2, N, 4, d))]


def _call(t, kw):
    q, k, v = (x.clone().requires_grad_(True) for x in t[:3])
    O = jm.masked_attention_via_map(q, k, v, **kw)
    return [O.detach(), *torch.autograd.grad(O, (q, k, v), t[3])]


@pytest.mark.parametrize("refuse", ["limit", "allocator"])
@pytest.mark.parametrize("N,L,d,kw", [
    (200, 200, 16, dict(is_causal=True)),
    (129, 193, 64, dict(block_size=10)),
    (260, 260, 128, dict(mask_fn=M.sliding_window_mask(70, 3))),
    (192, 192, 40, dict(mask_fn=lambda b, h, q, k: (q + k + h) % 3 != 0)),
], ids=["causal_d16", "full_d64", "window_d128", "table_d40"])
def test_without_planes(monkeypatch, refuse, N, L, d, kw):
    """Each side is within 2e-6 of the exact result in the 2-norm (tests/test_gpu_f32.py), so 4e-6 between them."""
    t = _inputs(N, L, d)
    want = _call(t, kw)
    calls = []
    if refuse == "limit":
        monkeypatch.setattr(A, "_F32_PLANES_LIMIT", 0)
    else:
        empty = torch.empty

        def no_planes(*a, **k):
            if k.get("dtype") is torch.uint8 and a[0][0] in sizes:
                calls.append(a[0][0])
                raise torch.OutOfMemoryError("no room")
            return empty(*a, **k)

        sizes = {route[3] for route in nat.host().routes(*t[:3], None, None, nat.BMA_BACKEND_AUTO, True, True)}
        monkeypatch.setattr(torch, "empty", no_planes)
    got = _call(t, kw)
    monkeypatch.undo()
    assert A.device_status() == 0
    assert refuse == "limit" or set(calls) == sizes
    for name, g, w in zip(("O", "dQ", "dK", "dV"), got, want):
        err = (g.double() - w.double()).norm() / w.double().norm()
        assert err <= 4e-6, (name, float(err))


def test_large_planes_do_not_fail():
    """A head dimension of 1 pads 64-fold: planes above the limit, inputs of a few MB."""
    N, H = 4096, 64
    q, k, v = (torch.randn(1, N, H, 1, device="cuda", generator=torch.Generator("cuda").manual_seed(i)) for i in range(3))
    before = A._F32_PLANES_LIMIT
    A._F32_PLANES_LIMIT = 64 << 20
    try:
        torch.cuda.reset_peak_memory_stats()
        base = torch.cuda.memory_allocated()
        O = jm.masked_attention_via_map(q, k, v, mask_fn=M.sliding_window_mask(200, 0))
        assert torch.cuda.max_memory_allocated() - base < 64 << 20
    finally:
        A._F32_PLANES_LIMIT = before
    want = jm.masked_attention_via_map(q, k, v, mask_fn=M.sliding_window_mask(200, 0))
    assert (O - want).norm() / want.norm() <= 4e-6
