"""The dS hand-over of the bf16 backward with per-head block lists, from one list head to more than one launch takes.  The dQ kernel that recomputes S and dP, which uses no slots, returns the same dQ up
to the order of its sums and the same dK and dV bit for bit."""
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import attention as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,N,per_batch", [(1, 1, 300, False), (1, 32, 300, False), (1, 33, 300, False), (3, 12, 1100, True), (5, 64, 260, True)])
def test_slots(B, H, N, per_batch):
    mask = (lambda b, h, q, k: (k <= q) & (q - k <= 40 + 9 * h + 70 * b)) if per_batch else (lambda h, q, k: (k <= q) & (q - k <= 40 + 9 * h))
    g = torch.Generator("cuda").manual_seed(H)
    q, k, v = (torch.randn(B, N, H, 64, device="cuda", generator=g).bfloat16().requires_grad_(True) for _ in range(3))
    dO = torch.randn(B, N, H, 64, device="cuda", generator=g)
    grads = []
    limit = A._scratch_limit
    try:
        for share in (limit, 0):
            A.set_backward_scratch_limit(share)
            grads.append(torch.autograd.grad(jm.masked_attention_via_map(q, k, v, mask_fn=mask), (q, k, v), dO))
            assert A.last_backward_info["whole"] == (share > 0)
    finally:
        A.set_backward_scratch_limit(limit)
    assert A.device_status() == 0
    for name, x, y in zip(("dQ", "dK", "dV"), *grads):
        if name != "dQ":
            assert torch.equal(x, y), name
        assert (x.float() - y.float()).norm() <= 4e-3 * y.float().norm(), name   # a rounding of dS and of dQ to bf16
