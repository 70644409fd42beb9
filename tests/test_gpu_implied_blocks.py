"""Masks whose blocks the kernels know without block lists: what list compilation refuses is refused there as well, and what lies in blocks
that no query sees reaches no output."""
import ctypes as C

import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat, attention as A, masks as M

pytestmark = pytest.mark.gpu

REFUSED = {
    "window without a block": M.MaskTerms(window=(0, 1, 1, 4)),
    "window that starts behind its queries": M.MaskTerms(window=(64, -2, 4, 4)),
    "window that ends before them": M.MaskTerms(window=(64, 4, -2, 4)),
    "window wider than the keys": M.MaskTerms(window=(64, 4, 4, 4)),
    "band without keys": M.MaskTerms(band=(-1, 3)),
    "band to the left": M.MaskTerms(band=(3, -1)),
}


@pytest.mark.parametrize("mask", REFUSED)
@pytest.mark.parametrize("N", [16, 256])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_terms_that_are_refused(dtype, N, mask):
    q, k = (torch.zeros((1, n, 2, 64), device="cuda", dtype=dtype) for n in (N, 256))
    for need_q_side in (False, True):
        with pytest.raises(nat.BmaError) as e:
            A.attention_forward(q, k, k, REFUSED[mask], need_q_side=need_q_side)
        assert e.value.status == -1


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_window_sizes_that_are_refused(dtype):
    q = torch.zeros((1, 512, 2, 64), device="cuda", dtype=dtype)
    for window in ((-300, 400), (400, -300)):
        with pytest.raises(nat.BmaError):
            jm.masked_attention_via_map(q, q, q, block_size=128, window_size=window)


UNSEEN = [
    # dtype, N, L, d, (block, left, right), first key of the blocks that no query sees
    (torch.bfloat16, 16, 2000, 128, (8, 1, 12), 128),      # few queries
    (torch.bfloat16, 300, 4000, 64, (64, 1, 25), 2048),    # one CTA per pair of query tiles
    (torch.float32, 300, 2000, 64, (64, 1, 2), 512),
    (torch.float32, 200, 1500, 128, (32, 0, 3), 384),
    (torch.float32, 16, 9000, 64, (8, 1, 12), 128),        # few queries: planes of listed blocks only
]


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("grad", [False, True], ids=["forward", "backward"])
@pytest.mark.parametrize("dtype,N,L,d,window,first", UNSEEN, ids=[f"{str(c[0])[6:]}_N{c[1]}_L{c[2]}_d{c[3]}" for c in UNSEEN])
def test_unseen_keys(dtype, N, L, d, window, first, grad, value):
    """A block window that changes inside the query tiles: values that are not finite outside every window leave the results as they are."""
    terms = M.MaskTerms(window=(*window, -(-L // window[0])))
    g = torch.Generator(device="cuda").manual_seed(N + L)
    q, k, v, do = (torch.randn((1, n, 2, d), device="cuda", generator=g).to(dtype) for n in (N, L, L, N))
    spec = M.to_device_mask(terms, N, L, q.device).spec
    assert nat.host().implies_lists(q, k, v, None, None, nat.BMA_BACKEND_AUTO, C.addressof(spec))
    bad = [t.clone() for t in (k, v)]
    for t in bad:
        t[:, first:] = value

    def call(k, v):
        O, lse, ctx = A.attention_forward(q, k, v, terms, need_q_side=grad)
        return [O, lse, *(A.attention_backward(q, k, v, O, lse, do.float(), ctx) if grad else ())]

    for name, x, y in zip(("O", "lse", "dQ", "dK", "dV"), call(k, v), call(*bad)):
        assert torch.equal(x, y) and torch.isfinite(x).all(), name
