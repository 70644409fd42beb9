"""Masks whose blocks the kernels know without block lists: what list compilation refuses is refused there as well."""
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
