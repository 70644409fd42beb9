"""Infinities, NaN and values next to the largest float32 in float32 attention: the tensor-core kernels carry an operand as three
bfloat16 planes, which no such value has, so the tiles it reaches are done by the FP32 tile functions.  Results are those of
the FP32 tile kernels at every element: NaN where they give NaN, the same infinities, and the finite values within float32 rounding."""
import numpy as np
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat
from jaxmodules_b200 import masks as M

pytestmark = pytest.mark.gpu
INF, BIG = float("inf"), 3.4e38     # BIG rounds to infinity in bfloat16

# (operand, batch, position, head, column, value)
CASES = {
    "v_inf": [("v", 0, 5, 0, 3, INF)],
    "v_both_inf": [("v", 0, 5, 0, 3, INF), ("v", 0, 70, 1, 0, -INF)],
    "k_minus_inf_score": [("k", 0, 9, 0, 1, -INF)],
    "k_nan_last": [("k", 1, 190, 1, 0, float("nan"))],
    "v_nan_behind_the_diagonal": [("v", 1, 100, 0, 2, float("nan"))],   # the same 128-block as the queries below 64, another 64-block
    "q_inf": [("q", 0, 130, 2, 0, INF)],
    "v_near_max": [("v", 0, 3, 0, 7, BIG)],
    "k_near_max": [("k", 0, 3, 1, 7, BIG)],
    "do_inf": [("do", 1, 150, 3, 4, INF)],
    "do_near_max": [("do", 0, 20, 0, 4, -BIG)],
}
MASKS = {
    "causal": lambda: dict(is_causal=True),
    "window": lambda: dict(mask_fn=M.sliding_window_mask(40, 10)),
    "table": lambda: dict(mask_fn=lambda b, h, q, k: (k <= q) & ((q - k) % 3 != 1) & (q - k < 90)),
}


def _inputs(d, N, case):
    g = torch.Generator().manual_seed(11)
    t = {n: torch.randn((2, N, 4 if n in ("q", "do") else 2, d), generator=g) for n in ("q", "k", "v", "do")}
    if case == "k_minus_inf_score":
        t["q"][..., 1] = t["q"][..., 1].abs() + 0.1       # every score of that key is -inf: its weight is 0
    for name, b, l, h, c, value in CASES[case]:
        t[name][b, l, h, c] = value
    return {n: x.cuda() for n, x in t.items()}


def _run(t, kw, backend):
    q, k, v = (t[n].clone().requires_grad_(True) for n in "qkv")
    O = jm.masked_attention_via_map(q, k, v, backend=backend, **kw)
    return [x.detach().cpu().numpy() for x in (O, *torch.autograd.grad(O, (q, k, v), t["do"]))]


@pytest.mark.parametrize("mask", MASKS)
@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("d,N", [(40, 200), (64, 256), (128, 200)])
def test_non_finite(d, N, case, mask):
    t, kw = _inputs(d, N, case), MASKS[mask]()
    got, want = _run(t, kw, nat.BMA_BACKEND_AUTO), _run(t, kw, nat.BMA_BACKEND_SIMT)
    for name, g, w in zip(("O", "dQ", "dK", "dV"), got, want):
        assert np.array_equal(np.isnan(g), np.isnan(w)), name
        assert np.array_equal(np.isinf(g), np.isinf(w)) and np.array_equal(np.sign(g[np.isinf(g)]), np.sign(w[np.isinf(w)])), name
        fin = np.isfinite(w)
        if fin.any():      # float32 sums in another order, relative to the largest of the finite values
            assert np.abs(g[fin].astype(np.float64) - w[fin]).max() <= 2e-5 * max(1.0, np.abs(w[fin].astype(np.float64)).max()), name


@pytest.mark.parametrize("d", [64, 128])
def test_expected_values(d):
    """What the two cases mean, without the other kernels: an infinite value is the result of every query that sees it (and, as
    0 * infinity, not a number for the queries before it in its block of 64, whatever the other columns); a key whose scores
    are -inf has weight 0."""
    t = _inputs(d, 256, "v_inf")
    O = jm.masked_attention_via_map(t["q"], t["k"], t["v"], is_causal=True).cpu()
    want = torch.zeros((2, 256, 4, d), dtype=torch.bool)
    want[0, 5:, :2, 3] = True
    assert torch.equal(O == INF, want)
    want[0, :5, :2, 3] = True
    assert torch.isfinite(O[~want]).all()
    t = _inputs(d, 256, "k_minus_inf_score")
    O = jm.masked_attention_via_map(t["q"], t["k"], t["v"], mask_fn=M.sliding_window_mask(300, 300)).cpu()
    s = torch.einsum("nhd,lhd->hnl", t["q"][0, :, :1].double().cpu(), t["k"][0, :, :1].double().cpu()) / d ** 0.5
    ref = torch.einsum("hnl,lhd->nhd", torch.softmax(s, -1), t["v"][0, :, :1].double().cpu())
    assert (O[0, :, :1] - ref).abs().max() <= 1e-5


@pytest.mark.parametrize("d", [64, 128])
def test_bf16_output_and_cotangent(d):
    """float32 inputs with a bfloat16 output, so that the cotangent is bfloat16 too.  delta is taken from the rounded O (2^-9), which
    bounds how far dQ and dK of the two sides may differ; O itself by a rounding."""
    t = _inputs(d, 200, "do_inf")
    t["do"] = t["do"].bfloat16()
    kw = dict(is_causal=True, out_dtype=torch.bfloat16)
    out = []
    for backend in (nat.BMA_BACKEND_AUTO, nat.BMA_BACKEND_SIMT):
        q, k, v = (t[n].clone().requires_grad_(True) for n in "qkv")
        O = jm.masked_attention_via_map(q, k, v, backend=backend, **kw)
        out.append([x.detach().float() for x in (O, *torch.autograd.grad(O, (q, k, v), t["do"]))])
    for name, g, w in zip(("O", "dQ", "dK", "dV"), *out):
        assert torch.equal(torch.isnan(g), torch.isnan(w)) and torch.equal(torch.isinf(g), torch.isinf(w)), name
        fin = torch.isfinite(w)
        assert (g[fin] - w[fin]).norm() <= (2e-6 if name == "dV" else 4e-3) * w[fin].norm(), name
