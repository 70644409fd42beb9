"""float32 forward passes whose tiles share their key lists out over the CTAs of a cluster (2 to 8 of them, and the last wave of an even launch in a
launch of its own), against float64: ragged ends, head dimensions without whole 16-byte rows, rows without a key, bfloat16 output, results that
are not finite.

Bound: 2e-6 in the 2-norm as for every float32 forward pass (tests/test_gpu_f32.py); the sum over parts adds one rounding per part."""
import math

import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import attention as A, masks as M

pytestmark = pytest.mark.gpu

CASES = [
    # B, N, L, Hq, Hkv, d, mask
    (1, 1, 3000, 1, 1, 64, "none"),           # one tile, eight parts
    (1, 257, 1500, 2, 1, 128, "none"),        # parts that end on the ragged last tile
    (1, 300, 1100, 3, 3, 33, "causal"),       # rows of 33 floats
    (2, 500, 500, 4, 4, 65, "causal"),
    (1, 140, 900, 4, 2, 128, "empty rows"),
    (1, 1500, 1500, 16, 4, 64, "none"),       # 148 tiles, and 44 in parts
    (1, 1000, 1000, 9, 9, 128, "causal"),     # 72 tiles of 1 to 8 key tiles
    (1, 700, 2500, 8, 8, 64, "band"),
]
MASKS = {
    "none": (None, lambda q, k, N, L: torch.ones_like(q + k, dtype=torch.bool)),
    "causal": (M.causal_mask(), lambda q, k, N, L: k <= q),
    "empty rows": (M.sliding_window_mask(20, 0), lambda q, k, N, L: (k <= q) & (k >= q - 20) & (q >= 0)),
    "band": (M.sliding_window_mask(400, 1900), lambda q, k, N, L: (k >= q - 400) & (k <= q + 1900)),
}


def _reference(q, k, v, mask):
    G = q.shape[2] // k.shape[2]
    kk, vv = (t.double().repeat_interleave(G, 2) for t in (k, v))
    s = torch.einsum("bnhd,blhd->bhnl", q.double(), kk) / math.sqrt(q.shape[-1])
    i, j = torch.arange(q.shape[1], device="cuda")[:, None], torch.arange(k.shape[1], device="cuda")[None]
    s = s.masked_fill(~MASKS[mask][1](i, j, q.shape[1], k.shape[1]), float("-inf"))
    p = torch.softmax(s, -1).nan_to_num(0.0)
    return torch.einsum("bhnl,blhd->bnhd", p, vv), torch.logsumexp(s, -1)


@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,mask", CASES, ids=[f"N{c[1]}_L{c[2]}_H{c[3]}_d{c[5]}_{c[6]}" for c in CASES])
def test_shared_rows(B, N, L, Hq, Hkv, d, mask, out):
    g = torch.Generator(device="cuda").manual_seed(N + d)
    q, k, v = (torch.randn(s, device="cuda", generator=g) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d)))
    O, lse = jm.masked_attention_via_map(q, k, v, mask_fn=MASKS[mask][0], block_size=N + 1, out_dtype=out, return_lse=True)
    want, wlse = _reference(q, k, v, mask)
    tol = 2e-6 if out == torch.float32 else 2.5e-3        # (bfloat16: 2^-9 per value)
    assert (O.double() - want).norm() <= tol * want.norm()
    dead = torch.isinf(wlse)
    assert torch.equal(torch.isinf(lse), dead) and (lse.double() - wlse)[~dead].abs().max() <= 1e-5
    assert A.device_status() == 0


@pytest.mark.parametrize("where", [0, 1400], ids=["first part", "last part"])
def test_not_finite_in_one_part(where):
    """An infinity in V of one part: all rows of the tile are done again, with the effect it has in float32 arithmetic."""
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn((1, n, 2, 64), device="cuda", generator=g) for n in (200, 1500, 1500))
    clean = v.clone()
    v[0, where, 1, 5] = float("inf")
    O = jm.masked_attention_via_map(q, k, v, block_size=201)
    want, _ = _reference(q, k, clean, "none")
    assert torch.isinf(O[0, :, 1, 5]).all()
    O = O.clone()
    O[0, :, 1, 5] = want[0, :, 1, 5].float()
    assert (O.double() - want).norm() <= 2e-6 * want.norm()


def test_key_bias_and_negative_scale():
    g = torch.Generator(device="cuda").manual_seed(2)
    q, k, v = (torch.randn((1, n, 3, 64), device="cuda", generator=g) for n in (130, 900, 900))
    bias = torch.tensor([0.01, -0.02, 0.0], device="cuda")
    O, lse, _ = A.attention_forward(q, k, v, M.MaskTerms(), scale=-0.2, key_bias=bias)
    s = -0.2 * torch.einsum("bnhd,blhd->bhnl", q.double(), k.double()) + bias.double()[None, :, None, None] * torch.arange(900, device="cuda").double()
    want = torch.einsum("bhnl,blhd->bnhd", torch.softmax(s, -1), v.double())
    assert (O.double() - want).norm() <= 2e-6 * want.norm() and (lse.double() - torch.logsumexp(s, -1)).abs().max() <= 2e-5
