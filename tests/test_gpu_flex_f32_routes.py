"""Which kernels a float32 flex_attention call takes, and that every one of its routes gives the BlockMask's meaning."""
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat
from jaxmodules_b200 import attention as A
from jaxmodules_b200 import flex as F
from jaxmodules_b200 import masks as M
from jaxmodules_b200.block_mask import get_dense_from_kv_blocks

pytestmark = pytest.mark.gpu
AUTO, SIMT = nat.BMA_BACKEND_AUTO, nat.BMA_BACKEND_SIMT
L = 512


def created(block, mask=None, **kw):
    return jm.create_block_mask(mask or M.causal_mask(), kw.get("B", 1), 1, L, L, block)


def rebuilt(block):
    """The same lists, from their dense form: not known to be those of the mask."""
    bm = created(block)
    return jm.BlockMask.from_blocks(bm.get_partial_blocks(), bm.get_full_blocks(), block, bm.mask_mod)


def dropped(block):
    bm = created(block)
    full = bm.get_full_blocks().clone()
    full[0, 0, -1, 0] = False
    return jm.BlockMask.from_blocks(bm.get_partial_blocks(), full, block, bm.mask_mod)


def listed_twice(block):
    """A block of the last row that is listed as full and as partial (it is full), and the diagonal block of the second row likewise."""
    bm = created(block)
    part, pidx, full, fidx = (t.clone() for t in (bm.kv_num_blocks, bm.kv_indices, bm.full_kv_num_blocks, bm.full_kv_indices))
    pidx[0, 0, -1, 1] = 0
    part[0, 0, -1] += 1
    fidx[0, 0, 1, 1] = 1
    full[0, 0, 1] += 1
    return jm.BlockMask.from_kv_blocks(part, pidx, full, fidx, block, bm.mask_mod, seq_lengths=(L, L))


def q_side_cut(block):
    """Only the kv side counts (the reference never reads the other one)."""
    bm = created(block)
    bm.full_q_num_blocks = bm.full_q_num_blocks.clone()
    bm.full_q_num_blocks[0, 0, 0] = 0
    return bm


def written_to(block):
    """The last full block of the last row taken out in place, on both sides (it is the last entry of its column too)."""
    bm = created(block)
    n = L // block
    bm.full_kv_num_blocks[0, 0, n - 1] -= 1
    bm.full_q_num_blocks[0, 0, n - 2] -= 1
    return bm


CASES = [   # BlockMask, block, (route, backend)
    (created, 128, ("lists", AUTO)), (created, 64, ("terms", AUTO)), (created, 32, ("terms", AUTO)),
    (rebuilt, 128, ("lists", AUTO)), (rebuilt, 64, ("terms", AUTO)),
    (dropped, 128, ("lists", AUTO)), (dropped, 64, ("lists", SIMT)), (dropped, 32, ("table", AUTO)),
    (listed_twice, 128, ("table", AUTO)), (q_side_cut, 128, ("terms", AUTO)), (written_to, 128, ("lists", AUTO)), (written_to, 64, ("lists", SIMT)),
    (lambda b: created(b, lambda b_, h, q, k: (k <= q) & (q - k <= 300)), 64, ("table", AUTO)),
    (lambda b: created(b, M.document_mask(torch.arange(L).repeat(2, 1) // 200, causal=True), B=2), 64, ("terms", AUTO)),
]


@pytest.mark.parametrize("make,block,want", CASES, ids=[f"{getattr(c[0], '__name__', 'mask')}_{c[1]}_{i}" for i, c in enumerate(CASES)])
def test_routes(monkeypatch, make, block, want):
    bm = make(block)
    g = torch.Generator().manual_seed(block)
    q, k, v, dO = (torch.randn(2, h, L, 32, generator=g).cuda() for h in (4, 2, 2, 4))
    taken = []
    route = F.float32_route
    monkeypatch.setattr(F, "float32_route", lambda *a: taken.append(route(*a)) or taken[-1])
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    O = jm.flex_attention(*leaves, block_mask=bm, enable_gqa=True)
    grads = torch.autograd.grad(O, leaves, dO)
    assert taken == [want] and A.device_status() == 0
    # the mask the lists mean, spelled out
    dense = torch.zeros((bm.B, 1, L, L), dtype=torch.bool)
    side = (bm.kv_num_blocks, bm.kv_indices, bm.full_kv_num_blocks, bm.full_kv_indices)
    part, full = (get_dense_from_kv_blocks(bm.B, bm.H, L // block, L // block, side[i], side[i + 1]) for i in (0, 2))
    up = lambda t: t.cpu().repeat_interleave(block, -2).repeat_interleave(block, -1)
    i = torch.arange(L)
    elem = torch.stack([torch.as_tensor(bm.mask_mod(b, 0, i[:, None].numpy(), i[None, :].numpy())) for b in range(bm.B)])[:, None]
    dense = up(full) | (up(part) & elem)
    ref = [t.double().cpu().requires_grad_(True) for t in (q, k, v)]
    s = (ref[0] @ ref[1].repeat_interleave(2, 1).transpose(-1, -2)) / 32 ** 0.5
    want_O = torch.softmax(s.masked_fill(~dense, float("-inf")), -1) @ ref[2].repeat_interleave(2, 1)
    for name, x, y in zip(("O", "dQ", "dK", "dV"), (O.detach(), *grads), (want_O.detach(), *torch.autograd.grad(want_O, ref, dO.double().cpu()))):
        assert (x.cpu().double() - y).norm() <= 2e-6 * y.norm(), name      # as for every float32 call, tests/test_gpu_f32.py
