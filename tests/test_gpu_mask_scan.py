"""Blocks that closed forms leave open: scanned inside the compaction (rows of up to 32 blocks) and by the passes of their
own (wider rows), at block sizes around the 32-row and 128-key steps of the scan.  Integer work: bit exact."""
import pytest

import jaxmodules_b200 as jm
from jaxmodules_b200 import masks as M
from test_gpu_block_mask import _segments, assert_same
from oracle import block_mask_oracle as bo

pytestmark = pytest.mark.gpu

# far from the diagonal everything is allowed or nothing, near it the mask is ragged: empty, cut and full blocks
RAGGED = lambda b, h, q, k: ((q - k) > 40) | ((abs(q - k) <= 40) & ((q * 7 + k * (h + 1)) % 3 == 0))


@pytest.mark.parametrize("BS,nq,nk", [(16, 32, 32), (16, 33, 20), (20, 9, 40), (31, 8, 8), ((33, 160), 13, 3), (128, 4, 4), ((8, 136), 40, 4)],
                         ids=lambda v: str(v).replace(" ", ""))
def test_ragged_table(BS, nq, nk):
    QB, KVB = (BS, BS) if isinstance(BS, int) else BS
    B, H, QL, KL = 1, 2, nq * QB, nk * KVB
    assert_same(jm.create_block_mask(RAGGED, B, H, QL, KL, BS), bo.create_block_mask(RAGGED, B, H, QL, KL, BS))


@pytest.mark.parametrize("nb", [32, 33])
def test_documents_cut_inside_blocks(nb):
    m = M.document_mask(_segments(2, nb * 16, 5, 60, seed=nb), causal=True)
    assert_same(jm.create_block_mask(m, 2, 2, nb * 16, nb * 16, 16), bo.create_block_mask(m, 2, 2, nb * 16, nb * 16, 16))


@pytest.mark.parametrize("at", ["first", "row31_key32", "row32_key31", "last"])
@pytest.mark.parametrize("BS", [16, 32, 33, 64, 160])
def test_one_element_decides(BS, at):
    """Blocks that are whole, or empty, but for one element inside and outside of the 32 x 32 that are looked at first."""
    r, c = {"first": (0, 0), "row31_key32": (31, 32), "row32_key31": (32, 31), "last": (BS - 1, BS - 1)}[at]
    one = lambda q, k: (q % BS == r % BS) & (k % BS == c % BS)
    mask = lambda b, h, q, k: (((q // BS + k // BS) % 2 == 0) & (one(q, k) == False)) | (((q // BS + k // BS) % 2 == 1) & ((k // BS) % 3 != 0) & one(q, k))
    assert_same(jm.create_block_mask(mask, 1, 1, 5 * BS, 7 * BS, BS), bo.create_block_mask(mask, 1, 1, 5 * BS, 7 * BS, BS))


@pytest.mark.parametrize("H", [32, 33])
def test_many_heads_of_short_rows(H):
    """32 x 32 blocks: scanned inside the compaction up to 32 heads, by the passes of their own beyond."""
    mask = lambda b, h, q, k: (k <= q) & (q - k <= 3 * h + 20)
    assert_same(jm.create_block_mask(mask, 1, H, 512, 512, 16), bo.create_block_mask(mask, 1, H, 512, 512, 16))
