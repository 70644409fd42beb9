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
