"""The split forward kernel (one query tile, keys cut into runs, query heads packed into a tile) against the float64 oracle.
Bounds as for every bfloat16 forward: max-abs 2e-2, mean-abs 2e-3; the log-sum-exp is float32."""
import numpy as np
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import masks as M
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu

CASES = [
    # B, N, L, Hq, Hkv, d, mask
    (1, 1, 129, 1, 1, 128, "tail"),        # the fewest: one row, two kv tiles, the second with one key
    (2, 16, 1000, 8, 2, 128, "tail"),      # four heads to a tile
    (1, 5, 3000, 6, 2, 64, "none"),        # three heads to a tile: 126 of 128 rows
    (1, 100, 700, 8, 1, 64, "tail"),       # 16 queries of eight heads to a tile, seven tiles
    (2, 128, 513, 4, 4, 128, "tail"),      # a whole tile of one head
    (1, 9, 600, 4, 1, 128, "per_head"),    # lists that depend on the head: not packed
    (1, 20, 900, 8, 8, 64, "window"),      # a window that leaves most kv tiles, and some runs, without a block
    (2, 7, 2048, 4, 2, 128, "dead"),       # a query that sees no key
]
MASKS = {
    "none": lambda N, L: None,
    "tail": lambda N, L: M.sliding_window_mask(L, L - N),
    "window": lambda N, L: M.sliding_window_mask(3, 40),
    "per_head": lambda N, L: (lambda b, h, q, k: (k + h) % (h + 2) != 0),
    "dead": lambda N, L: (lambda b, h, q, k: (q != 3) & (k >= 5 * q + 200 * b)),
}


@pytest.mark.parametrize("B,N,L,Hq,Hkv,d,mask", CASES, ids=[f"N{c[1]}_L{c[2]}_H{c[3]}_{c[4]}_{c[6]}" for c in CASES])
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16], ids=["f32out", "bf16out"])
def test_few_queries(B, N, L, Hq, Hkv, d, mask, out):
    g = torch.Generator().manual_seed(N * 7 + L)
    Q, K, V = (torch.randn(s, generator=g).to(torch.bfloat16) for s in ((B, N, Hq, d), (B, L, Hkv, d), (B, L, Hkv, d)))
    kw = dict(mask_fn=MASKS[mask](N, L), block_size=N + 1)   # (a block size that N is no multiple of: any L goes)
    O, lse = jm.masked_attention_via_map(Q.cuda(), K.cuda(), V.cuda(), out_dtype=out, return_lse=True, **kw)
    ref = ao.masked_attention_dense(Q.float().numpy(), K.float().numpy(), V.float().numpy(), **kw)
    err = np.abs(O.float().cpu().numpy() - ref["O"])
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (err.max(), err.mean())
    got, want = lse.cpu().numpy(), ref["lse"]
    dead = np.isinf(want)
    assert np.array_equal(np.isinf(got), dead) and np.abs(got - want)[~dead].max() <= 1e-3


def test_split_workspace_is_bounded():
    """The partial results of the runs stay below 32 waves of CTAs whatever the sizes (nothing is launched here)."""
    import ctypes as C
    from jaxmodules_b200 import _native as nat
    from jaxmodules_b200 import attention as A
    q, k = (torch.zeros(1, n, 1, 128, dtype=torch.bfloat16, device="cuda") for n in (16, 256))
    a, lists = A._make_args(q, k, k), nat.BlockLists()
    cta = 128 * (128 + 2) * 4
    most = 32 * torch.cuda.get_device_properties(0).multi_processor_count * cta
    asked = []
    for B, N, Hq, Hkv, L in ((4, 16, 32, 8, 8192), (16, 127, 64, 64, 65536), (250, 127, 16, 4, 524288), (312, 127, 64, 16, 524288), (4000, 1, 2, 2, 524288)):
        a.B, a.N, a.Hq, a.Hkv, a.L = B, N, Hq, Hkv, L
        lists.B = lists.H = lists.NQ = 1
        lists.NKV = L // 128
        asked.append(nat.lib().bma_attn_fwd_workspace_bytes(C.byref(a), C.byref(lists)))
    assert asked[0] > 0 and max(asked) <= most, asked
