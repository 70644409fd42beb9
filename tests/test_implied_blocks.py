"""The blocks that the kernels take a mask of interval terms to have when they are given no block lists (bma_mask_block_class, the function
the kernels themselves call): empty, partial or full exactly as the elements of the dense mask say, for windows that change inside a query
block, offsets, bands, causal masks and ragged ends."""
import ctypes as C
import random

import numpy as np
import pytest
import torch

from jaxmodules_b200 import _native as nat, masks as M


def _dense(t, N, L):
    """The mask of the terms over [N, L], as the reference writes each of them out."""
    q, k = np.arange(N)[:, None] + t.q_offset, np.arange(L)[None] + t.k_offset
    ok = np.ones((N, L), dtype=bool)
    if t.causal:
        ok &= k <= q
    if t.band is not None:
        ok &= (k >= q - t.band[0]) & (k <= q + t.band[1])
    if t.window is not None:
        block, left, right, n = t.window
        start = np.minimum(np.maximum(q // block - left, 0), n - left - right) * block
        ok &= (k >= start) & (k < start + (left + right) * block)
    return ok


def _classes(t, N, L, tile):
    spec = M.to_device_mask(t, N, L, torch.device("cpu")).spec
    f = nat.lib().bma_mask_block_class
    return np.array([[f(C.byref(spec), tile, tile, i, j) for j in range(-(-L // tile))] for i in range(-(-N // tile))])


def _want(t, N, L, tile):
    NQ, NKV = -(-N // tile), -(-L // tile)
    ok = np.zeros((NQ * tile, NKV * tile), dtype=bool)
    ok[:N, :L] = _dense(t, N, L)
    b = ok.reshape(NQ, tile, NKV, tile)
    return b.any((1, 3)).astype(int) + b.all((1, 3))


TILE = 128
SIZES = [(1024, 1024), (700, 1300), (130, 900), (1000, 333), (1, 1), (5, 640)]
WINDOWS = [(8, 4, 3), (32, 8, 1), (64, 4, 5), (96, 2, 3), (192, 2, 2), (100, 0, 1), (1, 200, 30), (128, 1, 2), (1000, 0, 1)]


@pytest.mark.parametrize("terms", ["window", "causal", "band", "offsets"])
@pytest.mark.parametrize("window", WINDOWS, ids=str)
def test_windows(window, terms):
    block, left, right = window
    for N, L in SIZES:
        n = max(-(-(max(N, L) + 700) // block), left + right)
        extra = {"window": {}, "causal": dict(causal=True), "band": dict(band=(90, 40)), "offsets": dict(q_offset=300, k_offset=77, causal=True)}[terms]
        t = M.MaskTerms(window=(block, left, right, n), **extra)
        assert np.array_equal(_classes(t, N, L, TILE), _want(t, N, L, TILE)), (N, L)
        t = M.MaskTerms(window=(block, left, right, left + right), **extra)      # the window is all the blocks there are
        assert np.array_equal(_classes(t, N, L, TILE), _want(t, N, L, TILE)), (N, L)


def test_random_terms():
    rng = random.Random(0)
    for _ in range(400):
        N, L = rng.randint(1, 600), rng.randint(1, 600)
        block, left, right = rng.randint(1, 300), rng.randint(0, 9), rng.randint(0, 9)
        t = M.MaskTerms(causal=rng.random() < 0.4, band=(rng.randint(0, 300), rng.randint(0, 300)) if rng.random() < 0.4 else None,
                        window=(block, left, right, left + right + rng.randint(0, 12)) if rng.random() < 0.8 else None,
                        q_offset=rng.choice([0, 0, rng.randint(0, 500)]), k_offset=rng.choice([0, 0, rng.randint(0, 500)]))
        tile = rng.choice([128, 64, 17])
        assert np.array_equal(_classes(t, N, L, tile), _want(t, N, L, tile)), (t, N, L, tile)


@pytest.mark.parametrize("N,window,count", [(4096, (64, 4, 5), 160), (8192, (64, 16, 9), 832), (16384, (64, 4, 5), 640)])
def test_count_of_visited_blocks(N, window, count):
    """The visited blocks stay in proportion to the window (these are the blocks of the exact lists)."""
    c = _classes(M.MaskTerms(window=(*window, N // 64)), N, N, TILE)
    assert int((c > 0).sum()) == count


@pytest.mark.parametrize("terms", [M.MaskTerms(window=(0, 1, 1, 4)), M.MaskTerms(window=(64, -2, 4, 4)), M.MaskTerms(window=(64, 4, 4, 4)), M.MaskTerms(band=(-1, 3))], ids=str)
def test_refused(terms):
    assert (_classes(terms, 200, 200, TILE) == -1).all()
