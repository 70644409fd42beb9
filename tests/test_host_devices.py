"""Devices that are not CUDA devices are refused before any native call: the kernels would be given addresses of host memory."""
import numpy as np
import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import _native as nat, attention as A, block_mask as BM, masks as M


@pytest.fixture
def no_native_call(monkeypatch):
    """A CUDA device seems to be there; a call of either library fails the test."""
    class Native:
        def __getattr__(self, name):
            raise AssertionError(f"native code was reached: {name}")
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 0, raising=False)
    monkeypatch.setattr(nat, "host", Native)
    monkeypatch.setattr(nat, "lib", Native)


MASKS = {"causal": M.causal_mask(), "documents": M.document_mask(np.repeat(np.arange(4, dtype=np.int32), 32)[None]), "callable": lambda b, h, q, k: q >= k}


@pytest.mark.parametrize("device", ["cpu", "cpu:0", "meta"])
@pytest.mark.parametrize("mask", MASKS)
def test_create_block_mask(no_native_call, mask, device):
    with pytest.raises(ValueError, match="cuda device"):
        jm.create_block_mask(MASKS[mask], 1, 1, 128, 128, 16, device=device)


@pytest.mark.parametrize("device", ["cpu", "cpu:0"])
def test_compile_block_lists(no_native_call, device):
    dmask = M.to_device_mask(M.MaskTerms(causal=True), 128, 128, torch.device("cpu"))
    for stream in (None, 0):
        with pytest.raises(ValueError, match="cuda device"):
            BM.compile_block_lists(dmask, 1, 1, 128, 128, 16, 16, device, stream=stream)


def test_attention(no_native_call):
    q = torch.zeros((1, 128, 1, 64))
    with pytest.raises(ValueError, match="cuda device"):
        A.attention_forward(q, q, q, M.MaskTerms())
    with pytest.raises(ValueError, match="cuda device"):
        A.attention_backward(q, q, q, q, q[..., 0], q, {})


def test_a_cuda_device_without_an_index_is_the_current_one(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    assert nat.device_guard(torch.device("cuda")) is nat._NO_GUARD and nat.device_guard(torch.device("cuda:0")) is nat._NO_GUARD
    assert nat.device_index(torch.device("cuda:3")) == 3
