"""The host side of a call (csrc/host.cc): what it refuses, saved tensors whose layout a hook has changed, calls from several threads."""
import threading

import pytest
import torch

import jaxmodules_b200 as jm
from jaxmodules_b200 import attention as A, masks as M

pytestmark = pytest.mark.gpu


def _inputs(dtype, B=2, N=200, Hq=4, Hkv=2, d=64, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    make = lambda H: torch.randn((B, N, H, d), device="cuda", generator=g).to(dtype).requires_grad_(True)
    return [make(Hq), make(Hkv), make(Hkv)], torch.randn((B, N, Hq, d), device="cuda", generator=g)


def _call(qkv, dO, **kw):
    O = jm.masked_attention_via_map(*qkv, **kw)
    return [O.detach(), *torch.autograd.grad(O, qkv, dO)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_saved_tensors_of_another_layout(dtype):
    """Hooks may hand back tensors of other strides and alignment than the forward pass had: here heads outermost, one element off
    a 16-byte boundary, which is no operand of a TMA load.  bfloat16 then runs the FP32 tile kernels: bounded like any two of its paths."""
    qkv, dO = _inputs(dtype)
    want = _call(qkv, dO, is_causal=True)

    def unpack(t):
        if t.ndim != 4:
            return t
        flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:]
        return flat.view(t.shape[0], t.shape[2], t.shape[1], t.shape[3]).transpose(1, 2).copy_(t)

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        O = jm.masked_attention_via_map(*qkv, is_causal=True)
        got = [O.detach(), *torch.autograd.grad(O, qkv, dO)]
    tol = 4e-6 if dtype == torch.float32 else 1.2e-2      # (tests/test_gpu_f32_memory.py; the roundings of bfloat16 outputs and of P)
    for name, x, y in zip(("O", "dQ", "dK", "dV"), got, want):
        assert (x.double() - y.double()).norm() <= tol * y.double().norm(), name
    assert A.device_status() == 0


def test_refused():
    (q, k, v), _ = _inputs(torch.bfloat16)
    with pytest.raises(KeyError):
        jm.masked_attention_via_map(q, k, v, out_dtype=torch.float16)
    with pytest.raises(TypeError):
        jm.masked_attention_via_map(q, k.float(), v)
    with pytest.raises(ValueError, match="innermost dimension"):
        A.attention_forward(q.transpose(2, 3), k.transpose(2, 3), v.transpose(2, 3), M.MaskTerms())


def test_threads_on_streams_of_their_own():
    cases = [(dtype, seed) for dtype in (torch.float32, torch.bfloat16) for seed in range(4)]
    inputs = [_inputs(dtype, seed=seed, N=300) for dtype, seed in cases]
    want = [_call(*i, mask_fn=M.sliding_window_mask(40, 0)) for i in inputs]
    torch.cuda.synchronize()
    got, errors = [None] * len(cases), []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    got[i] = _call(*inputs[i], mask_fn=M.sliding_window_mask(40, 0))
                torch.cuda.current_stream().synchronize()
        except Exception as e:      # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for x, y in zip(got, want):
        assert all(torch.equal(a, b) for a, b in zip(x, y))
