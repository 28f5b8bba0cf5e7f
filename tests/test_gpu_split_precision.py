"""Shapes that had fp32 probabilities on the CUDA-core kernels keep their accuracy on the tensor cores.

The yardstick is the error of the forced CUDA-core kernels on the same inputs against a float64 computation.  The
probabilities' hi + lo form loses 2^-17 of a value (bf16), against 2^-9 of the rounding of the result, so the two errors
agree up to the randomness of a few thousand roundings: 2 % is allowed for that."""

import math

import pytest
import torch

import torch_neuronx_b200 as T
from torch_neuronx_b200 import _lib

pytestmark = pytest.mark.gpu


def _reference(q, k, v, go, causal):
    q, k, v, go = (t.double() for t in (q, k, v, go))
    scale = 1.0 / math.sqrt(q.shape[-1])
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).tril(), float("-inf"))
    p = torch.softmax(s, -1)
    out = p @ v
    dp = go @ v.transpose(-1, -2)
    ds = p * (dp - (go * out).sum(-1, keepdim=True)) * scale
    return out, ds @ k, ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ go


def _error(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("E,Dv,L,causal", [(80, 80, 577, False), (96, 96, 130, True), (72, 128, 512, True),
                                           (192, 128, 700, True), (192, 128, 256, False), (256, 256, 333, True)])
def test_error_no_larger_than_cuda_cores(E, Dv, L, causal, dtype):
    g = torch.Generator(device="cuda").manual_seed(E + L)
    q, k, v, go = (torch.randn(2, 4, L, d, generator=g, device="cuda").to(dtype) for d in (E, E, Dv, Dv))
    want = _reference(q, k, v, go, causal)
    forward = {}
    for path in (_lib.PATH_AUTO, _lib.PATH_GENERIC):
        forward[path] = T.sdpa_forward(q, k, v, is_causal=causal, force_path=path)
    if E <= 128:
        assert _error(forward[_lib.PATH_AUTO][0], want[0]) <= 1.02 * _error(forward[_lib.PATH_GENERIC][0], want[0])
    out, lse = forward[_lib.PATH_GENERIC]
    new = T.sdpa_backward(go, q, k, v, out, lse, is_causal=causal)[:3]
    old = T.sdpa_backward(go, q, k, v, out, lse, is_causal=causal, force_path=_lib.PATH_GENERIC)[:3]
    T.check_device_status()
    for name, a, b, w in zip(("dq", "dk", "dv"), new, old, want[1:]):
        assert _error(a, w) <= 1.02 * _error(b, w), (name, _error(a, w), _error(b, w))
