"""fp16 gradients far from 1 in the tensor-core backward of the shapes that the CUDA-core kernels served with fp32
probabilities and softmax gradients: no further from float64 than those kernels, whatever the scale of the upstream
gradient (2 % for the randomness of the roundings of the result, as in test_gpu_split_precision.py)."""

import pytest
import torch

import torch_neuronx_b200 as T
from tests.test_gpu_split_precision import _error, _reference
from torch_neuronx_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,Dv,L,causal", [(80, 80, 577, False), (96, 96, 260, True), (72, 128, 512, True),
                                           (192, 128, 700, True), (256, 256, 333, False)])
@pytest.mark.parametrize("power", [-14, -10, -6, 6, 11])
def test_scaled_gradients(E, Dv, L, causal, power):
    g = torch.Generator(device="cuda").manual_seed(E + L)
    q, k, v, go = (torch.randn(2, 4, L, d, generator=g, device="cuda") for d in (E, E, Dv, Dv))
    # large keys and queries where the gradient is small, so that the results keep their bits in fp16
    up = 2.0 ** (4 if power < 0 else 0)
    q, k, v, go = (q * up).half(), (k * up).half(), v.half(), (go * 2.0**power).half()
    scale = E**-0.5 / up**2
    want = _reference(q * 1.0, k, v, go, causal) if up == 1 else _scaled_reference(q, k, v, go, causal, scale)
    out, lse = T.sdpa_forward(q, k, v, is_causal=causal, scale=scale, force_path=_lib.PATH_GENERIC)
    new = T.sdpa_backward(go, q, k, v, out, lse, is_causal=causal, scale=scale)[:3]
    old = T.sdpa_backward(go, q, k, v, out, lse, is_causal=causal, scale=scale, force_path=_lib.PATH_GENERIC)[:3]
    T.check_device_status()
    for name, a, b, w in zip(("dq", "dk", "dv"), new, old, want[1:]):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)), name
        assert _error(a, w) <= 1.02 * _error(b, w), (name, _error(a, w), _error(b, w))


def _scaled_reference(q, k, v, go, causal, scale):
    # the reference takes 1 / sqrt(E): fold the rest into the queries, whose gradient then carries it
    f = scale * q.shape[-1] ** 0.5
    out, dq, dk, dv = _reference(q.double() * f, k, v, go, causal)
    return out, dq * f, dk, dv


@pytest.mark.parametrize("E,Dv", [(80, 80), (192, 128)])
def test_many_small_probabilities(E, Dv):
    """4096 keys of equal weight: probabilities of 2^-12, whose 16-bit parts would lie below fp16's normal range."""
    g = torch.Generator(device="cuda").manual_seed(E)
    q, k, v, go = (torch.randn(1, 2, 4096, d, generator=g, device="cuda").half() for d in (E, E, Dv, Dv))
    q = q * 0.02
    want = _reference(q, k, v, go, False)
    out, lse = T.sdpa_forward(q, k, v, force_path=_lib.PATH_GENERIC)
    new = T.sdpa_backward(go, q, k, v, out, lse)[:3]
    old = T.sdpa_backward(go, q, k, v, out, lse, force_path=_lib.PATH_GENERIC)[:3]
    T.check_device_status()
    for name, a, b, w in zip(("dq", "dk", "dv"), new, old, want[1:]):
        assert _error(a, w) <= 1.02 * _error(b, w), (name, _error(a, w), _error(b, w))


def test_gradients_that_are_all_zero_or_hold_an_infinity():
    q, k, v = (torch.randn(1, 2, 200, 80, device="cuda").half() for _ in range(3))
    out, lse = T.sdpa_forward(q, k, v)
    zero = T.sdpa_backward(torch.zeros_like(out), q, k, v, out, lse)[:3]
    assert all((g == 0).all() for g in zero)
    go = torch.randn_like(out)
    go[0, 0, 17, 3] = float("inf")
    got = T.sdpa_backward(go, q, k, v, out, lse)[:3]
    ref = T.sdpa_backward(go, q, k, v, out, lse, force_path=_lib.PATH_GENERIC)[:3]
    T.check_device_status()
    for a, b in zip(got, ref):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b))
        ok = torch.isfinite(b)
        torch.testing.assert_close(a[ok], b[ok], rtol=2e-3, atol=2e-3)
