"""A NaN query row in the tiled fp32 backward: its own gradient and what it adds to the keys' are NaN, as in the
CUDA-core kernels, although its log-sum-exp reads as that of a row without keys."""

import pytest
import torch

import torch_neuronx_b200 as T
from torch_neuronx_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_nan_row(D, causal):
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v, go = (torch.randn(1, 2, 150, D, generator=g, device="cuda") for _ in range(4))
    q[0, 1, 70, 5] = float("nan")
    res = []
    for path in (_lib.PATH_AUTO, _lib.PATH_GENERIC):
        out, lse = T.sdpa_forward(q, k, v, is_causal=causal, force_path=path)
        res.append((out, lse) + T.sdpa_backward(go, q, k, v, out, lse, is_causal=causal, force_path=path)[:3])
    T.check_device_status()
    assert torch.isnan(res[0][0][0, 1, 70]).all() and torch.isnan(res[0][2][0, 1, 70]).all()
    # keys that the row does not see: 0 x NaN reaches those that share a tile with it, and the kernels' tiles differ
    seen = 71 if causal else 150
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), *res):
        if name in ("dk", "dv"):
            a, b = a[:, :, :seen], b[:, :, :seen]
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)), name
