"""Keys at or beyond kv_lens may hold anything in the tensor-core backward of head dimensions 72..128 and beyond 128:
the gradients of all rows are those of a tail of zeros, and the tail's own gradients are zero."""

import pytest
import torch

import torch_neuronx_b200 as T
from tests.test_gpu_padded_tails import _tensors, _with_tails

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("E,Dv", [(80, 80), (72, 128), (192, 128), (256, 256)])
@pytest.mark.parametrize("L,S", [(200, 300), (130, 513)])
def test_tails(E, Dv, L, S, causal, dtype):
    q, k, v = _tensors(4, 4, 2, L, S, E, Dv, dtype)
    lens = torch.tensor([1, S // 2 + 3, 64, S], dtype=torch.int32, device="cuda")
    go = torch.randn(4, 4, L, Dv, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(dtype)
    out, lse = T.sdpa_forward(q, _with_tails(k, lens, 0.0), _with_tails(v, lens, 0.0), kv_lens=lens, is_causal=causal,
                              q_offset=S - L)
    res = []
    for fill in (0.0, float("nan"), float("inf")):
        res.append(T.sdpa_backward(go, q, _with_tails(k, lens, fill), _with_tails(v, lens, fill), out, lse, kv_lens=lens,
                                   is_causal=causal, q_offset=S - L)[:3])
    T.check_device_status()
    for g in res[0]:
        assert torch.isfinite(g).all()
    for b, n in enumerate(lens.tolist()):
        assert (res[0][1][b, :, n:] == 0).all() and (res[0][2][b, :, n:] == 0).all()
    for other in res[1:]:
        for name, a, b in zip(("dq", "dk", "dv"), res[0], other):
            assert torch.equal(a, b), name
