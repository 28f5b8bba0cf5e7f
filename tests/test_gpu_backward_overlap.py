"""Backward calls back to back on one stream, each with its own data and all with the same scratch: the launches of a
call overlap each other and the next call's, and every kernel must see its own call's row statistics."""

import pytest
import torch

import torch_neuronx_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,Dv,dtype", [(64, 64, torch.bfloat16), (128, 128, torch.bfloat16), (80, 80, torch.float16),
                                        (192, 128, torch.float16), (256, 256, torch.bfloat16)])
@pytest.mark.parametrize("B,Hq,Hkv,L", [(1, 2, 1, 130), (2, 8, 2, 512)])   # fewer CTAs than SMs
def test_changing_data_at_one_scratch_address(E, Dv, dtype, B, Hq, Hkv, L):
    g = torch.Generator(device="cuda").manual_seed(E + L)
    calls, want = [], []
    for i in range(6):
        q, k, v, go = (torch.randn(B, h, L, d, generator=g, device="cuda").mul_(1 + i).to(dtype)
                       for h, d in ((Hq, E), (Hkv, E), (Hkv, Dv), (Hq, Dv)))
        out, lse = T.sdpa_forward(q, k, v, is_causal=True)
        calls.append((go, q, k, v, out, lse))
        torch.cuda.synchronize()
        want.append([t.clone() for t in T.sdpa_backward(*calls[-1], is_causal=True)[:3]])
        torch.cuda.synchronize()
    for _ in range(5):
        got = [[torch.empty_like(t) for t in w] for w in want]
        torch.cuda.synchronize()
        for c, o in zip(calls, got):
            T.sdpa_backward(*c, is_causal=True, grad_q=o[0], grad_k=o[1], grad_v=o[2])
        torch.cuda.synchronize()
        for o, w in zip(got, want):
            for a, b in zip(o, w):
                assert torch.equal(a, b)
    T.check_device_status()
