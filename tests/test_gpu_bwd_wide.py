"""Tensor-core backward at head dimensions 192/128 and 256 against the oracle: one to several tiles of either
operand, ragged ends at the streamed tile sizes (128 and 64), grouped heads, right padding, (B, S, H, D) storage."""

import pytest
import torch

from oracle import sdpa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dims", [(192, 128), (256, 256)])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (1, 4, 2, 63, 129), (2, 2, 1, 65, 64), (1, 2, 2, 128, 256),
                                   (2, 6, 3, 300, 130), (1, 2, 1, 520, 700)])
def test_wide_backward(shape, dims, causal, dtype):
    import torch_neuronx_b200 as T

    B, Hq, Hkv, L, S = shape
    E, Dv = dims
    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(sum(shape) + E)
    q = torch.randn(B, L, Hq, E, generator=g).to(dtype).transpose(1, 2)
    k = torch.randn(B, Hkv, S, E, generator=g).to(dtype)
    v = torch.randn(B, S, Hkv, Dv, generator=g).to(dtype).transpose(1, 2)
    go = torch.randn(B, Hq, L, Dv, generator=g).to(dtype)
    lens = torch.tensor([max(0, S - 40), S][:B], dtype=torch.int32) if B > 1 else None
    ld = lens.to(dev) if lens is not None else None
    qd, kd, vd = q.to(dev), k.to(dev), v.to(dev)
    out, lse = T.sdpa_forward(qd, kd, vd, is_causal=causal, kv_lens=ld)
    grads = [torch.full_like(t, float("nan")) for t in (qd, kd, vd)]
    T.reset_launch_counts()
    T.sdpa_backward(go.to(dev), qd, kd, vd, out, lse, is_causal=causal, kv_lens=ld,
                    grad_q=grads[0], grad_k=grads[1], grad_v=grads[2])
    torch.cuda.synchronize()
    T.check_device_status()
    counts = T.launch_counts()
    assert counts["bwd_prep"] == counts["bwd_dq"] == counts["bwd_dkv"] == 1
    want = O.sdpa_backward(go, q, k, v, out.cpu(), lse.cpu(), is_causal=causal, kv_lens=lens, compute_dtype=torch.float32)
    for got, ref, n in zip(grads, want[:3], ("dq", "dk", "dv")):
        assert not torch.isnan(got.float()).any(), n
        # P and dS are rounded to the 16-bit type once before their second product
        torch.testing.assert_close(got.cpu().float(), ref.float(), rtol=5e-2, atol=2e-2, msg=lambda m: f"{n}: {m}")
