"""Head dimensions between 64 and 128 on the tensor-core kernels' zero-filled 128-wide tiles: forward and backward
against the oracle at the edges of the k-steps (16), the copy boxes (64) and the row and key tiles (128)."""

import pytest
import torch

from oracle import sdpa_oracle as O
from tests.util import check_against_oracle, run_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("shape", [
    (2, 2, 2, 127, 129, 72, 72),
    (1, 4, 2, 300, 300, 80, 80),
    (1, 2, 1, 577, 577, 96, 96),
    (2, 2, 2, 129, 40, 120, 120),
    (1, 2, 2, 200, 260, 80, 128),
    (1, 4, 2, 130, 256, 128, 64),
    (1, 2, 2, 64, 200, 24, 88),
])
def test_padded_head_dims(shape, causal, dtype):
    import torch_neuronx_b200 as T

    B, Hq, Hkv, L, S, E, Dv = shape
    g = torch.Generator().manual_seed(sum(shape))
    q = torch.randn(B, Hq, L, E, generator=g).to(dtype)
    k = torch.randn(B, Hkv, S, E, generator=g).to(dtype)
    v = torch.randn(B, Hkv, S, Dv, generator=g).to(dtype)
    go = torch.randn(B, Hq, L, Dv, generator=g).to(dtype)
    lens = torch.tensor([S, max(1, S // 3)][:B], dtype=torch.int32) if B > 1 else None
    T.reset_launch_counts()
    out, lse = run_cuda(q, k, v, is_causal=causal, kv_lens=lens)
    assert T.launch_counts()["prefill"] == 1 and T.launch_counts()["generic"] == 0
    check_against_oracle(q, k, v, out, lse, is_causal=causal, kv_lens=lens, tag=f"{shape} causal={causal}")
    dev = torch.device("cuda", 0)
    ld = lens.to(dev) if lens is not None else None
    grads = [torch.full_like(t, float("nan"), device=dev) for t in (q, k, v)]
    T.sdpa_backward(go.to(dev), q.to(dev), k.to(dev), v.to(dev), out.to(dev), lse.to(dev), is_causal=causal, kv_lens=ld,
                    grad_q=grads[0], grad_k=grads[1], grad_v=grads[2])
    torch.cuda.synchronize()
    T.check_device_status()
    assert T.launch_counts()["bwd_prep"] == (1 if min(L, S) >= 64 else 0)   # a launch only the tensor-core kernels have
    want = O.sdpa_backward(go, q, k, v, out, lse, is_causal=causal, kv_lens=lens, compute_dtype=torch.float32)
    for got, ref, n in zip(grads, want[:3], ("dq", "dk", "dv")):
        assert not torch.isnan(got.float()).any(), n
        # P and dS are rounded to the 16-bit type once before their second product
        torch.testing.assert_close(got.cpu().float(), ref.float(), rtol=5e-2, atol=2e-2, msg=lambda m: f"{n} {shape}: {m}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_padded_head_dim_with_additive_bias(dtype):
    g = torch.Generator().manual_seed(9)
    q = torch.randn(1, 4, 200, 80, generator=g).to(dtype)
    k, v = (torch.randn(1, 2, 264, 80, generator=g).to(dtype) for _ in range(2))
    bias = (torch.randn(1, 4, 200, 264, generator=g) * 2).to(dtype)
    bias = bias.masked_fill(torch.rand(1, 4, 200, 264, generator=g) < 0.1, float("-inf"))
    out, lse = run_cuda(q, k, v, attn_bias=bias)
    check_against_oracle(q, k, v, out, lse, attn_mask=bias, tag="bias, head dim 80")
