"""The tiled fp32 kernels against the oracle: both head dimensions, one row to several blocks of 32 / 64 rows with ragged
ends on both axes, grouped heads, right padding (a sequence without keys included), causal offsets, strided storage."""

import pytest
import torch

from oracle import sdpa_oracle as O
from tests.util import check_against_oracle, make_qkv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode", ["full", "causal", "offset", "lens"])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (1, 2, 2, 33, 31), (2, 4, 2, 64, 65), (2, 6, 3, 130, 97), (1, 2, 1, 31, 200),
                                   (3, 40, 8, 200, 260)])
def test_fp32_tiled(shape, mode, D):
    import torch_neuronx_b200 as T

    B, Hq, Hkv, L, S = shape
    q, k, v = make_qkv(sum(shape) + D, B, Hq, Hkv, L, S, D, torch.float32)
    go = torch.randn(B, Hq, L, D, generator=torch.Generator().manual_seed(D))
    kw = {"full": {}, "causal": dict(is_causal=True), "offset": dict(is_causal=True, q_offset=40, k_offset=70),
          "lens": dict(is_causal=True, kv_lens=torch.tensor([S - 1, S // 2, 0][:B], dtype=torch.int32))}[mode]
    dev = torch.device("cuda", 0)
    put = lambda t: t.to(dev).transpose(1, 2).contiguous().transpose(1, 2)   # noqa: E731  (B, S, H, D) storage
    qd, kd, vd, gd = put(q), put(k), put(v), go.to(dev)
    on = dict(kw, kv_lens=kw["kv_lens"].to(dev)) if "kv_lens" in kw else kw
    out = torch.full_like(qd, float("nan"))
    out, lse = T.sdpa_forward(qd, kd, vd, out=out, **on)
    assert T.ops.last_plan["threads"] == 128 and T.ops.last_plan["path"] in ("generic", "decode")
    grads = [torch.full_like(t, float("nan")) for t in (qd, kd, vd)]
    T.sdpa_backward(gd, qd, kd, vd, out, lse, grad_q=grads[0], grad_k=grads[1], grad_v=grads[2], **on)
    torch.cuda.synchronize()
    T.check_device_status()
    check_against_oracle(q, k, v, out.cpu(), lse.cpu(), tag=f"{shape} {mode} {D}", **kw)
    if mode == "offset":   # the oracle's backward takes the rule as a mask
        kw = dict(attn_mask=torch.where(torch.arange(S)[None] + 70 <= torch.arange(L)[:, None] + 40, 0.0, float("-inf")))
    want = O.sdpa_backward(go, q, k, v, out.cpu(), lse.cpu(), compute_dtype=torch.float32, **kw)
    for got, ref, n in zip(grads, want[:3], ("dq", "dk", "dv")):
        assert not torch.isnan(got).any(), n
        torch.testing.assert_close(got.cpu(), ref, rtol=1e-4, atol=1e-5, msg=lambda m: f"{n} {shape} {mode} {D}: {m}")
