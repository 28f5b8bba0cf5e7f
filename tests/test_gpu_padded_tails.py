"""Keys at or beyond kv_lens may hold anything, NaN and infinity included, on the zero-filled 128-wide tiles: they are
summed with a weight of exactly 0, and 0 x NaN is NaN."""

import pytest
import torch

import torch_neuronx_b200 as T
from torch_neuronx_b200 import ops

pytestmark = pytest.mark.gpu


def _tensors(B, Hq, Hkv, L, S, E, Dv, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + L + S + E)
    return tuple(torch.randn(B, h, n, d, generator=g, device="cuda").to(dtype)
                 for h, n, d in ((Hq, L, E), (Hkv, S, E), (Hkv, S, Dv)))


def _with_tails(t, lens, value):
    t = t.clone()
    for b, n in enumerate(lens.tolist()):
        t[b, :, n:] = value
    return t


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mode", ["per_cta", "persistent"])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("E,Dv,L,S", [(80, 80, 200, 300), (96, 96, 130, 257), (72, 128, 300, 640), (128, 64, 64, 200)])
def test_padded_head_dims(monkeypatch, E, Dv, L, S, causal, mode, dtype):
    monkeypatch.setenv("B200_SDPA_PREFILL", mode)
    q, k, v = _tensors(4, 4, 2, L, S, E, Dv, dtype)
    lens = torch.tensor([1, S // 2 + 3, 128, S], dtype=torch.int32, device="cuda")
    res = []
    for fill in (0.0, float("nan"), float("inf")):
        res.append(T.sdpa_forward(q, _with_tails(k, lens, fill), _with_tails(v, lens, fill), kv_lens=lens, is_causal=causal,
                                  q_offset=S - L))
        assert ops.last_plan["path"] == "generic" and ops.last_plan["threads"] in (320, 512)
    T.check_device_status()
    assert torch.isfinite(res[0][0]).all()
    for out, lse in res[1:]:
        assert torch.equal(out, res[0][0]) and torch.equal(lse, res[0][1])


@pytest.mark.parametrize("mode", ["auto", "persistent"])   # (a small bias is not looked over of itself)
@pytest.mark.parametrize("D,S,kind", [(80, 400, "dense"), (80, 400, "blocks"), (128, 401, "dense"), (64, 401, "blocks")])
def test_with_a_bias(monkeypatch, D, S, kind, mode):
    """(head dimensions 64 and 128: a layout that is copied first, which the same tiles serve)"""
    if mode != "auto":
        monkeypatch.setenv("B200_SDPA_PREFILL", mode)
    q, k, v = _tensors(2, 4, 2, 300, S, D, D, torch.bfloat16)
    lens = torch.tensor([260, 333], dtype=torch.int32, device="cuda")
    bias = torch.randn(300, S, device="cuda").to(torch.bfloat16)
    if kind == "blocks":                       # every second key tile hidden, also the one the keys of b = 1 end before
        bias[:, 128:256] = float("-inf")
        bias[:128, 384:] = float("-inf")
    res = [T.sdpa_forward(q, _with_tails(k, lens, x), _with_tails(v, lens, x), kv_lens=lens, attn_bias=bias)
           for x in (0.0, float("nan"))]
    T.check_device_status()
    assert torch.isfinite(res[0][0]).all()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
