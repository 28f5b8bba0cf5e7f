"""Additive biases on the tensor-core kernels: hidden key tiles left out, unreadable layouts copied first."""

import pytest
import torch

import torch_neuronx_b200 as T
from torch_neuronx_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _bias(kind, B, Hq, L, S, dtype, g):
    i = torch.arange(L, device="cuda")[:, None]
    j = torch.arange(S, device="cuda")[None, :]
    if kind == "window":            # (L, S), broadcast over batch and heads
        keep = (j <= i + (S - L)) & (j > i + (S - L) - 100)
    elif kind == "blocks":          # per batch: whole tiles on and off, 256 rows of the first one without any key
        on = torch.rand(B, 1, -(-L // 128), -(-S // 128), generator=g, device="cuda") < 0.4
        on[0, :, :2] = False
        keep = on.repeat_interleave(128, 2).repeat_interleave(128, 3)[:, :, :L, :S]
    elif kind == "heads":           # per head
        keep = (j <= i) & (torch.arange(Hq, device="cuda")[:, None, None] % 3 != j // 256)
    elif kind == "single":          # one visible element in a tile: its last
        keep = torch.zeros(L, S, dtype=torch.bool, device="cuda")
        keep[:, 0] = True
        keep[min(L, 128) - 1, min(S, 384) - 1] = True
    else:                           # "row": one bias row for all query rows, per batch
        keep = torch.arange(S, device="cuda") < torch.linspace(S // 5, S, B, device="cuda").view(B, 1, 1, 1)
    val = torch.randn(keep.shape, generator=g, device="cuda").to(dtype)
    return val.masked_fill(~keep, float("-inf"))


def _qkv(B, Hq, Hkv, L, S, D, dtype, g):
    return (torch.randn(B, h, n, D, generator=g, device="cuda").to(dtype) for h, n in ((Hq, L), (Hkv, S), (Hkv, S)))


KINDS = ["window", "blocks", "heads", "single", "row"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize(
    "D,dtype,B,Hq,Hkv,L,S,causal",
    [
        (128, torch.bfloat16, 2, 8, 2, 640, 640, False),
        (128, torch.bfloat16, 1, 6, 6, 1000, 1000, True),
        (128, torch.float16, 1, 4, 2, 130, 8192, False),
        (64, torch.bfloat16, 2, 4, 4, 777, 520, False),
        (64, torch.float16, 1, 4, 2, 512, 512, True),
        (80, torch.bfloat16, 2, 6, 6, 300, 904, False),
    ],
)
def test_same_bits_as_every_tile(kind, D, dtype, B, Hq, Hkv, L, S, causal, monkeypatch):
    """A hidden tile adds exact zeros, so leaving it out changes no bit."""
    g = torch.Generator(device="cuda").manual_seed(D + L + S)
    q, k, v = _qkv(B, Hq, Hkv, L, S, D, dtype, g)
    bias = _bias(kind, B, Hq, L, S, dtype, g)
    monkeypatch.setenv("B200_SDPA_PREFILL", "persistent")   # (small problems are not looked over of themselves)
    got = T.sdpa_forward(q, k, v, attn_bias=bias, is_causal=causal)
    assert ops.last_plan["launches"] == 2
    monkeypatch.setenv("B200_SDPA_PREFILL", "per_cta")
    want = T.sdpa_forward(q, k, v, attn_bias=bias, is_causal=causal)
    assert ops.last_plan["launches"] == 1
    T.check_device_status()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert torch.isfinite(got[0]).all()


def test_nan_in_the_bias_is_not_hidden(monkeypatch):
    q, k, v = _qkv(1, 2, 2, 256, 512, 128, torch.bfloat16, torch.Generator(device="cuda").manual_seed(0))
    bias = torch.full((256, 512), float("-inf"), device="cuda", dtype=torch.bfloat16)
    bias[:, 0] = 0
    bias[200, 300] = float("nan")
    monkeypatch.setenv("B200_SDPA_PREFILL", "persistent")
    out = T.sdpa_forward(q, k, v, attn_bias=bias)[0]
    assert torch.isnan(out[:, :, 200]).all() and torch.isfinite(out[:, :, :200]).all()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize(
    "D,dtype,B,Hq,Hkv,L,S,causal,layout",
    [
        (128, torch.bfloat16, 2, 8, 2, 641, 641, False, "plain"),     # rows off the 16-byte grid
        (64, torch.bfloat16, 2, 4, 4, 300, 1003, True, "plain"),
        (64, torch.float16, 1, 4, 2, 16, 130, False, "plain"),        # fewer than four key tiles
        (96, torch.float16, 1, 4, 4, 257, 2050, False, "plain"),
        (128, torch.float16, 1, 4, 1, 260, 512, False, "shifted"),    # base off the grid
        (128, torch.bfloat16, 1, 4, 2, 512, 640, False, "transposed"),
    ],
)
def test_unreadable_layouts(kind, D, dtype, B, Hq, Hkv, L, S, causal, layout):
    """Against the CUDA-core kernel (fp32 probabilities) and float64: no further off than that kernel, but for the
    randomness of the roundings of the result (2 %)."""
    g = torch.Generator(device="cuda").manual_seed(D + L + S)
    q, k, v = _qkv(B, Hq, Hkv, L, S, D, dtype, g)
    bias = _bias(kind, B, Hq, L, S, dtype, g)
    if layout == "shifted":
        buf = torch.empty(*bias.shape[:-1], S + 8, device="cuda", dtype=dtype)
        bias = buf[..., 1 : S + 1].copy_(bias)
    elif layout == "transposed":
        bias = bias.transpose(-1, -2).contiguous().transpose(-1, -2)
    out, lse = T.sdpa_forward(q, k, v, attn_bias=bias, is_causal=causal)
    if not (kind == "row" and layout == "transposed"):   # (a single row has no other layout and is read in place)
        assert ops.last_plan["path"] == "generic" and ops.last_plan["threads"] in (320, 512)
    else:
        return
    ref, ref_lse = T.sdpa_forward(q, k, v, attn_bias=bias, is_causal=causal, force_path=_lib.PATH_GENERIC)
    T.check_device_status()
    s = q.double() @ k.double().repeat_interleave(Hq // Hkv, 1).transpose(-1, -2) * D**-0.5 + bias.double()
    if causal:
        s = s.masked_fill(~torch.ones(L, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.softmax(s, -1).nan_to_num(0.0) @ v.double().repeat_interleave(Hq // Hkv, 1)
    err = [(o.double() - want).norm().item() for o in (out, ref)]
    assert err[0] <= 1.02 * err[1], err
    assert torch.equal(torch.isinf(lse), torch.isinf(ref_lse))
    # the statistics differ by the order of the sums only
    torch.testing.assert_close(lse, ref_lse, rtol=1e-5, atol=1e-4)
