"""The direct native entry points against the Python layer they stand in for: same bits, same plan, same errors."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(L, S, D=128, dtype=torch.bfloat16):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(L + S)
    q = torch.randn(2, 8, L, D, generator=g, device=dev, dtype=dtype)
    k, v = (torch.randn(2, 2, S, D, generator=g, device=dev, dtype=dtype) for _ in range(2))
    return q, k, v, torch.tensor([S, S // 2], dtype=torch.int32, device=dev)


def _both(monkeypatch, call):
    from torch_neuronx_b200 import _lib, ops

    assert _lib.native is not None, "build it with python -m torch_neuronx_b200.build"
    a = call()
    plan = dict(ops.last_plan)
    with monkeypatch.context() as m:
        m.setattr(_lib, "native", None)
        b = call()
        other = dict(ops.last_plan)
    torch.cuda.synchronize()
    for x, y in zip(a, b):
        assert (x is None and y is None) or (torch.equal(x, y) and x.stride() == y.stride() and x.dtype == y.dtype)
    return plan, other


@pytest.mark.parametrize("L,S", [(1, 300), (1, 1), (16, 300), (300, 300)])
def test_forward_and_attention(monkeypatch, L, S):
    import torch_neuronx_b200 as T

    q, k, v, lens = _inputs(L, S)
    plan, other = _both(monkeypatch, lambda: T.sdpa_forward(q, k, v, is_causal=L > 1, q_offset=S - L, kv_lens=lens))
    assert plan == other
    lse = torch.empty(2, 8, L, device=q.device)
    _both(monkeypatch, lambda: T.sdpa_forward(q, k, v, scale=0.3, out=torch.empty_like(q), lse=lse))
    _both(monkeypatch, lambda: T.sdpa_forward(q, k, v, need_lse=False))
    for args in (dict(kv_lens=lens), dict(is_causal=True), dict(is_causal=True, kv_lens=lens, scale=0.2)):
        _both(monkeypatch, lambda: (T.scaled_dot_product_attention(q, k, v, enable_gqa=True, **args),))
    qg = q.detach().requires_grad_()
    assert T.scaled_dot_product_attention(qg, k, v, enable_gqa=True).requires_grad
    assert T.scaled_dot_product_attention(qg, k, v, enable_gqa=True, kv_lens=lens).requires_grad


@pytest.mark.parametrize("layout", ["NHD", "HND", "dense"])
@pytest.mark.parametrize("rope", [False, True])
def test_decode(monkeypatch, layout, rope):
    import torch_neuronx_b200 as T

    q, k, v, _ = _inputs(1, 256)
    dev = q.device
    lens = torch.tensor([255, 17], dtype=torch.int32, device=dev)
    new = [torch.randn(2, 2, 128, device=dev, dtype=q.dtype) for _ in range(2)]
    cs = [torch.randn(256, 64, device=dev) for _ in range(2)] if rope else [None, None]
    kw = dict(need_lse=True, rope_cos=cs[0], rope_sin=cs[1])
    if layout == "dense":
        _both(monkeypatch, lambda: T.decode_append(q, *new, k, v, lens, **kw))
        return
    kp, vp = (t.reshape(32, 2, 16, 128) for t in (k, v))
    if layout == "NHD":
        kp, vp = (t.transpose(1, 2).contiguous() for t in (kp, vp))
    table = torch.randperm(32, device=dev).to(torch.int32).view(2, 16)
    _both(monkeypatch, lambda: T.paged_decode(q, kp, vp, table, lens, layout=layout, k_new=new[0], v_new=new[1], **kw))
    if not rope:
        _both(monkeypatch, lambda: T.paged_decode(q, kp, vp, table, lens, layout=layout))


def test_errors_are_the_python_layers():
    import torch_neuronx_b200 as T

    q, k, v, lens = _inputs(4, 64)
    with pytest.raises(RuntimeError, match="pass enable_gqa=True"):
        T.scaled_dot_product_attention(q, k, v)
    with pytest.raises(RuntimeError, match="kv_lens must be an int32 CUDA tensor"):
        T.scaled_dot_product_attention(q, k, v, enable_gqa=True, kv_lens=lens.long())
    with pytest.raises(RuntimeError, match="same dtype"):
        T.scaled_dot_product_attention(q, k.half(), v, enable_gqa=True)
    with pytest.raises(RuntimeError, match="go together"):
        T.decode_append(q[:, :, :1], None, k[:, :, 0], k, v, lens)
