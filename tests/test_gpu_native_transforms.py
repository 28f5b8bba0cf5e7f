"""What the direct native entry points must leave to the dispatcher: forward-mode derivatives, tracing, functorch."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _qkv():
    g = torch.Generator(device="cuda").manual_seed(1)
    return tuple(torch.randn(1, 2, 32, 64, generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(3))


@pytest.mark.parametrize("lens", [False, True])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_forward_mode_derivatives_are_refused(which, lens):
    import torch.autograd.forward_ad as fw

    import torch_neuronx_b200 as T

    ts = list(_qkv())
    kw = {"kv_lens": torch.tensor([20], dtype=torch.int32, device="cuda")} if lens else {}
    with fw.dual_level():
        ts[which] = fw.make_dual(ts[which], torch.ones_like(ts[which]))
        with pytest.raises((NotImplementedError, RuntimeError)):   # no tangent is never an answer
            T.scaled_dot_product_attention(*ts, **kw)


@pytest.mark.filterwarnings("ignore")
def test_a_trace_records_the_call_or_is_refused():
    import torch_neuronx_b200 as T

    q, k, v = _qkv()
    try:
        traced = torch.jit.trace(lambda a, b, c: T.scaled_dot_product_attention(a, b, c), (q, k, v), check_trace=False)
    except Exception:
        return
    other = tuple(t.flip(2).contiguous() for t in (q, k, v))
    assert torch.equal(traced(*other), T.scaled_dot_product_attention(*other))


@pytest.mark.parametrize("transform", ["grad", "vjp", "jvp", "vmap"])
def test_inside_a_transform_of_something_else(transform):
    """q, k, v that the differentiated (or batched) input does not reach are plain tensors there."""
    import torch_neuronx_b200 as T

    q, k, v = _qkv()
    want = T.scaled_dot_product_attention(q, k, v).float().sum()
    x = torch.tensor(3.0, device="cuda")

    def f(t):
        return t * T.scaled_dot_product_attention(q, k, v).float().sum()

    if transform == "grad":
        got = torch.func.grad(f)(x)
    elif transform == "vjp":
        got = torch.func.vjp(f, x)[1](torch.ones_like(x))[0]
    elif transform == "jvp":
        got = torch.func.jvp(f, (x,), (torch.ones_like(x),))[1]
    else:
        got = torch.func.vmap(f)(torch.ones(2, device="cuda"))[1]
    torch.testing.assert_close(got, want)


def test_autocast_and_inference_mode_stay_on_the_direct_route():
    import torch_neuronx_b200 as T
    from torch_neuronx_b200 import _lib

    q, k, v = _qkv()
    want = T.scaled_dot_product_attention(q, k, v)
    # (a routing mode that another test may have installed for the process is none of this one's business)
    with torch._C.DisableTorchFunction(), torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        got = _lib.native.attention(q, k, v, False, None, False, None)
        assert got is not None and torch.equal(got, want)
    with torch._C.DisableTorchFunction(), torch.inference_mode():
        got = _lib.native.attention(q, k, v, False, None, False, None)
        assert got is not None and torch.equal(got, want)
