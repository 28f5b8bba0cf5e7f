"""The scratch that a copied bias takes belongs to its call, and a call whose scratch cannot be had runs without it."""

import pytest
import torch

import torch_neuronx_b200 as T
from torch_neuronx_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _inputs(L, dtype=torch.bfloat16, heads=4):
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = (torch.randn(1, heads, L, 64, generator=g, device="cuda").to(dtype) for _ in range(3))
    return q, k, v, torch.randn(1, heads, L, L, generator=g, device="cuda").to(dtype)


def test_nothing_is_kept():
    before = (len(ops._retired_workspaces), {k: w.numel() for k, w in ops._workspaces.items()})
    for L in (1001, 1003, 1101):
        q, k, v, bias = _inputs(L)
        T.sdpa_forward(q, k, v, attn_bias=bias)
        assert ops.last_plan["workspace_bytes"] > 4 * L * L * 2          # the copy was planned
    torch.cuda.synchronize()
    assert (len(ops._retired_workspaces), {k: w.numel() for k, w in ops._workspaces.items()}) == before


@pytest.mark.parametrize("entry", ["sdpa_forward", "aten"])
def test_a_failed_allocation_takes_the_kernel_that_needs_none(entry):
    q, k, v, bias = _inputs(2049, heads=8)   # a copy of 8 x 2049 x 2064 x 2 = 68 MB
    want, _ = T.sdpa_forward(q, k, v, attn_bias=bias, force_path=_lib.PATH_GENERIC)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (32 << 20)) / total)
    try:
        if entry == "aten":
            got = T.scaled_dot_product_attention(q, k, v, attn_mask=bias)
        else:
            got = T.sdpa_forward(q, k, v, attn_bias=bias)[0]
        torch.cuda.synchronize()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want)
