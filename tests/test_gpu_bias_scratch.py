"""The scratch that a copied bias takes belongs to its call, and a call whose scratch cannot be had runs without it."""

import subprocess
import sys

import pytest
import torch

import torch_neuronx_b200 as T
from torch_neuronx_b200 import ops

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


_FAILED_ALLOCATION = """
import sys, torch
import torch_neuronx_b200 as T
from torch_neuronx_b200 import _lib
g = torch.Generator(device="cuda").manual_seed(1)
q, k, v = (torch.randn(1, 8, 2049, 64, generator=g, device="cuda").bfloat16() for _ in range(3))
bias = torch.randn(1, 8, 2049, 2049, generator=g, device="cuda").bfloat16()   # its copy takes 68 MB
copied = T.sdpa_forward(q, k, v, attn_bias=bias)[0]
want = T.sdpa_forward(q, k, v, attn_bias=bias, force_path=_lib.PATH_GENERIC)[0]
assert not torch.equal(copied, want)
torch.cuda.synchronize()
torch.cuda.empty_cache()
total = torch.cuda.get_device_properties(0).total_memory
torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (32 << 20)) / total)
if sys.argv[1] == "aten":
    got = T.scaled_dot_product_attention(q, k, v, attn_mask=bias)
else:
    got = T.sdpa_forward(q, k, v, attn_bias=bias)[0]
torch.cuda.synchronize()
assert torch.equal(got, want)
"""


@pytest.mark.parametrize("entry", ["sdpa_forward", "aten"])
def test_a_failed_allocation_takes_the_kernel_that_needs_none(entry):
    """(in a process of its own, whose allocator holds nothing else that the copy could use)"""
    res = subprocess.run([sys.executable, "-c", _FAILED_ALLOCATION, entry], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
