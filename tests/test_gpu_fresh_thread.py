"""A call from a thread that has made no CUDA call before (the backward of a program's first step runs on one)."""

import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_SCRIPT = """
import threading, torch
import torch_neuronx_b200 as T
q, k, v = (torch.randn(5, h, 276, 128, device="cuda", dtype=torch.bfloat16) for h in (40, 8, 8))
out, lse = T.sdpa_forward(q, k, v, is_causal=True)
go = torch.randn_like(out)
grads = [torch.empty_like(t) for t in (q, k, v)]
T.sdpa_backward(go, q, k, v, out, lse, is_causal=True, grad_q=grads[0], grad_k=grads[1], grad_v=grads[2])
torch.cuda.synchronize()   # all memory that the next call takes is in the allocator's cache now
want = [g.clone() for g in grads]
error = []
def call():
    try:
        T.sdpa_backward(go, q, k, v, out, lse, is_causal=True, grad_q=grads[0], grad_k=grads[1], grad_v=grads[2])
    except Exception as e:
        error.append(repr(e))
for g in grads:
    g.zero_()
torch.cuda.synchronize()
t = threading.Thread(target=call)
t.start()
t.join()
torch.cuda.synchronize()
assert not error, error
assert all(torch.equal(a, b) for a, b in zip(grads, want))
"""

_FIRST_STEP = """
import torch
import torch_neuronx_b200 as T
q, k, v = (torch.randn(5, h, 276, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for h in (40, 8, 8))
go = torch.randn(5, 40, 276, 128, device="cuda", dtype=torch.bfloat16)
out = T.scaled_dot_product_attention(q, k, v, is_causal=True, enable_gqa=True)
torch.autograd.grad(out, (q, k, v), go)
torch.cuda.synchronize()
"""


@pytest.mark.parametrize("script", [_SCRIPT, _FIRST_STEP], ids=["thread", "first_step"])
def test_call_on_a_thread_without_a_context(script):
    res = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
