"""A decode workspace on any 4-byte boundary, through the C ABI."""

import ctypes as C

import pytest
import torch

from tests.test_zz_no_alloc import _params

pytestmark = pytest.mark.gpu


def _stream(dev):
    return C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("shift", [4, 8, 12])
def test_workspace_on_a_4_byte_boundary(D, shift):
    from torch_neuronx_b200 import _lib

    lib = _lib.load()
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(D)
    q = torch.randn(2, 8, 1, D, generator=g, device=dev, dtype=torch.bfloat16)
    k, v = (torch.randn(2, 2, 1500, D, generator=g, device=dev, dtype=torch.bfloat16) for _ in range(2))
    lens = torch.tensor([1500, 700], dtype=torch.int32, device=dev)
    res = []
    for at in (0, shift):
        out = torch.full((2, 8, 1, D), float("nan"), device=dev, dtype=torch.bfloat16)
        lse = torch.full((2, 8, 1), float("nan"), device=dev)
        p = _params(_lib, q, k, v, out, lse, lens, 256)
        plan = _lib.Plan()
        plan.struct_size = C.sizeof(_lib.Plan)
        assert lib.b200_sdpa_query_plan(C.byref(p), C.byref(plan)) == _lib.OK
        ws = torch.empty(int(plan.workspace_bytes) + at, dtype=torch.uint8, device=dev)[at:]
        p = _params(_lib, q, k, v, out, lse, lens, 256, workspace=ws)
        assert lib.b200_sdpa_decode(C.byref(p), _stream(dev)) == _lib.OK
        torch.cuda.synchronize()
        res.append((out, lse))
    assert torch.isfinite(res[0][0]).all()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
