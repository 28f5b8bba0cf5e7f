"""Decode with the built-in scratch and the library's own choice of split, through the C ABI."""

import ctypes as C

import pytest
import torch

from tests.test_zz_no_alloc import _params

pytestmark = pytest.mark.gpu


def _stream(dev):
    return C.c_void_p(torch.cuda.current_stream(dev).cuda_stream)


@pytest.mark.parametrize("B,S", [(64, 4096), (64, 8192), (48, 16384)])
def test_built_in_scratch_with_the_library_s_split(B, S):
    """(the partials of the split that a workspace of any size would get take up to 25.6 MB here)"""
    from torch_neuronx_b200 import _lib

    lib = _lib.load()
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(S)
    q = torch.randn(B, 64, 1, 128, generator=g, device=dev, dtype=torch.bfloat16)
    k, v = (torch.randn(1, 8, S, 128, generator=g, device=dev, dtype=torch.bfloat16).expand(B, 8, S, 128) for _ in range(2))
    lens = torch.randint(1, S + 1, (B,), generator=g, device=dev).to(torch.int32)
    res = []
    for static in (True, False):
        out = torch.full((B, 64, 1, 128), float("nan"), device=dev, dtype=torch.bfloat16)
        lse = torch.full((B, 64, 1), float("nan"), device=dev)
        if static:
            p = _params(_lib, q, k, v, out, lse, lens, 0)
            rc = lib.b200_sdpa_decode_static(C.byref(p), _stream(dev))
        else:
            ws = torch.empty(64 << 20, dtype=torch.uint8, device=dev)
            p = _params(_lib, q, k, v, out, lse, lens, 0, workspace=ws)
            rc = lib.b200_sdpa_decode(C.byref(p), _stream(dev))
        assert rc == _lib.OK, _lib.strerror(rc)
        torch.cuda.synchronize()
        res.append((out, lse))
    # other splits of the keys: P is rounded against another maximum (2^-9 of bf16)
    torch.testing.assert_close(res[0][0].float(), res[1][0].float(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(res[0][1], res[1][1], rtol=1e-5, atol=1e-4)
