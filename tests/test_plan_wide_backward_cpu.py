"""What b200_sdpa_bwd_query_plan() says about the kernels for head dimensions beyond 128 is what they launch."""

import ctypes as C

import pytest

from torch_neuronx_b200 import _lib


def _plan(E, Dv, dtype):
    B, Hq, Hkv, L, S = 2, 8, 4, 300, 520
    p = _lib.BwdParams()
    p.struct_size = C.sizeof(_lib.BwdParams)
    p.dtype, p.device, p.force_path = dtype, 0, _lib.PATH_AUTO
    for name in ("q", "k", "v", "out", "grad_out", "grad_q", "grad_k", "grad_v", "lse"):
        setattr(p, name, 4096)
    for name, h, n, d in (("q", Hq, L, E), ("grad_q", Hq, L, E), ("k", Hkv, S, E), ("grad_k", Hkv, S, E), ("v", Hkv, S, Dv),
                          ("grad_v", Hkv, S, Dv), ("out", Hq, L, Dv), ("grad_out", Hq, L, Dv)):
        getattr(p, name + "_stride")[:] = (h * n * d, n * d, d, 1)
    p.lse_stride[:] = (Hq * L, L, 1)
    p.B, p.Hq, p.Hkv, p.L, p.S, p.E, p.Dv, p.scale = B, Hq, Hkv, L, S, E, Dv, 0.1
    plan = _lib.Plan()
    plan.struct_size = C.sizeof(_lib.Plan)
    assert _lib.load().b200_sdpa_bwd_query_plan(C.byref(p), C.byref(plan)) == _lib.OK
    return plan


@pytest.mark.parametrize("dtype", [_lib.F16, _lib.BF16])
@pytest.mark.parametrize("E,Dv,smem", [
    # fixed operands of 128 rows, two tiles of the one streamed operand and one of the other, statistics, barriers
    (192, 128, 2 * (128 * 192 + 128 * 128 + 2 * 128 * 192 + 128 * 128) + 4 * 4 * 128 + 256),
    (256, 256, 2 * (128 * 256 + 128 * 256 + 2 * 64 * 256 + 64 * 256) + 4 * 4 * 64 + 256),
])
def test_geometry(E, Dv, smem, dtype):
    plan = _plan(E, Dv, dtype)
    assert plan.path == _lib.PATH_PREFILL and plan.launches == 3 and plan.threads == 576
    assert plan.grid_x == 3 * 8 * 2              # 128-row blocks x query heads x batches
    assert plan.grid_y == 2 * 5 * 4 * 2          # dK and dV: two CTAs per 128 keys of a (batch, kv head)
    assert plan.smem_bytes == smem
    assert plan.workspace_bytes >= 2 * 4 * 2 * 8 * 384
