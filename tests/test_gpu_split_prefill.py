"""The split form of the prefill kernel (rows of a kv head's query heads packed into a tile, key axis cut into ranges,
partials merged by a second launch) against the oracle: group sizes that do and do not divide 128, row counts around
the packed rows of a tile, key counts around the tile edge, ranges no row sees, sequences without keys."""

import pytest
import torch

from tests.util import check_against_oracle, make_qkv, run_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [
    # B, Hq, Hkv, L, S, D
    (1, 1, 1, 2, 129, 64),
    (2, 8, 2, 8, 1024, 128),
    (1, 10, 2, 26, 700, 128),      # five heads of 25 rows: one row in the second tile
    (1, 8, 1, 16, 2049, 64),
    (3, 4, 4, 33, 300, 128),
    (1, 16, 2, 100, 517, 128),
    (2, 6, 2, 130, 260, 64),
    (1, 128, 1, 3, 400, 64),       # a tile of one row of 128 heads
])
@pytest.mark.parametrize("mode", ["causal", "offset", "lens"])
def test_split_form(monkeypatch, shape, mode, dtype):
    import torch_neuronx_b200 as T

    monkeypatch.setenv("B200_SDPA_PREFILL", "split")
    B, Hq, Hkv, L, S, D = shape
    q, k, v = make_qkv(sum(shape), B, Hq, Hkv, L, S, D, dtype)
    kw = {"causal": dict(is_causal=True), "offset": dict(is_causal=True, q_offset=S - L),
          "lens": dict(kv_lens=torch.tensor([S - 1, 0, S // 2][:B], dtype=torch.int32))}[mode]
    T.reset_launch_counts()
    out, lse = run_cuda(q, k, v, **kw)
    counts = T.launch_counts()
    assert counts["prefill"] == 1 and counts["decode_combine"] == 1 and T.ops.last_plan["kv_splits"] > 1
    check_against_oracle(q, k, v, out, lse, tag=f"{shape} {mode}", **kw)
    again = run_cuda(q, k, v, **kw)
    assert torch.equal(out, again[0]) and torch.equal(lse, again[1])


def test_split_form_is_chosen_for_few_rows_only():
    import torch_neuronx_b200 as T

    q, k, v = make_qkv(5, 2, 8, 2, 8, 4096, 128, torch.bfloat16)
    out, lse = run_cuda(q, k, v, is_causal=True, q_offset=4088)
    assert T.ops.last_plan["kv_splits"] > 1
    check_against_oracle(q, k, v, out, lse, is_causal=True, q_offset=4088, tag="auto")
    q, k, v = make_qkv(5, 1, 8, 8, 256, 256, 128, torch.bfloat16)
    run_cuda(q, k, v)
    assert T.ops.last_plan["kv_splits"] == 1
