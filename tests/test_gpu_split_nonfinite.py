"""NaN and infinity in q, k and v through the split form of the prefill kernel: the same rows are NaN, and the same
elements infinite, as in the form that walks all keys in one CTA."""

import pytest
import torch

from tests.util import make_qkv, run_cuda

pytestmark = pytest.mark.gpu


def _forms(monkeypatch, q, k, v, **kw):
    import torch_neuronx_b200 as T

    res = []
    for mode in ("split", "per_cta"):
        monkeypatch.setenv("B200_SDPA_PREFILL", mode)
        res.append(run_cuda(q, k, v, **kw))
        assert (T.ops.last_plan["kv_splits"] > 1) == (mode == "split")
    return res


@pytest.mark.parametrize("D,dtype", [(64, torch.float16), (128, torch.bfloat16)])
@pytest.mark.parametrize("shape", [(1, 8, 2, 8, 1000), (1, 4, 4, 300, 900)])    # one row tile (dual order), several
@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("spread", ["one", "every"])
def test_same_elements_as_the_plain_form(monkeypatch, shape, D, dtype, where, value, spread):
    B, Hq, Hkv, L, S = shape
    q, k, v = make_qkv(L + S, B, Hq, Hkv, L, S, D, dtype)
    if where == "q":
        q[0, 1, L // 2, 3] = value          # one row; a NaN there makes every one of its scores NaN
    else:
        t = k if where == "k" else v
        for key in ([S // 2] if spread == "one" else range(5, S, 64)):   # one range of the keys, or all of them
            t[0, 0, key, 7] = value
    (out, lse), (want, want_lse) = _forms(monkeypatch, q, k, v)
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    assert torch.equal(torch.isinf(out), torch.isinf(want))
    assert torch.equal(torch.isfinite(lse), torch.isfinite(want_lse))
    if where == "q":
        assert torch.isnan(out[0, 1, L // 2]).all()
    ok = torch.isfinite(want)
    torch.testing.assert_close(out[ok].float(), want[ok].float(), rtol=2e-2, atol=2e-2)


def test_rows_without_keys_stay_zero(monkeypatch):
    q, k, v = make_qkv(3, 2, 4, 2, 16, 700, 128, torch.bfloat16)
    lens = torch.tensor([0, 130], dtype=torch.int32)
    (out, lse), _ = _forms(monkeypatch, q, k, v, kv_lens=lens)
    assert (out[0] == 0).all() and (lse[0] == float("-inf")).all() and torch.isfinite(out[1]).all()
