"""The attention calls whose speed matters to a user of this package.

Every case goes through a public entry point, the way a program calls it:

* ``decode``   one generated token per sequence against a dense key/value cache
* ``paged``    a serving step: append the new token to a paged cache, rotate, attend
* ``extend``   a few to a few hundred new tokens per sequence behind a cached prefix
* ``prefill``  causal self-attention over a prompt, with or without right padding
* ``encoder``  bidirectional self-attention over short ragged sequences
* ``masked``   self-attention under a dense boolean mask or an additive bias
* ``train``    forward and backward through autograd

``listed()`` fixes one or two members of each family, ``draw()`` takes others from the same ranges.
"""

import math

import torch

import torch_neuronx_b200 as T

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}


def listed():
    return [
        # the next token of one chat: one sequence, a short cache; the time is launches and host work
        {"name": "decode_one", "kind": "decode", "dtype": "bf16", "B": 1, "Hq": 32, "Hkv": 8, "D": 128,
         "S": 2048, "lo": 2048, "hi": 2048},
        # the decode step of a full batch of unequal sequences: reads a gigabyte of cache
        {"name": "decode_ragged", "kind": "decode", "dtype": "bf16", "B": 64, "Hq": 32, "Hkv": 8, "D": 128,
         "S": 8192, "lo": 512, "hi": 8192},
        # one step of a serving engine: paged cache, append and rotary embedding in the call
        {"name": "paged_step", "kind": "paged", "dtype": "bf16", "B": 16, "Hq": 32, "Hkv": 8, "D": 128,
         "S": 4096, "lo": 128, "hi": 4000, "page": 16, "layout": "NHD", "interleaved": False},
        # eight proposed tokens per sequence checked against their cached prefixes
        {"name": "extend_verify", "kind": "extend", "dtype": "bf16", "B": 8, "Hq": 32, "Hkv": 8, "D": 128,
         "L": 8, "S": 4096},
        # prompt of a small multi-head model, head dimension 64
        {"name": "prefill_small", "kind": "prefill", "dtype": "bf16", "B": 8, "Hq": 12, "Hkv": 12, "D": 64,
         "L": 1024, "lo": 1024, "hi": 1024, "std": 0.5, "bshd": False},
        # a batch of padded prompts of a grouped-query model
        {"name": "prefill_padded", "kind": "prefill", "dtype": "bf16", "B": 4, "Hq": 32, "Hkv": 8, "D": 128,
         "L": 4096, "lo": 2048, "hi": 4096, "std": 1.0, "bshd": False},
        # one long prompt, stored as (B, S, H, D)
        {"name": "prefill_long", "kind": "prefill", "dtype": "bf16", "B": 1, "Hq": 32, "Hkv": 8, "D": 128,
         "L": 32768, "lo": 32768, "hi": 32768, "std": 1.0, "bshd": True},
        # an encoder over 577 positions: no size is a multiple of a tile, head dimension 80
        {"name": "encoder_odd", "kind": "encoder", "dtype": "fp16", "B": 16, "Hq": 16, "Hkv": 16, "D": 80,
         "L": 577},
        # a sliding window written as a dense boolean mask
        {"name": "masked_window", "kind": "masked", "dtype": "bf16", "B": 2, "Hq": 32, "Hkv": 8, "D": 128,
         "L": 2048, "mask": "window", "window": 512},
        # a training step of a grouped-query model
        {"name": "train_gqa", "kind": "train", "dtype": "bf16", "B": 2, "Hq": 32, "Hkv": 8, "E": 128, "Dv": 128,
         "L": 4096, "causal": True},
        # a training step with unequal query/key and value head dimensions
        {"name": "train_192_128", "kind": "train", "dtype": "bf16", "B": 1, "Hq": 24, "Hkv": 24, "E": 192, "Dv": 128,
         "L": 2048, "causal": True},
        # full precision, forward and backward
        {"name": "train_fp32", "kind": "train", "dtype": "fp32", "B": 2, "Hq": 8, "Hkv": 8, "E": 64, "Dv": 64,
         "L": 512, "causal": True},
    ]


def _between(rng, lo, hi):
    """A whole number spread evenly over the logarithm of its range."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _heads(rng):
    return rng.choice([(8, 8), (12, 12), (16, 16), (24, 6), (32, 32), (32, 8), (32, 4), (40, 8), (64, 8), (8, 1)])


def draw(rng):
    kind = rng.choice(["decode", "paged", "extend", "prefill", "encoder", "masked", "train", "train", "train"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    Hq, Hkv = _heads(rng)
    D = rng.choice([64, 128, 128])
    if kind in ("decode", "paged"):
        # up to 128 sequences and 32768 positions, the caches together below 3 GB
        S = _between(rng, 256, 32768)
        B = _between(rng, 1, max(1, min(128, int(3e9 / (4 * Hkv * D * S)))))
        hi = rng.randint(S // 2, S - 1)
        case = {"kind": kind, "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hkv, "D": D, "S": S,
                "lo": rng.randint(max(1, hi // 8), hi), "hi": hi}
        if kind == "paged":
            page = rng.choice([16, 32, 64])
            case.update(S=-(-S // page) * page, page=page, layout=rng.choice(["NHD", "HND"]),
                        interleaved=rng.random() < 0.3)
        return case
    if kind == "extend":
        L = _between(rng, 2, 512)
        S = _between(rng, 1024, 32768)
        B = _between(rng, 1, max(1, min(32, int(2e9 / (4 * Hkv * D * S)), int(1e12 / (4 * D * Hq * L * S)))))
        return {"kind": kind, "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hkv, "D": D, "L": L, "S": S}
    if kind == "prefill":
        L = _between(rng, 64, min(32768, int(math.sqrt(8.7e12 / (2 * D * Hq)))))
        B = _between(rng, 1, max(1, min(32, int(2e12 / (2 * D * Hq * L * L)))))
        lo = rng.choice([L, max(1, L // 2)])
        return {"kind": kind, "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hkv, "D": D, "L": L, "lo": lo, "hi": L,
                "std": 1.0, "bshd": rng.random() < 0.5}
    if kind == "encoder":
        L = _between(rng, 50, 2048)
        D = rng.choice([64, 64, 80, 96, 128])
        B = _between(rng, 1, max(1, min(64, int(5e11 / (4 * D * Hq * L * L)))))
        return {"kind": kind, "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hq, "D": D, "L": L}
    if kind == "masked":
        L = _between(rng, 128, 4096)
        B = _between(rng, 1, max(1, min(16, int(5e11 / (4 * D * Hq * L * L)))))
        mask = rng.choice(["window", "bias"])
        return {"kind": kind, "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hkv, "D": D, "L": L, "mask": mask,
                "window": _between(rng, 32, L) if mask == "window" else 0}
    what = rng.choice(["half", "half", "wide", "fp32"])
    if what == "fp32":
        L = _between(rng, 64, 2048)
        E = Dv = rng.choice([64, 128])
        most = 1e11
        dtype = "fp32"
    elif what == "wide":
        L = _between(rng, 128, 4096)
        E, Dv = rng.choice([(192, 128), (192, 128), (256, 256)])
        Hkv = Hq
        most = 1e12
    else:
        L = _between(rng, 128, 8192)
        E = Dv = rng.choice([64, 64, 80, 96, 128, 128, 128])
        most = 3e12
    causal = rng.random() < 0.7
    B = _between(rng, 1, max(1, min(16, int(most / (7 * (E + Dv) * Hq * L * L)))))
    return {"kind": "train", "dtype": dtype, "B": B, "Hq": Hq, "Hkv": Hkv, "E": E, "Dv": Dv, "L": L, "causal": causal}


# ---- what a program has in hand before the call ---------------------------------------------------


def _lengths(case):
    """Valid lengths of the sequences: evenly spaced from the shortest to the longest."""
    B, lo, hi = case["B"], case["lo"], case["hi"]
    return [hi - (hi - lo) * i // max(1, B - 1) for i in range(B)]


def _window_mask(L, window):
    i = torch.arange(L, device="cuda")
    return (i[None, :] <= i[:, None]) & (i[None, :] > i[:, None] - window)


def _alibi(Hq, L, dtype):
    """A causal linear bias with one slope per head, (1, Hq, L, L) in the query's type."""
    i = torch.arange(L, device="cuda", dtype=torch.float32)
    slope = torch.exp2(-8.0 * torch.arange(1, Hq + 1, device="cuda", dtype=torch.float32) / Hq)
    bias = (slope[:, None, None] * (i[None, :] - i[:, None])).to(dtype)
    return bias.masked_fill_(i[None, :] > i[:, None], float("-inf"))[None]


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype, B, Hq, Hkv = _DTYPES[case["dtype"]], case["B"], case["Hq"], case["Hkv"]

    def randn(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=dtype)

    def lengths():
        n = torch.tensor(_lengths(case), dtype=torch.int32, device="cuda")
        return n[torch.randperm(B, generator=g, device="cuda")].contiguous()

    kind = case["kind"]
    s = {"kind": kind}
    if kind == "decode":
        D, S = case["D"], case["S"]
        s.update(q=randn(B, Hq, 1, D), k=randn(B, Hkv, S, D), v=randn(B, Hkv, S, D), lens=lengths())
    elif kind == "paged":
        D, page = case["D"], case["page"]
        pages = case["S"] // page
        pool = (B * pages, page, Hkv, D) if case["layout"] == "NHD" else (B * pages, Hkv, page, D)
        turn = torch.arange(case["S"], device="cuda", dtype=torch.float32)[:, None] * torch.exp2(
            -torch.arange(0, D, 2, device="cuda", dtype=torch.float32) * (math.log2(10000.0) / D))
        s.update(q=randn(B, Hq, 1, D), k=randn(*pool), v=randn(*pool), lens=lengths(),
                 k_new=randn(B, Hkv, D), v_new=randn(B, Hkv, D), cos=turn.cos(), sin=turn.sin(),
                 table=torch.randperm(B * pages, generator=g, device="cuda").to(torch.int32).view(B, pages),
                 layout=case["layout"], interleaved=case["interleaved"])
    elif kind == "extend":
        D, L, S = case["D"], case["L"], case["S"]
        s.update(q=randn(B, Hq, L, D), k=randn(B, Hkv, S, D), v=randn(B, Hkv, S, D), offset=S - L)
    elif kind == "prefill":
        D, L = case["D"], case["L"]
        if case["bshd"]:
            q, k, v = (randn(B, L, h, D).transpose(1, 2) for h in (Hq, Hkv, Hkv))
        else:
            q, k, v = (randn(B, h, L, D) for h in (Hq, Hkv, Hkv))
        for t in (q, k, v):
            t.mul_(case["std"])
        s.update(q=q, k=k, v=v, lens=lengths() if case["lo"] < L else None)
    elif kind == "encoder":
        D, L = case["D"], case["L"]
        s.update(q=randn(B, Hq, L, D), k=randn(B, Hkv, L, D), v=randn(B, Hkv, L, D))
    elif kind == "masked":
        D, L = case["D"], case["L"]
        mask = _window_mask(L, case["window"]) if case["mask"] == "window" else _alibi(Hq, L, dtype)
        s.update(q=randn(B, Hq, L, D), k=randn(B, Hkv, L, D), v=randn(B, Hkv, L, D), mask=mask)
    else:
        E, Dv, L = case["E"], case["Dv"], case["L"]
        s.update(q=randn(B, Hq, L, E).requires_grad_(), k=randn(B, Hkv, L, E).requires_grad_(),
                 v=randn(B, Hkv, L, Dv).requires_grad_(), grad=randn(B, Hq, L, Dv), causal=case["causal"])
    return s


# ---- one pass -------------------------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind == "train":
        out = T.scaled_dot_product_attention(s["q"], s["k"], s["v"], is_causal=s["causal"], enable_gqa=True)
        return (out,) + torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["grad"])
    with torch.no_grad():
        if kind == "decode":
            return T.scaled_dot_product_attention(s["q"], s["k"], s["v"], enable_gqa=True, kv_lens=s["lens"])
        if kind == "paged":
            out, _, lens = T.paged_decode(
                s["q"], s["k"], s["v"], s["table"], s["lens"], layout=s["layout"], k_new=s["k_new"],
                v_new=s["v_new"], rope_cos=s["cos"], rope_sin=s["sin"], rope_interleaved=s["interleaved"])
            return out, lens, s["k"], s["v"]
        if kind == "extend":
            return T.sdpa_forward(s["q"], s["k"], s["v"], is_causal=True, q_offset=s["offset"], need_lse=False)[0]
        if kind == "prefill":
            return T.scaled_dot_product_attention(s["q"], s["k"], s["v"], is_causal=True, enable_gqa=True,
                                                  kv_lens=s["lens"])
        if kind == "encoder":
            return T.scaled_dot_product_attention(s["q"], s["k"], s["v"])
        return T.scaled_dot_product_attention(s["q"], s["k"], s["v"], attn_mask=s["mask"], enable_gqa=True)


# ---- what a pass cannot do without ----------------------------------------------------------------


def work(case):
    """Inputs read once and outputs written once; four operations per visible (query, key) pair and head
    element forward (two products), ten for the five products of the backward."""
    kind, e, B, Hq, Hkv = case["kind"], _BYTES[case["dtype"]], case["B"], case["Hq"], case["Hkv"]
    if kind in ("decode", "paged"):
        D, total = case["D"], sum(_lengths(case))
        if kind == "paged":
            total += B      # the appended rows: read as inputs, attended to, written to the cache
        nbytes = e * (2 * B * Hq * D + 2 * Hkv * D * total) + 4 * B
        if kind == "paged":
            nbytes += e * 2 * B * Hkv * D + 4 * B + 4 * sum(-(-n // case["page"]) for n in _lengths(case)) + 4 * B * D
        return {"bytes": nbytes, "flops": 4 * D * Hq * total}
    if kind == "extend":
        D, L, S = case["D"], case["L"], case["S"]
        pairs = B * Hq * (L * (S - L) + L * (L + 1) // 2)
        return {"bytes": e * D * (2 * B * Hq * L + 2 * B * Hkv * S), "flops": 4 * D * pairs}
    if kind == "train":
        E, Dv, L = case["E"], case["Dv"], case["L"]
        pairs = B * Hq * (L * (L + 1) // 2 if case["causal"] else L * L)
        # read q, k, v, grad; write out, grad_q, grad_k, grad_v
        nbytes = e * B * L * (2 * Hq * (E + Dv) + 2 * Hkv * (E + Dv))
        return {"bytes": nbytes, "flops": pairs * (2 * (E + Dv) + 2 * (3 * E + 2 * Dv))}
    D, L = case["D"], case["L"]
    nbytes, pairs = e * D * 2 * B * L * (Hq + Hkv), B * Hq * L * L
    if kind == "prefill":
        nbytes = e * D * 2 * (B * L * Hq + sum(_lengths(case)) * Hkv)
        pairs = Hq * sum(n * (n + 1) // 2 + (L - n) * n for n in _lengths(case))
    elif kind == "masked" and case["mask"] == "window":
        w = min(case["window"], L)
        nbytes += L * L
        pairs = B * Hq * (w * (w + 1) // 2 + (L - w) * w)
    elif kind == "masked":
        nbytes += e * Hq * L * L
        pairs = B * Hq * (L * (L + 1) // 2)
    return {"bytes": nbytes, "flops": 4 * D * pairs}


def tolerance(case):
    """Results and probabilities are rounded to the storage type once each: half a unit in the last place of
    bf16 is 2^-9 of the value, of fp16 2^-12; the gradients add a rounded softmax gradient."""
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]}
