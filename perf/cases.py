"""The calls whose time counts: what a program that uses this package has it do.

Every case is one call of a public entry point (`flash_colsum`, `flash_colsum_causal`,
`flash_colsum_host`, `topk_columns`, `threshold_columns`) on inputs that are already where such a
program has them.  `listed()` holds the representative ones, `draw()` more of the same ranges.

A case is a dict with
    op      "encoder"   non-causal, every query row enters the mean (cls = 0) or the first `cls` do
            "causal"    the queries are the last Q of K keys: prompt suffix, decode step, prefill
            "host"      "encoder" on pinned host memory, result on the host
            "topk" / "threshold"   the pruning step on column means
    B, H, Q, K, D, dtype           sizes (encoder: Q = K) and element type of query and key
    layout  "bhsd": contiguous (B, H, S, D); "bshd": a (B, S, H, D) projection output seen as
            (B, H, S, D) through transpose(1, 2), as attention modules hand it over
    outliers  keys scaled by per-position factors in [0.5, 2]: a few columns draw most attention
"""

import math

import torch

from flash_colsum_b200 import (flash_colsum, flash_colsum_causal, flash_colsum_host, threshold_columns,
                               topk_columns)

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}


def _attention(op, B, H, Q, K, D, dtype, cls=0, layout="bhsd", outliers=False, name=None):
    case = {"op": op, "B": B, "H": H, "Q": Q, "K": K, "D": D, "dtype": dtype, "cls": cls, "layout": layout,
            "outliers": outliers}
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # a small batch in the precision a model is debugged in: the call is all latency
        _attention("encoder", 2, 4, 256, 256, 64, "fp32", name="encoder small fp32"),
        # token importance of a text or image encoder, the headline size
        _attention("encoder", 8, 16, 2048, 2048, 64, "fp16", name="encoder batch"),
        # token pruning by CLS attention: 1 + 24 x 24 patches, one query row enters the mean
        _attention("encoder", 32, 16, 577, 577, 64, "fp16", cls=1, name="patches cls row"),
        # the same patches by the mean over all rows: a ragged length, strided projection outputs
        _attention("encoder", 32, 16, 577, 577, 64, "bf16", layout="bshd", name="patches all rows"),
        # one very long document: the longest ordinary point of the single-sample sweep
        _attention("encoder", 1, 16, 131072, 131072, 64, "fp16", name="single long"),
        # cache pruning after a prompt: the last 128 queries against a few thousand keys
        _attention("causal", 1, 32, 128, 4096, 128, "fp16", name="suffix short"),
        # cache pruning of a long context, with outlier columns
        _attention("causal", 1, 32, 512, 131072, 128, "bf16", outliers=True, name="suffix long"),
        # one decode step over a grown cache: reads the keys once
        _attention("causal", 1, 32, 1, 32768, 128, "bf16", name="decode step"),
        # a batch of prompts, every token is a query; no multiple of any tile
        _attention("causal", 4, 32, 2000, 2000, 128, "bf16", name="prefill batch"),
        # the headline size from a data loader's pinned buffers, result back on the host
        _attention("host", 8, 16, 2048, 2048, 64, "fp16", name="encoder batch from host"),
        # the pruning step: the most attended eighth of a long cache ...
        {"op": "topk", "B": 1, "K": 131072, "keep": 16384, "name": "topk long"},
        # ... and the patches with more than a uniform share
        {"op": "threshold", "B": 32, "K": 577, "share": 1.0, "name": "threshold patches"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _dtype(rng):
    return rng.choice(("fp16", "fp16", "fp16", "bf16", "bf16", "bf16", "fp32"))


def draw(rng):
    kind = rng.choice(("encoder", "encoder", "cls", "single", "suffix", "suffix", "decode", "prefill", "host", "topk",
                       "threshold"))
    if kind == "topk":
        B, K = _log_int(rng, 1, 64), _log_int(rng, 64, 262144)
        return {"op": "topk", "B": B, "K": K, "keep": max(1, int(K * rng.uniform(0.05, 0.75)))}
    if kind == "threshold":
        return {"op": "threshold", "B": _log_int(rng, 1, 64), "K": _log_int(rng, 64, 262144),
                "share": rng.choice((0.5, 1.0, 2.0))}
    layout = rng.choice(("bhsd", "bhsd", "bshd"))
    if kind == "single":
        S = _log_int(rng, 1024, 32768)
        return _attention("encoder", 1, rng.choice((8, 12, 16)), S, S, rng.choice((64, 64, 80, 128)), _dtype(rng),
                          layout=layout)
    if kind in ("suffix", "decode"):
        H, D = rng.choice((8, 16, 32)), rng.choice((64, 128, 128))
        K = _log_int(rng, 512, 131072)
        Q = rng.randint(1, 4) if kind == "decode" else min(K, _log_int(rng, 5, 1024))
        return _attention("causal", 1, H, Q, K, D, rng.choice(("fp16", "bf16")), outliers=rng.random() < 0.5)
    if kind == "prefill":
        B, H, K = _log_int(rng, 1, 8), rng.choice((8, 16, 32)), _log_int(rng, 128, 8192)
        Q = K if rng.random() < 0.6 else max(1, int(K * rng.uniform(0.2, 0.9)))   # (Q < K: a chunk of a prompt)
        return _attention("causal", B, H, Q, K, rng.choice((64, 80, 128)), rng.choice(("fp16", "bf16")), layout=layout)
    B, H, S = _log_int(rng, 2, 64), rng.choice((4, 8, 12, 16)), _log_int(rng, 64, 4096)
    D = rng.choice((32, 64, 64, 64, 80, 96, 128))
    while B > 2 and B * H * S > 8 * 16 * 4096:      # (as many rows as twice the headline size has)
        B //= 2
    if kind == "host":
        return _attention("host", B, H, min(S, 2048), min(S, 2048), D, rng.choice(("fp16", "bf16")))
    cls = min(S, rng.choice((1, 1, _log_int(rng, 1, 128)))) if kind == "cls" else 0
    return _attention("encoder", B, H, S, S, D, _dtype(rng), cls=cls, layout=layout)


def _operand(case, rows, gen):
    B, H, D = case["B"], case["H"], case["D"]
    dtype = _DTYPES[case["dtype"]]
    if case["layout"] == "bshd":
        return torch.randn((B, rows, H, D), generator=gen, device="cuda", dtype=dtype).transpose(1, 2)
    return torch.randn((B, H, rows, D), generator=gen, device="cuda", dtype=dtype)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["op"] in ("topk", "threshold"):
        # column means: positive, rows summing to one, a heavy upper tail
        x = torch.randn((case["B"], case["K"]), generator=gen, device="cuda").exp_()
        return {"case": case, "colsum": x / x.sum(dim=1, keepdim=True)}
    q = _operand(case, case["Q"], gen)
    k = _operand(case, case["K"], gen)
    if case["outliers"]:
        k.mul_((0.5 + 1.5 * torch.rand((1, 1, case["K"], 1), generator=gen, device="cuda")).to(k.dtype))
    if case["op"] == "host":
        q, k = q.cpu().pin_memory(), k.cpu().pin_memory()
    return {"case": case, "q": q, "k": k, "cls": case["cls"] or None}


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "topk":
        return topk_columns(state["colsum"], case["keep"])
    if op == "threshold":
        return threshold_columns(state["colsum"], case["share"], relative=True)
    if op == "host":
        return flash_colsum_host(state["q"], state["k"])
    if op == "encoder":
        return flash_colsum(state["q"], state["k"], cls_len=state["cls"])
    if case["B"] == 1:
        return flash_colsum(state["q"], state["k"], is_causal=True)
    return flash_colsum_causal(state["q"], state["k"])


def work(case):
    """Inputs once, outputs once; two operations per element of every visible score's dot product
    (the scores of one pass: what any algorithm has to form)."""
    B, K = case["B"], case["K"]
    if case["op"] == "topk":
        return {"bytes": B * (4 * K + 8 * case["keep"]), "flops": 0}
    if case["op"] == "threshold":
        return {"bytes": B * (4 * K + 4 * K + 4), "flops": 0}
    H, D = case["H"], case["D"]
    rows = min(case["cls"], case["Q"]) if case["cls"] else case["Q"]
    scores = rows * K if case["op"] != "causal" else rows * K - rows * (rows - 1) // 2
    size = 4 if case["dtype"] == "fp32" else 2
    return {"bytes": B * H * (rows + K) * D * size + 4 * B * K, "flops": 2 * B * H * scores * D}


def tolerance(case):
    if case["op"] in ("topk", "threshold"):
        return "exact"
    # exps of relative accuracy 1e-4, summed in fp32; a form that holds the exps of a tile as fp16 is as good
    return {"rel": 2e-4, "max": 2e-3}
