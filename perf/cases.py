"""What a program that uses this library asks of it, as sizes to time and to check.

The product is one operator, forward attention on [B, H, S, D] 16-bit tensors: attention() and
attention_with_lse(), with the tile that get_tiling() names for the shape.  The listed cases run from one
call of two heads, which is all launch latency, to the 0.5 GiB tensors of the headline configuration;
draw() spreads further cases over the same ranges (head dimensions 16 to 256, sequences of 16 to 8192, one
head to thousands, both masks, both types, dense and [B, S, H, D] storage, with and without the
log-sum-exp).  Flops count the visible (query, key) pairs only; bytes are Q, K, V read once, O (and the
log-sum-exp) written once.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "ascend-rsfa_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ascend_rsfa.flash_attention_forward as fa  # noqa: E402

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_HEADS_D = (16, 32, 64, 64, 128, 128, 128, 256)


def _case(name, B, H, S, D, causal, scale, dtype="fp16", layout="bhsd", lse=False, std=1.0):
    c = {"B": B, "H": H, "S": S, "D": D, "causal": causal, "scale": scale, "dtype": dtype, "layout": layout,
         "lse": lse, "std": std}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # One call of two heads and one key tile: what a caller waits for when there is next to no work.
        _case("tiny", 1, 2, 128, 64, True, 0.5),
        # Windows or patches: thousands of independent sequences of 64, one small tile each.
        _case("windows_s64", 512, 8, 64, 64, False, 0.125),
        # The same with a ragged length, a small head dimension, bf16 and the causal mask.
        _case("short_ragged_d32", 256, 16, 100, 32, True, 1.0 / math.sqrt(32), dtype="bf16"),
        # Short sequences at the usual head dimension: as many bytes as arithmetic can hide behind.
        _case("short_s128", 512, 8, 128, 128, False, 1.0 / math.sqrt(128)),
        # A batch of two with four heads: fewer blocks of rows than the GPU has multiprocessors.
        _case("few_heads", 2, 4, 2048, 128, False, 0.5),
        # A training-size batch of short causal sequences with small heads.
        _case("causal_s512_d64", 4, 32, 512, 64, True, 0.125),
        # Prefill of a ragged length straight from a [B, S, H, D] projection, with the log-sum-exp kept.
        _case("prefill_ragged", 8, 16, 1000, 128, True, 1.0 / math.sqrt(128), dtype="bf16", layout="bshd", lse=True),
        # The headline configuration, whole: 1024 heads of 2048 x 128, near one-hot rows at this scale.
        _case("headline", 128, 8, 2048, 128, False, 0.5),
        # Its causal form at the share that one of eight GPUs gets.
        _case("headline_eighth_causal", 16, 8, 2048, 128, True, 0.5),
        # The largest head dimension.
        _case("wide_heads_causal", 64, 8, 1024, 256, True, 1.0 / 16),
        # Long causal sequences.
        _case("long_causal", 16, 16, 4096, 128, True, 1.0 / math.sqrt(128), dtype="bf16"),
        # Very long sequences with small heads and a wide range of scores.
        _case("very_long_d64", 4, 32, 8192, 64, False, 0.125, std=2.0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    D = rng.choice(_HEADS_D)
    S = _log_uniform(rng, 16, 8192)
    if rng.random() < 0.4:  # a round length, as most batches are padded to
        S = max(16, S // 64 * 64)
    H = rng.choice((1, 2, 3, 4, 8, 12, 16, 32))
    B = _log_uniform(rng, 1, 512)
    causal = rng.random() < 0.5
    # no more than the largest listed case, in scores (a head of 16 columns has as many as one of 64),
    # in arithmetic, and in bytes
    per_head = 4.0 * S * S * max(D, 64)
    cap = int(min(1.0e12 / per_head, 1.0e9 / (8.0 * S * D)))
    H = max(1, min(H, cap))
    B = max(1, min(B, cap // H))
    scale = 1.0 / math.sqrt(D) if rng.random() < 0.75 else 0.5
    return _case(None, B, H, S, D, causal, scale, dtype=rng.choice(("fp16", "bf16")),
                 layout=rng.choice(("bhsd", "bhsd", "bshd")), lse=rng.random() < 0.3,
                 std=rng.choice((0.5, 1.0, 1.0, 2.0) if D <= 64 else (0.5, 1.0, 1.0)))


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    B, H, S, D = case["B"], case["H"], case["S"], case["D"]
    shape = (B, H, S, D) if case["layout"] == "bhsd" else (B, S, H, D)
    out = []
    for _ in range(3):
        t = torch.randn(shape, generator=g, device="cuda", dtype=_DTYPES[case["dtype"]])
        if case["std"] != 1.0:
            t *= case["std"]
        out.append(t if case["layout"] == "bhsd" else t.transpose(1, 2))
    return out


def prepare(case, seed):
    q, k, v = _inputs(case, seed)
    # the tile is looked up once for a shape, as the reference's own benchmark does
    tile = fa.get_tiling(case["B"], case["H"], case["S"], case["D"], case["causal"])
    return {"q": q, "k": k, "v": v, "tile": tile, "causal": case["causal"], "scale": case["scale"],
            "lse": case["lse"]}


def run(state):
    bm, bn = state["tile"]
    if state["lse"]:
        return fa.attention_with_lse(state["q"], state["k"], state["v"], state["causal"], state["scale"], bm, bn)
    return fa.attention(state["q"], state["k"], state["v"], state["causal"], state["scale"], bm, bn)


def work(case):
    B, H, S, D = case["B"], case["H"], case["S"], case["D"]
    pairs = S * (S + 1) // 2 if case["causal"] else S * S
    nbytes = 4 * B * H * S * D * 2 + (4 * B * H * S if case["lse"] else 0)
    return {"bytes": nbytes, "flops": 4 * B * H * pairs * D}


def tolerance(case):
    # The weights and the result are rounded to 16 bits.  Measured against 64-bit sums over these cases:
    # 2.2e-4 to 2.9e-4 in fp16, 1.6e-3 to 2.1e-3 in bf16; four times that is allowed.
    return {"rel": 1.2e-3, "max": 2e-2} if case["dtype"] == "fp16" else {"rel": 8.5e-3, "max": 1.5e-1}


def exact(case, seed):
    q, k, v = _inputs(case, seed)
    B, H, S, D = case["B"], case["H"], case["S"], case["D"]
    o = torch.empty((B, H, S, D), dtype=torch.float64, device="cuda")
    lse = torch.empty((B, H, S), dtype=torch.float64, device="cuda") if case["lse"] else None
    hidden = torch.ones((S, S), dtype=torch.bool, device="cuda").triu(1) if case["causal"] else None
    step = max(1, int(1.0e9 / (8.0 * S * S)))
    for b in range(B):
        for h in range(0, H, step):
            s = q[b, h:h + step].double() @ k[b, h:h + step].double().transpose(-1, -2)
            s *= case["scale"]
            if hidden is not None:
                s.masked_fill_(hidden, -math.inf)
            if lse is not None:
                lse[b, h:h + step] = torch.logsumexp(s, dim=-1)
            o[b, h:h + step] = torch.softmax(s, dim=-1) @ v[b, h:h + step].double()
    return (o, lse) if case["lse"] else o
