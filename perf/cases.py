"""The attention work that is timed: one case per way in which a model's code calls `tyr_b200.nn`.

A case is a dict of plain values; "path" says which calls one pass makes:

  token   one step of a generating loop over a dense KV cache: norm + rotary of the new query, norm + rotary +
          append of the new key, append of the new value, single-token attention over the cache
  step    the same attention through the typed call on a cache slice (q_seq = 1)
  decode  one token for each of many sequences with caches of their own lengths
  append  the prologue of a whole prompt: norm + rotary + layout of Q, K and V, K and V into the cache
  prefill the typed attention calls on a prompt (q_seq = kv_seq causal or not, q_seq != kv_seq not causal)
  padded  the typed call with a padding mask over a batch of prompts of different lengths
  window  the typed call with a sliding window
  train   forward with the row statistics, then dQ, dK and dV

Model shapes are the repository's own: a char-level GPT (6 heads of 64), Qwen3-0.6B and Qwen3-8B (grouped-query
attention, heads of 128, Q and K normalised per head), Flux (24 heads of 128, joint attention without a mask).
"""
from __future__ import annotations

import math
import random

import torch

from tyr_b200 import nn

# query heads, KV heads, head_dim, Q and K normalised per head
SHAPES = {
    "char": (6, 6, 64, False),
    "mha64": (12, 12, 64, False),
    "gqa64": (32, 8, 64, False),
    "qwen3_0p6b": (16, 8, 128, True),
    "qwen3_8b": (32, 8, 128, True),
    "flux": (24, 24, 128, True),
}


def listed():
    return [
        # one user, one token: four launches' worth of host work around a few microseconds of device work
        {"name": "token_one_sequence", "path": "token", "shape": "qwen3_8b", "batch": 1, "cap": 4096, "len": 1537,
         "ragged": False},
        # the reference's own generating loop: the typed call with one query row on a slice of the cache
        {"name": "step_typed_call", "path": "step", "shape": "qwen3_0p6b", "batch": 4, "cap": 4096, "len": 2051},
        # a serving batch: the benchmark's ragged 64 sequences (4.8 GB of KV)
        {"name": "decode_64_ragged", "path": "decode", "shape": "qwen3_8b", "batch": 64, "min_len": 512,
         "max_len": 32768, "len_seed": 3},
        # the prompt's prologue in one layer: Q, K and V of four prompts of 4096 tokens
        {"name": "append_prompt", "path": "append", "shape": "qwen3_8b", "batch": 4, "seq": 4096, "cap": 4608,
         "rotary": "half"},
        # one chat prompt of odd length: latency, few work items
        {"name": "prefill_one_prompt", "path": "prefill", "shape": "qwen3_8b", "batch": 1, "q_seq": 517, "kv_seq": 517,
         "causal": True},
        # the benchmark's three long forward shapes
        {"name": "prefill_qwen3_0p6b", "path": "prefill", "shape": "qwen3_0p6b", "batch": 8, "q_seq": 2048,
         "kv_seq": 2048, "causal": True},
        {"name": "prefill_qwen3_8b", "path": "prefill", "shape": "qwen3_8b", "batch": 4, "q_seq": 8192,
         "kv_seq": 8192, "causal": True},
        {"name": "joint_flux", "path": "prefill", "shape": "flux", "batch": 4, "q_seq": 4608, "kv_seq": 4608,
         "causal": False},
        # a batch of prompts padded to the longest, odd length, the tokenizer's int64 mask
        {"name": "padded_batch", "path": "padded", "shape": "qwen3_0p6b", "batch": 8, "seq": 1111, "causal": True,
         "len_seed": 5, "mask": "int64"},
        # sliding-window layers on a long prompt, odd length
        {"name": "window_prompt", "path": "window", "shape": "qwen3_8b", "batch": 2, "seq": 5003, "window": 1024},
        # the char-level training run of the examples, and a training step's attention at the 0.6B shape
        {"name": "train_char", "path": "train", "shape": "char", "batch": 64, "seq": 256, "causal": True},
        {"name": "train_qwen3_0p6b", "path": "train", "shape": "qwen3_0p6b", "batch": 8, "seq": 2048, "causal": True},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# A drawn case stays below these (flops, bytes), which no listed path exceeds by its largest case.
_CAPS = {"token": (0, 0.5e9), "step": (0, 1.0e9), "decode": (0, 4.5e9), "append": (0, 1.5e9), "prefill": (1.6e12, 2.0e9),
         "padded": (0.5e12, 1.0e9), "window": (0.4e12, 1.0e9), "train": (0.8e12, 1.0e9)}


def draw(rng: random.Random) -> dict:
    while True:
        c = _draw(rng)
        w, cap = work(c), _CAPS[c["path"]]
        if (cap[0] == 0 or w["flops"] <= cap[0]) and w["bytes"] <= cap[1]:
            return c


def _draw(rng: random.Random) -> dict:
    path = rng.choice(["token", "step", "decode", "append", "prefill", "prefill", "padded", "window", "train", "train"])
    shape = rng.choice(list(SHAPES))
    c = {"path": path, "shape": shape}
    if path in ("token", "step"):
        c["batch"] = _log_int(rng, 1, 16)
        c["len"] = _log_int(rng, 1, 16000)
        c["cap"] = (c["len"] + 512) // 512 * 512
        if path == "token":
            c["ragged"] = rng.random() < 0.5
    elif path == "decode":
        c["batch"] = _log_int(rng, 1, 96)
        c["max_len"] = _log_int(rng, 64, 32768)
        c["min_len"] = max(1, c["max_len"] // rng.choice([1, 2, 8, 64]))
        c["len_seed"] = rng.randrange(1 << 20)
    elif path == "append":
        c["batch"] = _log_int(rng, 1, 16)
        c["seq"] = _log_int(rng, 8, 16384)
        c["cap"] = c["seq"] + rng.choice([0, 1, 512])
        c["rotary"] = "pairs" if shape == "flux" else "half"
    elif path == "prefill":
        c["batch"] = _log_int(rng, 1, 32)
        c["causal"] = rng.random() < 0.6
        c["kv_seq"] = _log_int(rng, 16, 12000)
        # a causal prompt has one length; without a mask the queries may be fewer or more than the keys
        c["q_seq"] = c["kv_seq"] if (c["causal"] or rng.random() < 0.5) else _log_int(rng, 16, 8000)
    elif path == "padded":
        c["batch"] = _log_int(rng, 2, 32)
        c["seq"] = _log_int(rng, 24, 4096)
        c["causal"] = rng.random() < 0.6
        c["len_seed"] = rng.randrange(1 << 20)
        c["mask"] = rng.choice(["int64", "bool", "float32"])
    elif path == "window":
        c["batch"] = _log_int(rng, 1, 8)
        c["seq"] = _log_int(rng, 200, 12000)
        c["window"] = _log_int(rng, 32, 4096)
    else:
        c["batch"] = _log_int(rng, 1, 64)
        c["seq"] = _log_int(rng, 48, 8192)
        c["causal"] = rng.random() < 0.8
    return c


def _lengths(case) -> list:
    """The sequences' own lengths of a decode or padded case (the case alone decides them)."""
    r = random.Random(case["len_seed"])
    if case["path"] == "decode":
        return [r.randint(case["min_len"], case["max_len"]) for _ in range(case["batch"])]
    top = case["seq"]
    return [top] + [r.randint(max(1, top // 4), top) for _ in range(case["batch"] - 1)]  # padded to the longest


def _step_lengths(case) -> list:
    """Keys each sequence of a token case holds once the new one is appended."""
    n, b = case["len"], case["batch"]
    return [max(1, n - (i * n) // (2 * b)) for i in range(b)] if case["ragged"] else [n] * b


# ------------------------------------------------------------------------------------------- inputs
def _randn(gen, *shape, norm=False):
    t = torch.randn(shape, generator=gen, device="cuda", dtype=torch.bfloat16)
    if norm:  # QK-norm models hand over vectors of unit root mean square
        t = (t.float() / torch.sqrt(t.float().pow(2).mean(-1, keepdim=True) + 1e-6)).bfloat16()
    return t


def _rotary(max_pos, d):
    inv = 1.0 / (1.0e6 ** (torch.arange(0, d, 2, device="cuda", dtype=torch.float32) / d))
    ang = torch.arange(max_pos, device="cuda", dtype=torch.float32)[:, None] * inv[None]
    return ang.cos().contiguous(), ang.sin().contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    hq, hkv, d, norm = SHAPES[case["shape"]]
    path, b = case["path"], case["batch"]
    s = {"case": case}
    if path == "token":
        lens = _step_lengths(case)
        s["lens"] = lens
        s["x"] = [_randn(gen, b, 1, h, d) for h in (hq, hkv, hkv)]
        s["cache"] = [_randn(gen, b, hkv, case["cap"], d, norm=norm), _randn(gen, b, hkv, case["cap"], d)]
        s["q"] = torch.empty(b, hq, 1, d, device="cuda", dtype=torch.bfloat16)
        s["w"] = [1.0 + 0.1 * torch.randn(d, generator=gen, device="cuda") if norm else None for _ in range(2)]
        s["rot"] = _rotary(case["cap"], d)
        # sequences of one length: the host knows it; of several lengths: they live on the device
        s["pos"] = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda") if case["ragged"] else None
        s["kv_lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda") if case["ragged"] else None
    elif path == "step":
        s["q"] = _randn(gen, b, hq, 1, d, norm=norm)
        s["cache"] = [_randn(gen, b, hkv, case["cap"], d, norm=norm), _randn(gen, b, hkv, case["cap"], d)]
    elif path == "decode":
        lens = _lengths(case)
        s["q"] = _randn(gen, b, hq, d)
        s["plan"] = nn.DecodePlan([_randn(gen, hkv, n, d) for n in lens], [_randn(gen, hkv, n, d) for n in lens], hq)
    elif path == "append":
        seq, cap = case["seq"], case["cap"]
        s["x"] = [_randn(gen, b, seq, h, d) for h in (hq, hkv, hkv)]
        s["out"] = [torch.zeros(b, hq, seq, d, device="cuda", dtype=torch.bfloat16)] + [
            torch.zeros(b, hkv, cap, d, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        s["w"] = [1.0 + 0.1 * torch.randn(d, generator=gen, device="cuda") if norm else None for _ in range(2)]
        cos, sin = _rotary(cap, d)
        if case["rotary"] == "pairs":
            s["rot"] = {"pe": torch.stack([cos, -sin, sin, cos], -1).view(1, cap, d // 2, 2, 2).contiguous()}
        else:
            s["rot"] = {"cos": cos, "sin": sin}
    else:
        sq = case["q_seq"] if path == "prefill" else case["seq"]
        skv = case["kv_seq"] if path == "prefill" else case["seq"]
        s["q"] = _randn(gen, b, hq, sq, d, norm=norm)
        s["k"] = _randn(gen, b, hkv, skv, d, norm=norm)
        s["v"] = _randn(gen, b, hkv, skv, d)
        if path == "padded":
            lens = torch.tensor(_lengths(case), device="cuda")
            m = torch.arange(skv, device="cuda")[None] < lens[:, None]
            s["mask"] = m.to(getattr(torch, case["mask"]))
        if path == "train":
            s["d_o"] = _randn(gen, b, hq, sq, d)
    return s


# --------------------------------------------------------------------------------------------- a pass
def run(s):
    c = s["case"]
    path = c["path"]
    hq, hkv, d, _ = SHAPES[c["shape"]]
    if path == "token":
        (xq, xk, xv), (kc, vc), (wq, wk), (cos, sin) = s["x"], s["cache"], s["w"], s["rot"]
        at = {"positions": s["pos"]} if c["ragged"] else {"position0": c["len"] - 1}
        nn.qkPrologue(xk, kc, wk, cos, sin, **at)
        nn.qkPrologue(xv, vc, **at)
        nn.qkPrologue(xq, s["q"], wq, cos, sin, out_at_row0=True, **at)
        o, lse = nn.flashDecodeDense(s["q"], kc, vc, kv_lens=s["kv_lens"], kv_len=c["len"])
        return {"o": o, "lse": lse, "k_cache": kc, "v_cache": vc}
    if path == "step":
        kc, vc = s["cache"]
        n = c["len"]
        return nn.scaledDotProductAttentionGQAQKV(s["q"], kc[:, :, :n], vc[:, :, :n], 0.0, False, True)
    if path == "decode":
        o, lse = nn.flashDecode(s["q"], s["plan"])
        return {"o": o, "lse": lse}
    if path == "append":
        (xq, xk, xv), (oq, kc, vc), (wq, wk) = s["x"], s["out"], s["w"]
        nn.qkPrologue(xq, oq, wq, **s["rot"])
        nn.qkPrologue(xk, kc, wk, **s["rot"])
        nn.qkPrologue(xv, vc)
        return {"q": oq, "k_cache": kc, "v_cache": vc}
    q, k, v = s["q"], s["k"], s["v"]
    if path == "prefill":
        if c["q_seq"] != c["kv_seq"]:
            return nn.scaledDotProductAttentionGQAQKV(q, k, v, 0.0, c["causal"], True)
        if hq == hkv:
            return nn.scaled_dot_product_attention(q, k, v, 0.0, c["causal"])
        return nn.scaledDotProductAttentionGQA(q, k, v, 0.0, c["causal"], True)
    if path == "padded":
        return nn.scaledDotProductAttentionGQAMask(q, k, v, s["mask"], 0.0, c["causal"], True)
    if path == "window":
        return nn.scaledDotProductAttentionGQAWindow(q, k, v, 0.0, True, True, c["window"])
    o, lse = nn.attentionFwd(q, k, v, is_causal=c["causal"])
    d_q, d_k, d_v = nn.attentionBwd(q, k, v, o, lse, s["d_o"], is_causal=c["causal"])
    return {"o": o, "lse": lse, "d_q": d_q, "d_k": d_k, "d_v": d_v}


# ------------------------------------------------------------------------------------ what it comes to
def _pairs(case) -> int:
    """(query row, key) pairs one query head of the whole batch needs, the masks taken exactly."""
    path, b = case["path"], case["batch"]
    if path == "prefill":
        sq, skv = case["q_seq"], case["kv_seq"]
        return b * (sq * (sq + 1) // 2 if case["causal"] else sq * skv)
    s = case["seq"]
    if path == "window":
        w = min(case["window"], s)
        return b * (w * (w + 1) // 2 + (s - w) * w)
    if path == "padded":  # padding rows are computed too: the call returns them
        return sum(n * (n + 1) // 2 + (s - n) * n if case["causal"] else s * n for n in _lengths(case))
    return b * (s * (s + 1) // 2 if case["causal"] else s * s)


def work(case):
    hq, hkv, d, norm = SHAPES[case["shape"]]
    path, b = case["path"], case["batch"]
    row = 2 * d  # bytes of one bf16 row
    if path in ("token", "step", "decode"):
        keys = sum(_lengths(case)) if path == "decode" else (
            sum(_step_lengths(case)) if path == "token" else b * case["len"])
        kv = 2 * keys * hkv * row
        qo = 2 * b * hq * row + (0 if path == "step" else 4 * b * hq)
        new = 2 * b * (hq + 2 * hkv) * row if path == "token" else 0
        return {"bytes": kv + qo + new, "flops": 4 * keys * hq * d}
    if path == "append":
        tok = b * case["seq"]
        tab = case["seq"] * d * (8 if case["rotary"] == "pairs" else 4)
        return {"bytes": 2 * tok * (hq + 2 * hkv) * row + tab, "flops": 10 * tok * (hq + hkv) * d}
    sq = case["q_seq"] if path == "prefill" else case["seq"]
    skv = case["kv_seq"] if path == "prefill" else case["seq"]
    q, kv = b * hq * sq * row, b * hkv * skv * row
    flops = 4 * d * hq * _pairs(case)
    if path == "train":  # forward: Q, K, V in, O and row statistics out; backward: those and dO in, the gradients out
        stat = 4 * b * hq * sq
        return {"bytes": 2 * q + 2 * kv + stat + (3 * q + 2 * kv + stat) + (q + 2 * kv), "flops": flops * 7 // 2}
    mask = b * skv * {"int64": 8, "bool": 1, "float32": 4}[case["mask"]] if path == "padded" else 0
    return {"bytes": 2 * q + 2 * kv + mask, "flops": flops}


# Relative errors against the same formula in float64 over the ranges of `draw`: bf16 P, dS and outputs give
# 2.1e-3 to 2.9e-3 for O and the gradients, the one rounding of the prologue 1.7e-3; about four times that.
_TOL = {"append": 7.0e-3}


def tolerance(case):
    return {"rel": _TOL.get(case["path"], 1.0e-2)}
