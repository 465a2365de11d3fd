"""The attention calls whose speed matters, as data: what a program that serves or trains with this
package has it compute, through the package's public entry points.

Most cases go through the front door, ``torch.compile(fn, backend=loopfuse_backend)``, with the
attention written the way a model writes it; the serving cases that have no graph form (a prefill
chunk that continues a cached sequence, a decode step that first appends to the paged cache) call
``loopfuse_b200.functional`` directly.

``kind`` of a case:
  causal         softmax(causal(q k^T / sqrt(D))) v; grouped heads when Hq > Hkv
  softcap        the same with the scores through cap * tanh(s / cap) first
  window         softcap scores, and only the last ``window`` keys of each row are visible
  chunk          rows [offset, offset + Sq) of a sequence against all its keys so far
  decode         one new row per sequence against a dense cache
  paged_decode   one new row per sequence against a paged cache (whole pages)
  paged_step     append one token to a paged cache, then attend to all of it
  paged_prefill  causal prefill whose keys are read through a block table of one-token pages
  biased         query bias, scaled scores plus a full score bias, causal, output bias

All tensors are bfloat16, the package's one data type, with N(0, 1) values (projections of
normalised activations).
"""
from __future__ import annotations

import math

import torch

from loopfuse_b200 import functional as F
from loopfuse_b200 import loopfuse_backend
from loopfuse_b200 import spec as S

DTYPE = torch.bfloat16
MAX_FLOPS = 560e9      # of a drawn case: the largest listed prefill
MAX_BYTES = 2.2e9      # of a drawn case: the largest listed decode


def listed() -> list[dict]:
    return [
        # A small model or a unit of a test suite: four heads, one short sequence pair. The time is
        # the latency of one call.
        dict(name="causal_tiny", kind="causal", B=2, Hq=4, Hkv=4, S=512, D=64),
        # A batch of prompts of no round length with grouped heads, small head dim.
        dict(name="causal_ragged", kind="causal", B=4, Hq=8, Hkv=4, S=593, D=64),
        # One long prompt, grouped heads: the largest prefill.
        dict(name="causal_long_gqa", kind="causal", B=1, Hq=32, Hkv=8, S=8192, D=128),
        # The headline configuration: batch prefill with logit softcap.
        dict(name="causal_softcap", kind="softcap", B=8, Hq=32, Hkv=32, S=2048, D=128, cap=50.0),
        # The local-attention layers of softcap models: sliding window, grouped heads.
        dict(name="window_gqa_softcap", kind="window", B=8, Hq=32, Hkv=8, S=2048, D=128, cap=50.0,
             window=256),
        # Chunked prefill: the next, ragged chunk of a sequence that already has keys in its cache.
        dict(name="chunk_gqa", kind="chunk", B=1, Hq=32, Hkv=8, Sq=777, offset=3319, D=128,
             cap=0.0),
        # Decode of a full batch, no head grouping: the largest cache read.
        dict(name="decode", kind="decode", B=64, Hq=32, Hkv=32, S=2048, D=128, cap=0.0),
        # Interactive decode: one sequence with a long, odd-sized cache, grouped heads, softcap.
        dict(name="decode_single", kind="decode", B=1, Hq=32, Hkv=8, S=8190, D=128, cap=50.0),
        # Decode of a full batch from a paged cache with grouped heads.
        dict(name="paged_decode_gqa", kind="paged_decode", B=64, Hq=32, Hkv=8, S=2048, D=128,
             page=16),
        # One step of a serving loop at moderate load: append to the cache, then attend.
        dict(name="paged_step", kind="paged_step", B=16, Hq=32, Hkv=8, S=1001, D=128, page=16),
        # Prefill over keys that live in a cache of one-token pages.
        dict(name="paged_prefill", kind="paged_prefill", B=4, Hq=8, Hkv=4, S=1024, D=64),
        # Attention with additive biases (relative positions as a full score matrix).
        dict(name="biased", kind="biased", B=4, Hq=8, Hkv=8, S=1024, D=64),
    ]


KINDS = ["causal", "softcap", "window", "chunk", "decode", "paged_decode", "paged_step",
         "paged_prefill", "biased"]


def draw(rng) -> dict:
    def log_int(lo: int, hi: int) -> int:
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(KINDS)
    D = rng.choice((64, 128))
    Hkv = rng.choice((1, 2, 4, 8, 16, 32))
    group = rng.choice([g for g in (1, 2, 4, 8) if Hkv * g <= 64])
    c = dict(kind=kind, B=0, Hq=Hkv * group, Hkv=Hkv)
    if kind in ("causal", "softcap", "window", "paged_prefill"):
        c.update(B=log_int(1, 8), S=log_int(64, 8192), D=D)
        if kind == "paged_prefill":
            c["S"] = log_int(64, 4096)
        if kind in ("softcap", "window"):
            c["cap"] = rng.choice((20.0, 30.0, 50.0))
        if kind == "window":
            c["window"] = log_int(64, 1024)
    elif kind == "biased":
        c.update(B=log_int(1, 8), S=8 * log_int(8, 256), D=D)
        c["Hkv"] = c["Hq"]
    elif kind == "chunk":
        c.update(B=log_int(1, 4), Sq=log_int(16, 2048), offset=log_int(64, 8192), D=D,
                 cap=rng.choice((0.0, 0.0, 50.0)))
    else:
        c.update(B=log_int(1, 64), S=log_int(64, 16384), D=D)
        if kind == "decode":
            c["cap"] = rng.choice((0.0, 0.0, 50.0))
        else:
            c["page"] = rng.choice((1, 16, 32, 64))
            if kind == "paged_decode":  # the graph form reads whole pages
                c["S"] = -(-c["S"] // c["page"]) * c["page"]
    while work(c)["flops"] > MAX_FLOPS or work(c)["bytes"] > MAX_BYTES:
        if c["B"] > 1:
            c["B"] -= 1
        elif kind == "chunk":
            c["offset"] //= 2
        else:
            c["S"] = c["S"] // 2 // 64 * 64
    return c


# -- the attention functions, as a model writes them ----------------------------------------------
def _repeat(k, v, n: int):
    return k.repeat_interleave(n, dim=1), v.repeat_interleave(n, dim=1)


def _causal(q, k, v):
    s = q @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
    return torch.softmax(torch.ops.loopfuse.causal_mask(s), dim=-1) @ v


def _causal_gqa(q, k, v):
    k, v = _repeat(k, v, q.shape[1] // k.shape[1])
    s = q @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
    return torch.softmax(torch.ops.loopfuse.causal_mask(s), dim=-1) @ v


def _softcap(cap: float, window: int, grouped: bool):
    def attention(q, k, v):
        if grouped:
            k, v = _repeat(k, v, q.shape[1] // k.shape[1])
        s = q @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
        s = torch.tanh(s / cap) * cap
        if window:
            s = torch.ops.loopfuse.sliding_mask(s, window)
        return torch.softmax(torch.ops.loopfuse.causal_mask(s), dim=-1) @ v
    return attention


def _decode(cap: float, grouped: bool):
    def attention(q, k, v):
        if grouped:
            k, v = _repeat(k, v, q.shape[1] // k.shape[1])
        s = q @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
        if cap:
            s = torch.tanh(s / cap) * cap
        return torch.softmax(s, dim=-1) @ v
    return attention


def _paged_decode(q, k_pool, v_pool, table):   # q: [B, Hkv, group, D]
    b = q.shape[0]
    k = torch.ops.loopfuse.paged_load(k_pool, table)
    v = torch.ops.loopfuse.paged_load(v_pool, table)
    k = k.reshape(b, -1, k.shape[-2], k.shape[-1]).transpose(1, 2)
    v = v.reshape(b, -1, v.shape[-2], v.shape[-1]).transpose(1, 2)
    return torch.softmax(q @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5), dim=-1) @ v


def _paged_prefill(grouped: bool):
    def attention(q, k_pool, table, v):
        k = torch.ops.loopfuse.paged_load(k_pool, table).transpose(1, 2)
        if grouped:
            k, v = _repeat(k, v, q.shape[1] // k.shape[1])
        s = q @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
        return torch.softmax(torch.ops.loopfuse.causal_mask(s), dim=-1) @ v
    return attention


def _biased(q, k, v, q_bias, score_bias, out_bias):
    s = (q + q_bias) @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
    s = s * 3.5 + score_bias
    return torch.softmax(torch.ops.loopfuse.causal_mask(s), dim=-1) @ v + out_bias


def _function(case: dict):
    kind, grouped = case["kind"], case["Hq"] != case["Hkv"]
    if kind == "causal":
        return _causal_gqa if grouped else _causal
    if kind in ("softcap", "window"):
        return _softcap(case["cap"], case.get("window", 0), grouped)
    if kind == "decode":
        return _decode(case["cap"], grouped)
    if kind == "paged_decode":
        return _paged_decode
    if kind == "paged_prefill":
        return _paged_prefill(grouped)
    return _biased


_compiled: dict = {}


def _compile(case: dict):
    """One compiled function per case. A program compiles its model's attention once; another case
    is another program, so it starts from a clean compiler."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _compiled:
        torch._dynamo.reset()
        _compiled.clear()
        _compiled[key] = torch.compile(_function(case), backend=loopfuse_backend, dynamic=True)
    return _compiled[key]


# -- inputs, one pass, its work, its tolerance ----------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=DTYPE)

    kind, B, Hq, Hkv, D = (case[n] for n in ("kind", "B", "Hq", "Hkv", "D"))
    st: dict = {"kind": kind}

    def paged_cache(tokens: int, page: int):
        blocks = -(-tokens // page)
        table = torch.randperm(B * blocks, generator=g, device="cuda").view(B, blocks).int()
        return (B * blocks, page, Hkv, D), table

    if kind == "chunk":
        Skv = case["offset"] + case["Sq"]
        mods = ()
        if case["cap"]:
            mods = (S.ScoreMod(S.MOD_DIV, case["cap"]), S.ScoreMod(S.MOD_TANH),
                    S.ScoreMod(S.MOD_MUL, case["cap"]))
        st["args"] = (normal(B, Hq, case["Sq"], D), normal(B, Hkv, Skv, D), normal(B, Hkv, Skv, D))
        st["options"] = dict(scale=D ** -0.5, mods=mods, mask_kind=S.MASK_CAUSAL,
                             causal_offset=case["offset"])
        return st
    if kind == "paged_step":
        shape, table = paged_cache(case["S"], case["page"])
        st.update(q=normal(B, Hkv, Hq // Hkv, D), k_new=normal(B, Hkv, 1, D),
                  v_new=normal(B, Hkv, 1, D), k_pool=normal(*shape), v_pool=normal(*shape),
                  table=table, last=case["S"] - 1, scale=D ** -0.5,
                  workspace=F.DecodeWorkspace())
        return st
    st["fn"] = _compile(case)
    if kind == "decode":
        st["args"] = (normal(B, Hq, 1, D), normal(B, Hkv, case["S"], D),
                      normal(B, Hkv, case["S"], D))
    elif kind == "paged_decode":
        shape, table = paged_cache(case["S"], case["page"])
        st["args"] = (normal(B, Hkv, Hq // Hkv, D), normal(*shape), normal(*shape), table)
    elif kind == "paged_prefill":
        shape, table = paged_cache(case["S"], 1)
        st["args"] = (normal(B, Hq, case["S"], D), normal(*shape).squeeze(1), table,
                      normal(B, Hkv, case["S"], D))
    else:
        n = case["S"]
        st["args"] = (normal(B, Hq, n, D), normal(B, Hkv, n, D), normal(B, Hkv, n, D))
        if kind == "biased":
            st["args"] += (normal(B, Hq, n, D), normal(B, Hq, n, n), normal(B, Hq, n, D))
    return st


def run(state: dict):
    if state["kind"] == "chunk":
        return F.prefill_attention(*state["args"], **state["options"])
    if state["kind"] == "paged_step":
        F.kv_append(state["k_new"], state["v_new"], state["k_pool"], state["v_pool"],
                    state["table"], start_pos=state["last"])
        out = F.paged_decode_attention(state["q"], state["k_pool"], state["v_pool"],
                                       state["table"], seq_len=state["last"] + 1,
                                       scale=state["scale"], workspace=state["workspace"])
        return {"out": out, "k_pool": state["k_pool"], "v_pool": state["v_pool"]}
    return state["fn"](*state["args"])


def work(case: dict) -> dict:
    """Each input read once, each output written once; four operations per visible (row, key)
    pair and column."""
    kind, B, Hq, Hkv, D = (case[n] for n in ("kind", "B", "Hq", "Hkv", "D"))
    if kind in ("decode", "paged_decode", "paged_step"):
        n = case["S"]
        values = 2 * B * Hq * D + 2 * B * Hkv * n * D
        if kind == "paged_step":
            values += 2 * B * Hkv * D       # the new rows are read too; their pages are in n
        tables = 0 if kind == "decode" else 4 * B * -(-n // case["page"])
        return {"bytes": 2 * values + tables, "flops": 4 * B * Hq * n * D}
    if kind == "chunk":
        rows, first = case["Sq"], case["offset"] + 1
        keys = case["offset"] + rows
    else:
        rows, first, keys = case["S"], 1, case["S"]
    window = case.get("window", 0)
    last = first + rows - 1                  # row r sees first + r keys, at most `window`
    if not window or window >= last:
        pairs = rows * (first + last) // 2
    elif window <= first:
        pairs = rows * window
    else:
        pairs = (window - first) * (first + window - 1) // 2 + (last - window + 1) * window
    values = 2 * B * Hq * rows * D + 2 * B * Hkv * keys * D
    extra = 0
    if kind == "biased":
        values += 2 * B * Hq * rows * D + B * Hq * pairs      # the bias of visible pairs
    elif kind == "paged_prefill":
        extra = 4 * B * keys
    return {"bytes": 2 * values + extra, "flops": 4 * B * Hq * pairs * D}


def tolerance(case: dict) -> dict:
    """Probabilities and outputs are bfloat16 (8 bits): each rounds by up to 2^-9 of its value, and
    another correct implementation rounds them against another reference."""
    return {"rel": 1e-2}
