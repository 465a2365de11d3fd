"""The prefill kernels deal query tiles out in several forms, by their number and length: pairs of tiles per
CTA, one tile split over the two slots of a CTA (running-max kernel, no more tiles than SMs), or two CTAs
per SM. Every kind of call on the two-CTA side of the rules, at the edges of tiles, against another form of
the same call and against fp32."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from loopfuse_b200 import functional as F, spec as S

pytestmark = pytest.mark.gpu
# Two bf16 results of the same row differ by the rounding of P (2^-9 of each weight, in numerator and
# sum) and of the result (2^-9 of it): 3 * 2^-9 of max |v| < 5.5 at the very most, 2^-8 of the norm.
MAX_ABS = 3 * 2.0 ** -9 * 5.5
REL = 2.0 ** -8


def _close(out, want):
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    d = (out.float() - want.float()).nan_to_num()
    assert d.abs().max().item() <= MAX_ABS
    assert (d.norm() / want.float().nan_to_num().norm()).item() <= REL


def _by_heads(fn, q, *per_head, chunk):
    """fn on `chunk` query heads at a time (and whatever else is cut by head with them)."""
    parts = []
    for h in range(0, q.shape[1], chunk):
        group = q.shape[1] // per_head[0].shape[1]
        cut = [t if t is None else t[:, h // group:(h + chunk) // group] if t.shape[1] != q.shape[1]
               else t[:, h:h + chunk] for t in per_head]
        parts.append(fn(q[:, h:h + chunk], *cut))
    return torch.cat(parts, dim=1)


def _fp32(q, k, v, mask, off, window=0, scale=None, bias=None):
    k, v = (t.float().repeat_interleave(q.shape[1] // k.shape[1], dim=1) for t in (k, v))
    s = q.float() @ k.transpose(-2, -1) * (scale or q.shape[-1] ** -0.5)
    if bias is not None:
        s = s + bias.float()
    i = torch.arange(q.shape[2], device="cuda")[:, None] + off
    j = torch.arange(k.shape[2], device="cuda")[None]
    if mask != S.MASK_NONE:
        s = s.masked_fill(j > i, float("-inf"))
    if mask == S.MASK_CAUSAL_WINDOW:
        s = s.masked_fill(j <= i - window, float("-inf"))
    return torch.softmax(s, dim=-1) @ v


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,mask,off,window", [
    (2, 152, 38, 1, 1, S.MASK_CAUSAL, 0, 0),          # one tile per head, one row
    (3, 104, 52, 128, 65, S.MASK_NONE, 0, 0),
    (5, 60, 20, 129, 129, S.MASK_CAUSAL, 0, 0),       # a last tile of one row
    (3, 52, 13, 300, 1100, S.MASK_CAUSAL, 800, 0),    # three tiles a head, a chunk
    (1, 304, 38, 100, 2100, S.MASK_CAUSAL, 2000, 0),  # one tile a head, long rows
    (3, 52, 26, 257, 200, S.MASK_CAUSAL, -60, 0),     # rows without a key
    (2, 76, 19, 250, 250, S.MASK_CAUSAL_WINDOW, 0, 70),
    (2, 40, 10, 520, 520, S.MASK_CAUSAL, 0, 0),
])
def test_two_ctas_per_sm(B, Hq, Hkv, Sq, Skv, mask, off, window, D):
    torch.manual_seed(1)
    # Heads inside the rows, and K and V in one tensor: strides of a packed projection.
    q = torch.randn(B, Sq, Hq, D, device="cuda").bfloat16().transpose(1, 2)
    kv = torch.randn(B, Skv, 2 * Hkv, D, device="cuda").bfloat16().transpose(1, 2)
    k, v = kv[:, :Hkv], kv[:, Hkv:]
    st = F.new_status("cuda")
    kw = dict(scale=D ** -0.5, mask_kind=mask, window=window, causal_offset=off)
    assert F.prefill_form(q, k, v, **kw) == "narrow"
    call = lambda q, k, v: F.prefill_attention(q, k, v, status=st, **kw)
    out = call(q, k, v)
    F.check_status(st)
    _close(out, _fp32(q, k, v, mask, off, window))
    _close(out, _by_heads(call, q, k, v, chunk=Hq // Hkv))
    assert torch.equal(out.nan_to_num(), call(q, k, v).nan_to_num())


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,D", [
    (1, 80, 10, 520, 520, 128), (1, 64, 8, 700, 1400, 128), (1, 80, 10, 520, 520, 64), (1, 136, 34, 300, 620, 64)])
def test_pairs_and_two_ctas_per_sm_give_the_same_bits(B, Hq, Hkv, Sq, Skv, D):
    """Half of the heads run as pairs, all of them as two CTAs per SM: the same steps for every tile."""
    torch.manual_seed(5)
    q = torch.randn(B, Hq, Sq, D, device="cuda").bfloat16()
    k, v = (torch.randn(B, Hkv, Skv, D, device="cuda").bfloat16() for _ in range(2))
    kw = dict(scale=D ** -0.5, mask_kind=S.MASK_CAUSAL, causal_offset=Skv - Sq)
    assert F.prefill_form(q, k, v, **kw) == "narrow"
    out = F.prefill_attention(q, k, v, **kw)
    for i in range(2):
        half = (q[:, i * Hq // 2:(i + 1) * Hq // 2], *(t[:, i * Hkv // 2:(i + 1) * Hkv // 2] for t in (k, v)))
        assert F.prefill_form(*half, **kw) == "pairs"
        assert torch.equal(out[:, i * Hq // 2:(i + 1) * Hq // 2], F.prefill_attention(*half, **kw))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Sq,Skv,pad,form", [
    (3, 52, 200, 200, 0, "narrow"), (2, 40, 513, 260, 8, "narrow"), (2, 150, 40, 72, 0, "narrow"),
    (1, 320, 60, 1000, 8, "split"),  # split tiles, more of them than SMs
])
def test_two_ctas_per_sm_with_biases(B, H, Sq, Skv, pad, form, D):
    torch.manual_seed(2)
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    q, k, v, qb, ob = mk(B, H, Sq, D), mk(B, H, Skv, D), mk(B, H, Skv, D), mk(B, H, Sq, D), mk(B, H, Sq, D)
    bias = mk(B, H, Sq, (Skv + 7) // 8 * 8 + pad)[..., :Skv]
    off = Skv - Sq if form == "split" else 0
    kw = dict(scale=D ** -0.5, mods=[S.ScoreMod(S.MOD_MUL, 2.0)], mask_kind=S.MASK_CAUSAL, causal_offset=off)
    assert F.prefill_form(q, k, v, score_bias=bias, **kw) == form
    call = lambda q, k, v, bias, qb, ob: F.prefill_attention(q, k, v, score_bias=bias, q_bias=qb, out_bias=ob, **kw)
    out = call(q, k, v, bias, qb, ob)
    few = _by_heads(call, q, k, v, bias, qb, ob, chunk=2)
    _close(out.float() - ob.float(), few.float() - ob.float())
    # (the sum with the output bias is rounded once more: half a bf16 step of it)
    want = _fp32(q + qb, k, v, S.MASK_CAUSAL, off, scale=2 * D ** -0.5, bias=bias)
    assert ((out.float() - (want + ob.float())).abs() <= MAX_ABS + (want + ob.float()).abs() / 256).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("P,heads_first", [(1, False), (16, False), (16, True)])
@pytest.mark.parametrize("which,Sq,Skv", [("k", 330, 330), ("v", 330, 330), ("kv", 380, 700)])
def test_two_ctas_per_sm_paged(which, Sq, Skv, P, heads_first, D):
    """Row gathers (more than one window of eight tiles among them), and pools whose rows the producer warp
    copies itself, which has the two-CTA form at D = 64 only."""
    torch.manual_seed(3)
    B, Hkv, G = 4, 8, 4
    blocks = -(-Skv // P)
    shape = (B * blocks + 2, Hkv, P, D) if heads_first else (B * blocks + 2, P, Hkv, D)
    table = torch.randperm(B * blocks + 2, device="cuda")[:B * blocks].view(B, blocks).int()
    q = torch.randn(B, Hkv * G, Sq, D, device="cuda").bfloat16()
    given, dense, kw = [], [], dict(scale=D ** -0.5, mask_kind=S.MASK_CAUSAL, causal_offset=Skv - Sq, seq_len=Skv)
    for n in "kv":
        if n in which:
            pool = torch.randn(*shape, device="cuda").bfloat16()
            pool = pool.transpose(1, 2) if heads_first else pool
            given.append(pool)
            dense.append(pool[table.long()].reshape(B, blocks * P, Hkv, D)[:, :Skv].transpose(1, 2))
            kw[n + "_block_table"] = table
        else:
            given.append(torch.randn(B, Hkv, Skv, D, device="cuda").bfloat16())
            dense.append(given[-1])
    assert F.prefill_form(q, *given, **kw) == ("pairs" if heads_first and D == 128 else "narrow")
    st = F.new_status("cuda")
    out = F.prefill_attention(q, *given, status=st, **kw)
    F.check_status(st)
    _close(out, _fp32(q, *dense, S.MASK_CAUSAL, Skv - Sq))


FIRST_IN_CAPTURE = """
import torch
from loopfuse_b200 import functional as F, spec as S
cap = [S.ScoreMod(S.MOD_DIV, 50.0), S.ScoreMod(S.MOD_TANH), S.ScoreMod(S.MOD_MUL, 50.0)]
mk = lambda h, n: [torch.randn(1, h, n, 128, device="cuda").bfloat16() for _ in range(3)]
bias = lambda h, n: dict(score_bias=torch.randn(1, h, n, n, device="cuda").bfloat16())
for mods, with_bias, first, second in (([], False, (8, 512), (128, 512)), ([], True, (8, 512), (128, 512)),
                                       (cap, False, (40, 2048), (8, 512))):
    calls = []
    for h, n in (first, second):
        kw = dict(scale=128 ** -0.5, mask_kind=S.MASK_CAUSAL, mods=mods, **(bias(h, n) if with_bias else {}))
        calls.append((mk(h, n), kw))
    (a, kwa), (b, kwb) = calls
    assert F.prefill_form(*a, **kwa) != "narrow" and F.prefill_form(*b, **kwb) == "narrow"
    F.prefill_attention(*a, **kwa)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = F.prefill_attention(*b, **kwb)
    g.replay()
    assert torch.equal(out, F.prefill_attention(*b, **kwb))
"""


def test_a_form_can_be_first_used_inside_a_capture():
    """A program that has called a kernel once, and then captures a call of another size."""
    root = str(Path(__file__).resolve().parents[1])
    r = subprocess.run([sys.executable, "-c", FIRST_IN_CAPTURE], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


SOFTCAP = [S.ScoreMod(S.MOD_DIV, 30.0), S.ScoreMod(S.MOD_TANH), S.ScoreMod(S.MOD_MUL, 30.0)]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,mask,off,window,gain", [
    (1, 2, 2, 1, 1, S.MASK_CAUSAL, 0, 0, 1.0),
    (2, 3, 1, 129, 129, S.MASK_CAUSAL, 0, 0, 1.0),
    (1, 4, 4, 130, 1000, S.MASK_NONE, 0, 0, 30.0),             # the stronger forms of tanh
    (2, 40, 40, 600, 600, S.MASK_CAUSAL, 0, 0, 1.0),           # more items than CTAs
    (1, 2, 1, 700, 300, S.MASK_CAUSAL, -200, 0, 1.0),          # tiles and rows without a key
    (3, 8, 8, 515, 515, S.MASK_CAUSAL_WINDOW, 0, 100, 1.0),
    (2, 8, 4, 515, 515, S.MASK_CAUSAL_WINDOW, 0, 65, 1.0),     # packed: two heads a tile,
    (1, 16, 4, 515, 515, S.MASK_CAUSAL_WINDOW, 0, 64, 10.0),   # four
    (4, 32, 8, 300, 300, S.MASK_CAUSAL_WINDOW, 0, 1, 1.0),     # one key a row
    (1, 4, 1, 33, 400, S.MASK_CAUSAL_WINDOW, 367, 256, 1.0),
])
def test_softcap_two_ctas_per_sm(B, Hq, Hkv, Sq, Skv, mask, off, window, gain, D):
    """Against the form of one CTA per SM, which a margin of one SM asks for."""
    torch.manual_seed(4)
    q = (torch.randn(B, Sq, Hq, D, device="cuda") * gain).bfloat16().transpose(1, 2)
    k, v = (torch.randn(B, Hkv, Skv, D, device="cuda").bfloat16() for _ in range(2))
    st = F.new_status("cuda")
    kw = dict(scale=D ** -0.5, mods=SOFTCAP, mask_kind=mask, window=window, causal_offset=off)
    lone = D == 128 and Sq == 1  # (one tile a head and an SM for each)
    assert F.prefill_form(q, k, v, **kw) == ("pairs" if lone else "narrow")
    assert F.prefill_form(q, k, v, sm_margin=1, **kw) == "pairs"
    out = F.prefill_attention(q, k, v, status=st, **kw)
    _close(out, F.prefill_attention(q, k, v, sm_margin=1, status=st, **kw))
    F.check_status(st)
    group = Hq // Hkv
    s = q.float() @ k.float().repeat_interleave(group, 1).transpose(-2, -1) * D ** -0.5
    s = torch.tanh(s / 30.0) * 30.0
    i, j = torch.arange(Sq, device="cuda")[:, None] + off, torch.arange(Skv, device="cuda")[None]
    if mask != S.MASK_NONE:
        s = s.masked_fill(j > i, float("-inf"))
    if mask == S.MASK_CAUSAL_WINDOW:
        s = s.masked_fill(j <= i - window, float("-inf"))
    _close(out, torch.softmax(s, -1) @ v.float().repeat_interleave(group, 1))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,mask,window", [
    (2, 38, 38, 1100, S.MASK_CAUSAL, 0),               # nine tiles a head: the last one without a partner
    (3, 32, 16, 700, S.MASK_CAUSAL_WINDOW, 200),       # packed: two heads a tile, an odd number of chunks
    (3, 32, 16, 705, S.MASK_CAUSAL_WINDOW, 200),       # ... an even one
    (3, 40, 10, 1000, S.MASK_CAUSAL_WINDOW, 257),      # four heads a tile, even
    (3, 40, 10, 990, S.MASK_CAUSAL_WINDOW, 700),       # odd
    (3, 40, 10, 950, S.MASK_CAUSAL_WINDOW, 1),
])
def test_softcap_both_forms_with_many_items(B, Hq, Hkv, Sq, mask, window, D):
    """Both forms of the persistent kernel with more items than CTAs and several blocks an item: the hand-over
    between items, tiles without a partner, and the key blocks that each tile visits."""
    torch.manual_seed(6)
    q = (torch.randn(B, Hq, Sq, D, device="cuda") * 2).bfloat16()
    k, v = (torch.randn(B, Hkv, Sq, D, device="cuda").bfloat16() for _ in range(2))
    kw = dict(scale=D ** -0.5, mods=SOFTCAP, mask_kind=mask, window=window)
    rows = F.prefill_q_tile(q, k, v, **kw)
    n = -(-Sq // rows)
    s = q.float() @ k.float().repeat_interleave(Hq // Hkv, 1).transpose(-2, -1) * D ** -0.5
    s = torch.tanh(s / 30.0) * 30.0
    i, j = torch.arange(Sq, device="cuda")[:, None], torch.arange(Sq, device="cuda")[None]
    s = s.masked_fill((j > i) | ((j <= i - window) if window else (j > i)), float("-inf"))
    want = torch.softmax(s, -1) @ v.float().repeat_interleave(Hq // Hkv, 1)
    table = torch.tensor(S.skip_table(mask, window, 0, Sq, Sq, tile_q=rows))
    for margin in (0, 1, 100):
        dbg = torch.full((B * Hq * n * 2,), -1, dtype=torch.int32, device="cuda")
        st = F.new_status("cuda")
        out = F.prefill_attention(q, k, v, sm_margin=margin, dbg_ranges=dbg, status=st, **kw)
        F.check_status(st)
        _close(out, want)
        assert (dbg.view(B * Hq, n, 2).cpu() == table).all()
    assert F.prefill_form(q, k, v, sm_margin=1, **kw) == "pairs"
