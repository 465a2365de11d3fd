"""The prefill kernels deal query tiles out in several forms, by their number and length: pairs of tiles per
CTA, one tile split over the two slots of a CTA (running-max kernel, no more tiles than SMs), or two CTAs
per SM. Every kind of call on the two-CTA side of the rules, at the edges of tiles, against another form of
the same call and against fp32."""
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


def _fp32(q, k, v, mask, off, window=0):
    k, v = (t.float().repeat_interleave(q.shape[1] // k.shape[1], dim=1) for t in (k, v))
    s = q.float() @ k.transpose(-2, -1) * q.shape[-1] ** -0.5
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
    (2, 52, 13, 300, 1100, S.MASK_CAUSAL, 800, 0),    # three tiles a head, a chunk
    (3, 52, 26, 257, 200, S.MASK_CAUSAL, -60, 0),     # rows without a key
    (2, 76, 19, 250, 250, S.MASK_CAUSAL_WINDOW, 0, 70),
    (2, 40, 10, 520, 520, S.MASK_CAUSAL, 0, 0),
])
def test_two_ctas_per_sm(B, Hq, Hkv, Sq, Skv, mask, off, window, D):
    assert -(-Sq // 128) * Hq * B > 2 * torch.cuda.get_device_properties(0).multi_processor_count
    torch.manual_seed(1)
    # Heads inside the rows, and K and V in one tensor: strides of a packed projection.
    q = torch.randn(B, Sq, Hq, D, device="cuda").bfloat16().transpose(1, 2)
    kv = torch.randn(B, Skv, 2 * Hkv, D, device="cuda").bfloat16().transpose(1, 2)
    k, v = kv[:, :Hkv], kv[:, Hkv:]
    st = F.new_status("cuda")
    call = lambda q, k, v: F.prefill_attention(q, k, v, scale=D ** -0.5, mask_kind=mask, window=window,
                                               causal_offset=off, status=st)
    out = call(q, k, v)
    F.check_status(st)
    _close(out, _fp32(q, k, v, mask, off, window))
    _close(out, _by_heads(call, q, k, v, chunk=Hq // Hkv))
    assert torch.equal(out.nan_to_num(), call(q, k, v).nan_to_num())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Sq,Skv,pad", [(3, 52, 200, 200, 0), (2, 40, 513, 260, 8), (2, 150, 40, 72, 0)])
def test_two_ctas_per_sm_with_biases(B, H, Sq, Skv, pad, D):
    torch.manual_seed(2)
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    q, k, v, qb, ob = mk(B, H, Sq, D), mk(B, H, Skv, D), mk(B, H, Skv, D), mk(B, H, Sq, D), mk(B, H, Sq, D)
    bias = mk(B, H, Sq, (Skv + 7) // 8 * 8 + pad)[..., :Skv]
    call = lambda q, k, v, bias, qb, ob: F.prefill_attention(
        q, k, v, scale=D ** -0.5, mods=[S.ScoreMod(S.MOD_MUL, 2.0)], mask_kind=S.MASK_CAUSAL, score_bias=bias,
        q_bias=qb, out_bias=ob)
    out = call(q, k, v, bias, qb, ob)
    few = _by_heads(call, q, k, v, bias, qb, ob, chunk=2)
    _close(out.float() - ob.float(), few.float() - ob.float())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("P,heads_first", [(1, False), (16, False), (16, True)])
def test_two_ctas_per_sm_paged(P, heads_first, D):
    """Row gathers, and pools whose rows the producer warp copies itself."""
    torch.manual_seed(3)
    B, Hkv, G, Sq, Skv = 4, 8, 4, 330, 330
    blocks = -(-Skv // P)
    shape = (B * blocks + 2, Hkv, P, D) if heads_first else (B * blocks + 2, P, Hkv, D)
    pool = torch.randn(*shape, device="cuda").bfloat16()
    pool = pool.transpose(1, 2) if heads_first else pool
    table = torch.randperm(B * blocks + 2, device="cuda")[:B * blocks].view(B, blocks).int()
    q = torch.randn(B, Hkv * G, Sq, D, device="cuda").bfloat16()
    v = torch.randn(B, Hkv, Skv, D, device="cuda").bfloat16()
    st = F.new_status("cuda")
    out = F.prefill_attention(q, pool, v, scale=D ** -0.5, mask_kind=S.MASK_CAUSAL, k_block_table=table,
                              seq_len=Skv, status=st)
    F.check_status(st)
    k = pool[table.long()].reshape(B, blocks * P, Hkv, D)[:, :Skv].transpose(1, 2)
    _close(out, _fp32(q, k, v, S.MASK_CAUSAL, 0))


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
    kw = dict(scale=D ** -0.5, mods=SOFTCAP, mask_kind=mask, window=window, causal_offset=off, status=st)
    out = F.prefill_attention(q, k, v, **kw)
    _close(out, F.prefill_attention(q, k, v, sm_margin=1, **kw))
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
