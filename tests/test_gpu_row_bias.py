"""Query and output biases inside the biased prefill kernel: the same bits as adding them with passes of
their own in front of and behind it. One query tile, a ragged last tile, both ways of giving a CTA its
tiles (up to 148 tiles share one CTA each between its two slots, hundreds come in pairs), biases that
repeat along a dimension, one bias alone, all masks, grouped heads, operands and score chains that the
fused form cannot take, and the result itself in 64 bits."""
import pytest
import torch

from loopfuse_b200 import _native, functional as F, loopfuse_backend, spec as S
from oracle import attention_oracle as O
import loopfuse_b200.ops  # noqa: F401  (registers loopfuse::causal_mask)

pytestmark = pytest.mark.gpu


def _biased(q, k, v, q_bias, score_bias, out_bias):
    s = (q + q_bias) @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
    s = s * 3.5 + score_bias
    return torch.softmax(torch.ops.loopfuse.causal_mask(s), dim=-1) @ v + out_bias


def _separate(q, k, v, q_bias, score_bias, out_bias):
    out = F.prefill_attention(F.add_bf16(q, q_bias), k, v, scale=q.shape[-1] ** -0.5,
                              mods=[S.ScoreMod(S.MOD_MUL, 3.5)], mask_kind=S.MASK_CAUSAL,
                              score_bias=score_bias)
    return F.add_bf16(out, out_bias)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,n", [(1, 2, 8), (1, 3, 136), (2, 3, 776), (5, 16, 264)])
def test_same_bits_as_separate_adds(B, H, n, D):
    g = torch.Generator(device="cuda").manual_seed(n + D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    q, k, v = mk(B, H, n, D), mk(B, H, n, D), mk(B, H, n, D)
    args = (q, k, v, mk(B, H, n, D), mk(B, H, n, n), mk(B, H, n, D))
    fn = torch.compile(_biased, backend=loopfuse_backend, dynamic=True)
    assert torch.equal(fn(*args), _separate(*args))
    one_row = mk(1, H, 1, D).expand(B, H, n, D)                       # strides of 0
    args = (q, k, v, one_row, args[4], one_row)
    assert torch.equal(fn(*args), _separate(*args))
    odd = mk(B, H, n, D + 4)[..., :D]                                 # rows that are not 16-byte aligned
    with pytest.raises(_native.LfError, match="lf_add_bf16 failed.*align"):
        fn(q, k, v, odd, args[4], one_row)


@pytest.mark.parametrize("D", [64, 128])
def test_rows_past_the_last_one_get_no_query_bias(D):
    """Rows past Sq share a warp with the last ones, and a warp repeats a block with its own maximum when any
    row's sum leaves its range. Here only those rows could ask for it, by the query bias of the last row
    (which that row's Q cancels), in a block where valid rows score 2^10 above their reference."""
    n = 200
    g = torch.Generator(device="cuda").manual_seed(D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16() * 0.2
    q, k, v, q_bias, score_bias, out_bias = mk(1, 1, n, D), mk(1, 1, n, D), mk(1, 1, n, D), \
        mk(1, 1, n, D), mk(1, 1, n, n), mk(1, 1, n, D)
    up = D ** 0.5 / 3.5 / 1.4427       # q . k that moves a score by 1 in the log2 domain
    for t in (q, k, q_bias):
        t[..., :2] = 0
    q_bias[..., n - 1, 0], q[..., n - 1, 0] = 16.0, -16.0
    k[..., 128:192, 0] = 24 * up / 16
    q[..., 192:n - 1, 1] = 8.0
    k[..., 150, 1] = 11 * up / 8
    args = (q, k, v, q_bias, score_bias, out_bias)
    fn = torch.compile(_biased, backend=loopfuse_backend, dynamic=True)
    assert torch.equal(fn(*args), _separate(*args))


def _allocations(call):
    """Device allocations of one call (its inputs' and the compiler's are behind it)."""
    call()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    call()
    return torch.cuda.memory_stats()["allocation.all.allocated"] - before


def test_status_checking_calls_run_the_fused_kernel(monkeypatch):
    """A call with a status word takes the same single launch: the output is all it allocates (adds of
    their own would also allocate a Q), and the word stays clean."""
    g = torch.Generator(device="cuda").manual_seed(8)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    n, D = 136, 64
    args = (mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, n),
            mk(1, 2, n, D))
    want = _separate(*args)
    monkeypatch.setenv("LF_CHECK_STATUS", "1")
    fn = torch.compile(_biased, backend=loopfuse_backend, dynamic=True)
    assert torch.equal(fn(*args), want)
    assert _allocations(lambda: fn(*args)) == 1
    q, k, v, q_bias, score_bias, out_bias = args
    st = F.new_status("cuda")
    out = F.prefill_attention(q, k, v, scale=D ** -0.5, mods=[S.ScoreMod(S.MOD_MUL, 3.5)],
                              mask_kind=S.MASK_CAUSAL, score_bias=score_bias, q_bias=q_bias,
                              out_bias=out_bias, status=st)
    F.check_status(st)
    assert torch.equal(out, want)


@pytest.mark.parametrize("which", ["q_bias", "out_bias"])
@pytest.mark.parametrize("fits", [True, False])
def test_misaligned_row_biases_are_refused_before_any_launch(which, fits):
    """Whether the graph could take the biases in one launch or not (a tanh in front of the score bias)."""
    g = torch.Generator(device="cuda").manual_seed(9)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    n, D = 136, 64
    q, k, v, sb, good = mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, n), mk(1, 2, n, D)
    odd = mk(1, 2, n, D + 4)[..., :D]
    mods = [S.ScoreMod(S.MOD_MUL, 3.5)] if fits else [S.ScoreMod(S.MOD_TANH)]
    rows = dict(q_bias=good, out_bias=good)
    call = lambda: F.prefill_attention(q, k, v, mods=mods, score_bias=sb, **rows)
    call()
    rows[which] = odd
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    with pytest.raises(_native.LfError, match="lf_add_bf16 failed.*align"):
        call()
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before


def test_biases_that_are_added_by_passes_of_their_own_cost_one_buffer():
    """A tanh in front of the score bias: the biased Q and the output are all that a call allocates."""
    def attention(q, k, v, q_bias, score_bias, out_bias):
        s = (q + q_bias) @ k.transpose(-2, -1) * (q.shape[-1] ** -0.5)
        return torch.softmax(torch.tanh(s) + score_bias, dim=-1) @ v + out_bias

    g = torch.Generator(device="cuda").manual_seed(10)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    n, D = 136, 64
    args = (mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, n),
            mk(1, 2, n, D))
    fn = torch.compile(attention, backend=loopfuse_backend, dynamic=True)
    assert _allocations(lambda: fn(*args)) == 2


def _in_passes(q, k, v, q_bias=None, out_bias=None, **options):
    """The same with each bias added by a pass of its own."""
    if q_bias is not None:
        q = F.add_bf16(q, q_bias)
    out = F.prefill_attention(q, k, v, **options)
    return out if out_bias is None else F.add_bf16(out, out_bias)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows", [("q_bias",), ("out_bias",), ("q_bias", "out_bias")])
@pytest.mark.parametrize("mask,Sq,Skv", [
    (dict(), 130, 193), (dict(mask_kind=S.MASK_CAUSAL), 257, 257),
    (dict(mask_kind=S.MASK_CAUSAL, causal_offset=300), 77, 377),
    (dict(mask_kind=S.MASK_CAUSAL_WINDOW, window=70), 321, 321)])
def test_one_or_both_biases_under_each_mask(mask, Sq, Skv, rows, D):
    """Grouped heads, score bias rows padded to 16 bytes; against separate passes bit for bit, and
    against 64 bits: P, the row sum, the attention and its sum with the output bias are each rounded by
    at most 2^-8 of their value."""
    g = torch.Generator().manual_seed(Sq + D)
    mk = lambda *s: torch.randn(*s, generator=g).bfloat16()
    q, k, v = mk(2, 4, Sq, D), mk(2, 2, Skv, D), mk(2, 2, Skv, D)
    wide = mk(2, 4, Sq, (Skv + 7) // 8 * 8)
    bias = {n: mk(2, 4, Sq, D) for n in rows}
    dev = {n: t.cuda() for n, t in bias.items()}
    options = dict(scale=D ** -0.5, mods=[S.ScoreMod(S.MOD_MUL, 3.5)],
                   score_bias=wide.cuda()[..., :Skv], **mask)
    st = F.new_status("cuda")
    got = F.prefill_attention(q.cuda(), k.cuda(), v.cuda(), status=st, **options, **dev)
    F.check_status(st)
    assert torch.equal(got, _in_passes(q.cuda(), k.cuda(), v.cuda(), **options, **dev))
    qq = (q + bias["q_bias"] if "q_bias" in bias else q).double()
    kk, vv = (t.double().repeat_interleave(2, dim=1) for t in (k, v))
    s = qq @ kk.transpose(-2, -1) * (D ** -0.5 * 3.5) + wide[..., :Skv].double()
    if "window" in mask:
        s = O.sliding_mask_ref(s, mask["window"])
    elif mask:
        s = O.causal_mask_general(s, mask.get("causal_offset", 0))
    p = torch.softmax(s, dim=-1)
    attention = p @ vv
    want = attention + bias["out_bias"].double() if "out_bias" in bias else attention
    bound = (p @ vv.abs() + 2 * attention.abs() + want.abs()) * 2.0 ** -8 + 1e-5
    assert ((got.cpu().double() - want).abs() <= bound).all()


def _operands(n, D, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    return (mk(2, 4, n, D), mk(2, 4, n, D), mk(2, 4, n, D), mk(2, 4, n, D), mk(2, 4, n, n),
            mk(2, 4, n, D))


@pytest.mark.parametrize("chain,pos", [
    ([(S.MOD_MUL, 0.5), (S.MOD_TANH, 0.0), (S.MOD_MUL, 20.0)], None),   # tanh in front of the bias
    ([(S.MOD_MUL, 3.5), (S.MOD_DIV, 2.0)], 1),                          # a divisor behind it
    ([(S.MOD_ADD, 1.0)], 0)])
def test_chains_that_take_the_biases_in_passes(chain, pos):
    q, k, v, q_bias, score_bias, out_bias = _operands(200, 64, 11)
    options = dict(scale=0.125, mods=[S.ScoreMod(*m) for m in chain], score_bias=score_bias,
                   bias_pos=pos, mask_kind=S.MASK_CAUSAL)
    call = lambda: F.prefill_attention(q, k, v, q_bias=q_bias, out_bias=out_bias, **options)
    assert torch.equal(call(), _in_passes(q, k, v, q_bias, out_bias, **options))
    assert _allocations(call) == 2


def test_q_that_tma_cannot_take():
    """One row for all queries (a stride of 0): its sum with the query bias is an ordinary tensor, so the
    passes take it; without a query bias it is refused, as without any bias."""
    q, k, v, q_bias, score_bias, out_bias = _operands(200, 64, 12)
    q = q[:, :, :1].expand(2, 4, 200, 64)
    options = dict(scale=0.125, score_bias=score_bias, mask_kind=S.MASK_CAUSAL)
    got = F.prefill_attention(q, k, v, q_bias=q_bias, out_bias=out_bias, **options)
    assert torch.equal(got, _in_passes(q.contiguous(), k, v, q_bias, out_bias, **options))
    for rows in (dict(), dict(out_bias=out_bias)):
        with pytest.raises(_native.LfError, match="lf_prefill_bf16 failed.*align"):
            F.prefill_attention(q, k, v, **options, **rows)


@pytest.mark.parametrize("two_products", [False, True])
def test_biases_without_a_score_bias(two_products):
    q, k, v, q_bias, _, out_bias = _operands(200, 64, 13)
    pe = dict(q_pe=q_bias[..., :8].contiguous(), k_pe=k[..., :8].contiguous()) if two_products else {}
    options = dict(scale=0.125, mask_kind=S.MASK_CAUSAL, **pe)
    got = F.prefill_attention(q, k, v, q_bias=q_bias, out_bias=out_bias, **options)
    assert torch.equal(got, _in_passes(q, k, v, q_bias, out_bias, **options))
