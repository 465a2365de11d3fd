"""The running-max prefill kernel takes exp2 against the reference a row already has and looks for
a block's maximum only when a row sum leaves its range: rows whose later keys score far above (and
far below) everything before, at sizes around the tile edges and on both sides of the rule that
gives a CTA one query tile or two."""
import pytest
import torch

from loopfuse_b200 import functional as F, spec as S
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("gain", [0.0, 3.0, 40.0])
@pytest.mark.parametrize("B,H,S_", [(1, 2, 127), (1, 3, 449), (4, 20, 257)])
def test_rows_whose_later_keys_score_far_above_the_first(B, H, S_, D, gain):
    g = torch.Generator().manual_seed(3)
    mk = lambda *s: torch.randn(*s, generator=g).bfloat16()
    q, k, v = mk(B, H, S_, D), mk(B, H, S_, D), mk(B, H, S_, D)
    k[:, :, S_ // 2:] *= gain      # 40: logits of +-300 in the log2 domain after blocks of +-6
    st = F.new_status("cuda")
    out = F.prefill_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5,
                              mask_kind=S.MASK_CAUSAL, status=st)
    F.check_status(st)
    want = O.attention_ref(q, k, v, mask="causal", batch_chunk=B)
    assert (out.float().cpu() - want).abs().max().item() <= TOL


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Skv,pad,shift", [(130, 193, 7, 0), (65, 64, 16, 8), (257, 1001, 15, 0)])
def test_score_bias_behind_multipliers(Sq, Skv, pad, shift, D):
    """Bias rows of 32- and of only 16-byte alignment (`shift`), blocks that cross Skv in the middle
    of an 8-column group, rows past the last tile."""
    g = torch.Generator().manual_seed(4)
    mk = lambda *s: torch.randn(*s, generator=g).bfloat16()
    q, k, v = mk(2, 3, Sq, D), mk(2, 3, Skv, D), mk(2, 3, Skv, D)
    wide = mk(2, 3, Sq, (Skv + pad + shift + 7) // 8 * 8)
    bias = wide[..., shift:shift + Skv]
    out = F.prefill_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5,
                              mods=[S.ScoreMod(S.MOD_MUL, 3.0), S.ScoreMod(S.MOD_DIV, 1.5)],
                              score_bias=wide.cuda()[..., shift:shift + Skv])
    s = q.float() @ k.float().transpose(-2, -1) * D ** -0.5 * 2.0 + bias.float()
    want = torch.softmax(s, dim=-1) @ v.float()
    assert (out.float().cpu() - want).abs().max().item() <= TOL


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("P,Skv,heads_first", [(1, 67, False), (3, 130, False), (16, 577, False),
                                               (16, 577, True)])
def test_paged_prefill_pool_layouts(P, Skv, heads_first, D):
    """Pages of one token, of no power of two, and a pool whose heads lie outside its slots (no single
    tensor of token rows: the rows are then copied by the producer warp); keys that end inside a
    tile; K and V through tables of their own."""
    g = torch.Generator().manual_seed(5)
    mk = lambda *s: torch.randn(*s, generator=g).bfloat16()
    B, Hkv, G = 2, 2, 2
    blocks = -(-Skv // P)
    pages = B * blocks + 3
    q = mk(B, Hkv * G, 150, D)
    pool = lambda: (mk(pages, Hkv, P, D).transpose(1, 2) if heads_first else mk(pages, P, Hkv, D))
    kp, vp = pool(), pool()
    table = lambda: torch.randperm(pages, generator=g)[:B * blocks].view(B, blocks).int()
    kt, vt = table(), table()
    dev = lambda t: t.cuda() if t.is_contiguous() else t.transpose(1, 2).cuda().transpose(1, 2)
    st = F.new_status("cuda")
    out = F.prefill_attention(q.cuda(), dev(kp), dev(vp), scale=D ** -0.5, k_block_table=kt.cuda(),
                              v_block_table=vt.cuda(), seq_len=Skv, status=st)
    F.check_status(st)
    want = O.attention_ref(q, O.paged_kv_ref(kp, kt)[:, :, :Skv], O.paged_kv_ref(vp, vt)[:, :, :Skv],
                           batch_chunk=B)
    assert (out.float().cpu() - want).abs().max().item() <= TOL


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,offset", [
    (1, 1, 1, 5, 5, 0),           # one block: the second slot has none
    (1, 2, 1, 33, 150, 117),      # three blocks, two and one
    (1, 3, 3, 257, 257, 0),       # tiles of two and four blocks and one row
    (1, 2, 2, 384, 256, -200),    # rows and a tile that see nothing
    (2, 160, 4, 70, 200, 130),    # more heads than SMs, one tile each
    (3, 10, 5, 1100, 1100, 0),    # 270 tiles, singles although they are not all resident
    (5, 10, 5, 1300, 1300, 0),    # pairs, two heads' worth of tiles per SM and more
])
def test_one_tile_split_over_both_slots(B, Hq, Hkv, Sq, Skv, offset, D):
    """Each slot's rows grow past the other's reference (the second half of the keys scores far above
    the first), so that the merge weighs them very differently."""
    g = torch.Generator().manual_seed(8)
    mk = lambda *s: torch.randn(*s, generator=g).bfloat16()
    q, k, v = mk(B, Hq, Sq, D), mk(B, Hkv, Skv, D), mk(B, Hkv, Skv, D)
    k[:, :, Skv // 2::3] *= 6.0
    st = F.new_status("cuda")
    out = F.prefill_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5,
                              mask_kind=S.MASK_CAUSAL, causal_offset=offset, status=st)
    F.check_status(st)
    want = O.attention_ref(q, k, v, mask="causal", offset=offset, batch_chunk=B)
    got = out.float().cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert (got - want).nan_to_num().abs().max().item() <= TOL


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("biased", [False, True])
@pytest.mark.parametrize("B,H,Sq", [(1, 2, 100), (4, 40, 256)])
def test_large_values_behind_a_low_reference_do_not_overflow(B, H, Sq, D, biased):
    """Later keys score 2^30 above the first ones and the values are of the order of 1e30: P against
    the first keys' reference, times V, would leave fp32 although the result is of V's order. 2^-8 of
    the largest value: P and the output are bf16."""
    g = torch.Generator().manual_seed(11)
    Skv = 1024
    q = torch.ones(B, H, Sq, D).bfloat16()
    k = torch.zeros(B, H, Skv, D).bfloat16()
    v = (torch.randn(B, H, Skv, D, generator=g) * 1e30).bfloat16()
    bias = None
    if biased:
        bias = torch.zeros(B, H, Sq, Skv, dtype=torch.bfloat16, device="cuda")
        bias[..., Skv // 2:] = 20.75
    else:
        k[:, :, Skv // 2:] = 20.75 / D
    out = F.prefill_attention(q.cuda(), k.cuda(), v.cuda(), score_bias=bias)
    want = v[:, :, Skv // 2:].double().mean(2, keepdim=True).expand(B, H, Sq, D)
    assert (out.double().cpu() - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item()


@pytest.mark.parametrize("biased", [False, True])
def test_row_sums_of_masked_and_first_blocks_hold_fp32_probabilities(biased):
    """All keys but the first score x1 < 0, so every P but one is exp(x1), which bf16 rounds by nearly half
    a step, and with the identity as V column 0 of a row is the reciprocal of its row sum. In 192 rows of
    one head every block is a row's first one or a masked one; their sums are taken over P in fp32 (error
    below 1e-6), so the reciprocal rounds to the bf16 nearest to the exact value. Rows where that value
    lies within 2e-5 of a rounding boundary are left out."""
    n, D = 192, 64
    x1 = -torch.arange(1, 200, dtype=torch.float64) / 128          # exact in bf16
    P = torch.exp(x1)
    off = ((P.bfloat16().double() - P) / P).abs()
    x1 = x1[off.argmax()].item()
    q, k, v = torch.zeros(1, 1, n, D), torch.zeros(1, 1, n, D), torch.zeros(1, 1, n, D)
    q[..., 0] = 1.0
    k[..., 1:, 0] = x1
    v[0, 0, 0, 0] = 1.0
    q, k, v = (t.bfloat16().cuda() for t in (q, k, v))
    bias = torch.zeros(1, 1, n, n, dtype=torch.bfloat16, device="cuda") if biased else None
    got = F.prefill_attention(q, k, v, mask_kind=S.MASK_CAUSAL, score_bias=bias)[0, 0, :, 0].cpu()
    want = 1 / (1 + torch.arange(n, dtype=torch.float64) * torch.exp(torch.tensor(x1).double()))
    clear = (want * (1 - 2e-5)).bfloat16() == (want * (1 + 2e-5)).bfloat16()
    assert clear.sum() > n - 8
    assert torch.equal(got[clear], want.bfloat16()[clear])


@pytest.mark.parametrize("D,D_pe", [(64, 0), (128, 0), (64, 8)])
@pytest.mark.parametrize("scale", [1e-38, 1e-40, 1e-45])
def test_masked_scores_with_a_scale_below_the_normal_numbers(scale, D, D_pe):
    """Scores that vanish next to 1: each row is the mean of the values that it sees. The P are 1 and
    sums of 200 values err by less than 1e-5, so half a bf16 step of the result remains."""
    g = torch.Generator().manual_seed(6)
    mk = lambda *s: torch.randn(*s, generator=g).bfloat16()
    n = 200
    q, k, v = mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, D)
    pe = dict(q_pe=mk(1, 2, n, D_pe).cuda(), k_pe=mk(1, 2, n, D_pe).cuda()) if D_pe else {}
    out = F.prefill_attention(q.cuda(), k.cuda(), v.cuda(), scale=scale, mask_kind=S.MASK_CAUSAL, **pe)
    want = v.double().cumsum(2) / torch.arange(1, n + 1, dtype=torch.float64).view(1, 1, n, 1)
    assert ((out.double().cpu() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("window", [1, 31, 32, 33, 64, 65])
def test_windows_around_the_words_of_a_block(window, D):
    """The visible columns of a row in a block are two words of 32 bits; every first and last column of a
    row occurs. A window of one key returns the values themselves."""
    g = torch.Generator().manual_seed(window)
    mk = lambda *s: torch.randn(*s, generator=g).bfloat16()
    n = 200
    q, k, v = mk(1, 2, n, D), mk(1, 2, n, D), mk(1, 2, n, D)
    out = F.prefill_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5,
                              mask_kind=S.MASK_CAUSAL_WINDOW, window=window).cpu()
    s = O.sliding_mask_ref(q.double() @ k.double().transpose(-2, -1) * D ** -0.5, window)
    want = torch.softmax(s, dim=-1) @ v.double()
    assert (out.double() - want).abs().max().item() <= TOL
    if window == 1:
        assert torch.equal(out, v)
