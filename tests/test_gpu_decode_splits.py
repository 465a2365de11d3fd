"""Decode where its splits, CTA shapes and score functions change: clusters of 2 to 16 that merge in
shared memory (the last splits ragged or empty, block-table slices of different padding), the combine
kernel beyond 16, eight, four and two warps per CTA, the folded softcap beside the interpreted chain,
and P at more than one bf16's precision."""
import ctypes as C
import threading

import pytest
import torch

from loopfuse_b200 import _native, functional as F, spec as S
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

MODS = {
    "none": [],
    "softcap": [S.ScoreMod(S.MOD_DIV, 30.0), S.ScoreMod(S.MOD_TANH), S.ScoreMod(S.MOD_MUL, 30.0)],
    "chain": [S.ScoreMod(S.MOD_TANH), S.ScoreMod(S.MOD_ADD, 0.5), S.ScoreMod(S.MOD_MUL, 3.0)],
}


def want_of(q, k, v, mods):
    """(result, allowed error) in fp64. The result is rounded to bf16, up to 2^-8 of itself. P has two
    bf16 parts at least, 2^-18 of each weight; scores, exp2 and sums in fp32 add about 2^-19 each: 2^-16
    of the weighted |v|. tanh.approx (which fast-math tanhf is too) is 2^-11 off its value at most: a
    logit l that comes from it moves its weight, and by it the sum, by 2^-11 |l|."""
    s = (q.double() @ k.double().transpose(-1, -2)) * q.shape[-1] ** -0.5
    from_tanh = torch.zeros_like(s)
    if mods == "softcap":
        s = from_tanh = torch.tanh(s / 30.0) * 30.0
    elif mods == "chain":
        from_tanh = torch.tanh(s) * 3.0
        s = from_tanh + 1.5
    p, v = torch.softmax(s, -1), v.double()
    want, moved = p @ v, p * from_tanh.abs()
    return want, (2.0 ** -8 * want.abs() + 2.0 ** -16 * (p @ v.abs())
                  + 2.0 ** -11 * (moved @ v.abs() + moved.sum(-1, keepdim=True) * want.abs()))


def check(out, q, k, v, mods="none"):
    want, allowed = want_of(q, k, v, mods)
    assert bool(((out.double().cpu() - want).abs() <= allowed).all())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mods", ["none", "softcap", "chain"])
@pytest.mark.parametrize("B,Hkv,G,Skv,splits", [
    (1, 1, 1, 1, 0), (1, 2, 2, 3, 2), (2, 3, 1, 257, 2), (2, 3, 8, 515, 4), (1, 3, 2, 2100, 16),
    (1, 2, 4, 2100, 8), (2, 5, 4, 700, 20), (40, 8, 1, 65, 1), (56, 8, 2, 33, 1), (17, 16, 4, 130, 2),
])
def test_dense_splits(B, Hkv, G, Skv, splits, mods, D):
    g = torch.Generator().manual_seed(5)
    q, k, v = [torch.randn(B, Hkv, n, D, generator=g).bfloat16() for n in (G, Skv, Skv)]
    out = F.decode_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5, mods=MODS[mods],
                             splits=splits)
    check(out, q, k, v, mods)


@pytest.mark.parametrize("mods", ["none", "softcap", "chain"])
@pytest.mark.parametrize("B,Hkv,G,Skv,splits", [(2, 3, 1, 257, 2), (1, 3, 2, 2100, 16),
                                                (1, 2, 4, 2100, 8), (2, 5, 4, 700, 20)])
def test_the_allowed_error_sees_a_missing_split(B, Hkv, G, Skv, splits, mods):
    """Zeros, and results that lack the first or the last split, are outside of it (in the oracle)."""
    g = torch.Generator().manual_seed(5)
    q, k, v = [torch.randn(B, Hkv, n, 64, generator=g).bfloat16() for n in (G, Skv, Skv)]
    chunk = -(-Skv // splits)
    with pytest.raises(AssertionError):
        check(torch.zeros(B, Hkv, G, 64), q, k, v, mods)
    for lacking in (slice(chunk, None), slice(0, (splits - 1) * chunk)):
        out = want_of(q, k[:, :, lacking], v[:, :, lacking], mods)[0]
        with pytest.raises(AssertionError):
            check(out, q, k, v, mods)
    check(want_of(q, k, v, mods)[0].bfloat16(), q, k, v, mods)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("P,Skv,splits", [(16, 1, 0), (16, 1000, 2), (16, 2111, 16), (1, 517, 4),
                                          (24, 700, 8), (64, 1217, 8), (16, 1203, 20)])
def test_paged_splits(P, Skv, splits, D):
    B, Hkv, G = 2, 3, 4
    g = torch.Generator().manual_seed(6)
    blocks = -(-Skv // P)
    q = torch.randn(B, Hkv, G, D, generator=g).bfloat16()
    kp, vp = [torch.randn(B * blocks + 3, P, Hkv, D, generator=g).bfloat16() for _ in range(2)]
    kt, vt = [torch.randperm(B * blocks + 3, generator=g)[:B * blocks].view(B, blocks).int()
              for _ in range(2)]
    for table_v in (None, vt):
        st = F.new_status("cuda")
        out = F.paged_decode_attention(q.cuda(), kp.cuda(), vp.cuda(), kt.cuda(), seq_len=Skv,
                                       block_table_v=None if table_v is None else table_v.cuda(),
                                       scale=D ** -0.5, splits=splits, status=st)
        F.check_status(st)
        k = O.paged_kv_ref(kp, kt)[:, :, :Skv]
        v = O.paged_kv_ref(vp, kt if table_v is None else table_v)[:, :, :Skv]
        check(out, q, k, v)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hkv,G,Skv,splits", [(1, 2, 1, 40, 1), (1, 2, 2, 700, 4), (1, 2, 4, 40, 1)])
def test_infinite_values_stay_infinite(B, Hkv, G, Skv, splits, D):
    """A value row with an infinity: its weight is positive, so that column is that infinity (the
    finer parts of P must not turn it into inf - inf); a NaN stays in its column; the others are
    untouched."""
    g = torch.Generator().manual_seed(9)
    q, k, v = [torch.randn(B, Hkv, n, D, generator=g).bfloat16() for n in (G, Skv, Skv)]
    v[:, :, 5, 3], v[:, :, 17, 9], v[:, :, 21, 40] = float("inf"), float("-inf"), float("nan")
    out = F.decode_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5, splits=splits).cpu()
    assert bool((out[..., 3] == float("inf")).all()) and bool((out[..., 9] == float("-inf")).all())
    assert bool(out[..., 40].isnan().all())
    v[:, :, [5, 17, 21], [3, 9, 40]] = 0.0
    keep = [c for c in range(D) if c not in (3, 9, 40)]
    check(out[..., keep], q, k, v[..., keep])


@pytest.mark.parametrize("B,Hkv,G,Skv", [(2, 8, 4, 1100), (3, 1, 1, 2055), (2, 4, 4, 7369)])
def test_library_chosen_splits_of_ragged_lengths(B, Hkv, G, Skv):
    """Lengths that a chunk of 64 would cut into 6, 11 and 15 splits: eights and sixteens, the last of
    them with few tokens or none."""
    g = torch.Generator().manual_seed(10)
    q, k, v = [torch.randn(B, Hkv, n, 128, generator=g).bfloat16() for n in (G, Skv, Skv)]
    auto = _native.load().lf_decode_auto_splits(B, Hkv, G, Skv, 128, 0)
    assert auto in (8, 16)
    out = F.decode_attention(q.cuda(), k.cuda(), v.cuda(), scale=128 ** -0.5)
    check(out, q, k, v)
    again = F.decode_attention(q.cuda(), k.cuda(), v.cuda(), scale=128 ** -0.5, splits=auto)
    assert torch.equal(out, again)


def test_static_scratch_splits_only_as_far_as_its_partials_fit():
    """A grid of many waves that the library would split in two, with partials of 17 MB: unsplit."""
    lib = _native.load()
    q = torch.randn(64, 32, 8, 128, device="cuda").bfloat16()
    k, v = [torch.randn(64, 1, 2000, 128, device="cuda").bfloat16().expand(64, 32, 2000, 128)
            for _ in range(2)]
    assert lib.lf_decode_auto_splits(64, 32, 8, 2000, 128, 0) == 2
    want = F.decode_attention(q, k, v, scale=128 ** -0.5, splits=1)
    out = torch.empty_like(q)
    a = _native.LfDecodeArgs()
    a.q, a.k, a.v, a.out = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr()
    a.B, a.Hkv, a.G, a.Skv, a.D, a.scale = 64, 32, 8, 2000, 128, 128 ** -0.5
    for i in range(3):
        a.q_stride[i], a.o_stride[i] = q.stride(i), out.stride(i)
        a.k_stride[i], a.v_stride[i] = k.stride(i), v.stride(i)
    assert lib.lf_decode_bf16_static(C.byref(a), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(out, want)
    a.splits = 2
    assert lib.lf_decode_bf16_static(C.byref(a), torch.cuda.current_stream().cuda_stream) == -7


def many_splits(seed):
    """20 splits, whose partials go through a workspace; the values tell the seeds apart."""
    g = torch.Generator().manual_seed(seed)
    q, k, v = [torch.randn(2, 4, n, 128, generator=g).bfloat16().cuda() for n in (4, 1700, 1700)]
    return lambda **kw: F.decode_attention(q, k, v + seed, scale=128 ** -0.5, splits=20, **kw)


def test_two_streams_and_two_threads_do_not_share_partials():
    calls = [many_splits(1), many_splits(2)]
    want = [c() for c in calls]
    torch.cuda.synchronize()
    got = [[], []]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    ws = F.DecodeWorkspace()
    for kw in ({}, {"workspace": ws}):
        for _ in range(100):
            for i in range(2):
                with torch.cuda.stream(streams[i]):
                    got[i].append(calls[i](**kw))

    def loop(i):
        for _ in range(200):
            got[i].append(calls[i]())

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(2):
        assert len(got[i]) == 400 and all(torch.equal(o, want[i]) for o in got[i])


def test_a_workspace_keeps_its_buffer_on_its_stream_only():
    ws, call = F.DecodeWorkspace(), many_splits(3)
    want = call(workspace=ws)
    first = ws._buf
    assert torch.equal(call(workspace=ws), want) and ws._buf is first
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
        assert torch.equal(call(workspace=ws), want) and ws._buf is not first
    torch.cuda.synchronize()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("G,Skv,splits", [(1, 130, 2), (4, 17, 2), (1, 300, 4), (2, 200, 16)])
def test_splits_of_grids_of_many_waves(G, Skv, splits, D):
    """More than eight CTAs per SM: the partials go through the workspace (and counts are trimmed to
    chunks of 64 tokens)."""
    B, Hkv = 40, 32
    g = torch.Generator().manual_seed(14)
    q, k, v = [torch.randn(B, Hkv, n, D, generator=g).bfloat16() for n in (G, Skv, Skv)]
    out = F.decode_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5, splits=splits)
    check(out, q, k, v)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hkv,G,Skv,splits,page", [
    (1, 2, 4, 700, 1, 0), (1, 2, 8, 2100, 16, 0), (2, 3, 4, 515, 0, 0), (40, 8, 8, 65, 1, 0),
    (2, 3, 1, 517, 4, 1), (2, 2, 8, 1000, 2, 16), (70, 8, 4, 130, 1, 16), (2, 2, 2, 1203, 20, 24),
])
def test_probabilities_keep_two_bf16_parts(B, Hkv, G, Skv, splits, page, D):
    """However the keys are dealt out to warps and splits, P's rounding does not show (with P in one
    bf16, 2^-9 of each weight, it does)."""
    g = torch.Generator().manual_seed(15)
    q, k, v = [torch.randn(B, Hkv, n, D, generator=g).bfloat16() for n in (G, Skv, Skv)]
    if not page:
        out = F.decode_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5, splits=splits)
    else:
        blocks = -(-Skv // page)
        table = torch.randperm(B * blocks, generator=g).view(B, blocks).int()
        pools = []
        for x in (k, v):
            pool = torch.zeros(B * blocks, page, Hkv, D).bfloat16()
            rows = torch.nn.functional.pad(x, (0, 0, 0, blocks * page - Skv)).transpose(1, 2)
            pool[table.long()] = rows.reshape(B, blocks, page, Hkv, D)
            pools.append(pool.cuda())
        out = F.paged_decode_attention(q.cuda(), *pools, table.cuda(), seq_len=Skv,
                                       scale=D ** -0.5, splits=splits)
    check(out, q, k, v)


@pytest.mark.parametrize("splits", range(2, 21))
def test_every_split_count_merges(splits):
    """Clusters of up to 16, which a whole B200 can hold, and the combine kernel beyond."""
    B, Hkv, G, Skv, D = 1, 3, 4, 1003, 128
    g = torch.Generator().manual_seed(16)
    q, k, v = [torch.randn(B, Hkv, n, D, generator=g).bfloat16() for n in (G, Skv, Skv)]
    out = F.decode_attention(q.cuda(), k.cuda(), v.cuda(), scale=D ** -0.5, splits=splits)
    check(out, q, k, v)
    a = _native.LfDecodeArgs()
    a.q = a.k = a.v = a.out = a.workspace = q.data_ptr()     # (only looked at)
    a.workspace_bytes = 1 << 30
    a.B, a.Hkv, a.G, a.Skv, a.D, a.splits = B, Hkv, G, Skv, D, splits
    assert _native.load().lf_decode_launches(C.byref(a), 0) == (1 if splits <= 16 else 2)
