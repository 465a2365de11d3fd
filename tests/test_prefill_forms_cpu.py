"""The forms of the prefill kernels, as far as they can be checked without a GPU."""
import ctypes as C
import os
import re
import subprocess
import sys

import pytest

from loopfuse_b200 import _native, build as B, spec as S


def test_registers_change_hands_once_per_warpgroup():
    """setmaxnreg has to be the same instruction for the four warps of a warpgroup, under a condition that all
    of them evaluate alike: one `dec` in front of the roles of the upper warpgroup, one `inc` at the top of the
    softmax branch, and a sum that the block was launched with (a larger one would never be granted)."""
    code = re.sub(r"//.*", "", (B.CSRC / "lf_prefill.cu").read_text())
    assert re.findall(r"setmaxnreg\.(\w+)", code) == ["dec", "inc"]
    dec = re.search(r"if constexpr \(NARROW\) \{\s*if \(warp >= kSoftmaxWarps\) "
                    r'asm volatile\("setmaxnreg\.dec\.sync\.aligned\.u32 (\d+);"\);\s*\}', code)
    inc = re.search(r"\} else if \(warp < kSoftmaxWarps\) \{\s*if constexpr \(NARROW\) "
                    r'asm volatile\("setmaxnreg\.inc\.sync\.aligned\.u32 (\d+);"\);', code)
    roles = code.index("if ((warp == kProducerWarp || warp == kGatherWarp) && p.gather)")
    assert dec and inc and dec.end() < roles < inc.start()
    few, many = int(dec[1]), int(inc[1])
    assert few % 8 == 0 and many % 8 == 0
    for name in ("build.log", "build_dbg.log"):
        log = B.CSRC / name
        if not log.exists():
            pytest.skip(f"{name}: not built in this tree")
        forms = re.findall(r"Compiling entry function '\w*prefill_kernelILi\d+ELi\d+ELb[01]ELb1E\w*'.*?"
                           r"(\d+) bytes spill stores.*?Used (\d+) registers", log.read_text(), re.S)
        assert len(forms) == 4
        for spill, regs in forms:
            assert 4 * few + 4 * many <= 8 * int(regs) and int(regs) * 512 <= 65536


PAIRS, SPLIT, NARROW = range(3)
SOFTCAP = [(S.MOD_DIV, 50.0), (S.MOD_TANH, 0.0), (S.MOD_MUL, 50.0)]


def call(B, Hq, Hkv, Sq, Skv, D, *, mask=S.MASK_CAUSAL, window=0, off=None, softcap=False, bias=False, page=0,
         margin=0, kv_tile=0):
    """The arguments of a prefill on made-up addresses, for what only looks at them."""
    a = _native.LfPrefillArgs()
    a.q = a.k = a.v = a.out = 0x1000
    a.B, a.Hq, a.Hkv, a.Sq, a.Skv, a.D = B, Hq, Hkv, Sq, Skv, D
    for i, (s, t) in enumerate(((Hq * Sq * D, Hkv * Skv * D), (Sq * D, Skv * D), (D, D))):
        a.q_stride[i] = a.o_stride[i] = s
        a.k_stride[i] = a.v_stride[i] = t
    a.scale, a.mask_kind, a.window = D ** -0.5, mask, window
    a.causal_offset = Skv - Sq if off is None else off
    a.sm_margin, a.kv_tile = margin, kv_tile
    if softcap:
        a.n_mod = len(SOFTCAP)
        for i, (op, arg) in enumerate(SOFTCAP):
            a.mod_op[i], a.mod_arg[i] = op, arg
    if bias:
        a.score_bias = 0x1000
        row = (Skv + 7) // 8 * 8
        for i, s in enumerate((Hq * Sq * row, Sq * row, row)):
            a.bias_stride[i] = s
    if page:
        a.k_block_table = 0x1000
        a.page_size, a.n_pages, a.bt_stride = page, B * -(-Skv // page), -(-Skv // page)
        for i, s in enumerate((page * Hkv * D, Hkv * D, D)):
            a.k_stride[i] = s
    return a


def form(lib, *args, sms=148, **kw):
    return lib.lf_prefill_form(C.byref(call(*args, **kw)), sms)


def test_form_query(native_lib):
    """The query answers for any number of SMs without a device, by the same rules as a call."""
    ask = lambda *a, **kw: form(native_lib, *a, **kw)
    assert ask(4, 8, 8, 593, 593, 64) == ask(4, 8, 8, 593, 593, 128) == SPLIT      # 160 tiles
    assert ask(1, 8, 8, 512, 512, 64) == SPLIT                                     # fewer than SMs
    assert ask(8, 32, 32, 2048, 2048, 64) == NARROW
    assert ask(8, 32, 32, 2048, 2048, 128) == PAIRS
    assert ask(8, 32, 8, 512, 512, 128) == NARROW
    assert ask(8, 32, 8, 512, 512, 128, sms=4000) == SPLIT
    assert ask(8, 32, 8, 512, 512, 128, page=16) == NARROW
    assert ask(8, 16, 16, 512, 512, 128, bias=True) == NARROW
    assert ask(8, 32, 32, 2048, 2048, 128, softcap=True) == PAIRS
    assert ask(8, 32, 32, 2048, 2048, 64, softcap=True) == NARROW
    assert ask(8, 32, 32, 2048, 2048, 64, softcap=True, margin=1) == PAIRS
    assert ask(8, 32, 32, 2048, 2048, 64, softcap=True, kv_tile=128) == PAIRS
    assert ask(8, 32, 8, 2048, 2048, 128, softcap=True, mask=S.MASK_CAUSAL_WINDOW, window=256) == PAIRS
    assert ask(1, 32, 8, 1024, 1024, 128, softcap=True, mask=S.MASK_CAUSAL_WINDOW, window=256) == NARROW
    a = call(8, 32, 32, 2048, 2048, 128)
    assert native_lib.lf_prefill_form(C.byref(a), -1) == -1
    assert native_lib.lf_prefill_q_tile(C.byref(a)) == 128
    a.D = 96
    assert native_lib.lf_prefill_form(C.byref(a), 148) == -2


def test_one_tile_a_head(native_lib):
    """Narrow, but for long biased rows where split tiles take three rounds of half the steps against two."""
    ask = lambda heads, keys, D=64, **kw: form(native_lib, 1, heads, heads, 128, keys, D, **kw)
    for D in (64, 128):
        assert [ask(n, 2048, D, bias=True) for n in (149, 296, 297, 444, 445, 900)] == [
            NARROW, NARROW, SPLIT, SPLIT, NARROW, NARROW]
        assert [ask(320, keys, D, bias=True) for keys in (64, 700, 704, 705, 8192)] == [
            NARROW, NARROW, NARROW, SPLIT, SPLIT]
        assert [ask(n, 2048, D) for n in (149, 320, 444, 900)] == [NARROW] * 4
        assert ask(148, 2048, D) == SPLIT


def test_empty_slots_of_pairs(native_lib):
    """D = 128, past two tiles per SM: long rows take narrow only where a head has three tiles, or five and there are
    many of them; three plain tiles a head keep pairs in between where narrow needs half a round more."""
    ask = lambda heads, rows, keys, **kw: form(native_lib, 1, heads, heads, rows, keys, 128, **kw)
    for kw in ({}, dict(page=16)):
        assert [ask(h, 300, 4300, **kw) for h in (99, 108, 109, 128, 147, 148, 900)] == [NARROW] * 2 + [PAIRS] * 3 + [NARROW] * 2
        assert [ask(128, 300, keys, **kw) for keys in (1280, 1281, 6336, 6337)] == [NARROW, PAIRS, PAIRS, NARROW]
        assert [ask(148, 300, keys, **kw) for keys in (1280, 1281, 6336)] == [NARROW] * 3
        assert [ask(h, 600, 4300, **kw) for h in (60, 128, 177, 178, 500)] == [PAIRS] * 3 + [NARROW] * 2
        assert [ask(h, rows, 4300, **kw) for h in (160, 900) for rows in (200, 500, 900, 1100)] == [PAIRS] * 8
        assert [ask(h, rows, 1500, **kw) for h in (160, 900) for rows in (200, 500, 600, 900, 1100)] == [NARROW] * 10
    assert [ask(h, 300, 4300, bias=True) for h in (99, 128, 148)] == [NARROW] * 3


@pytest.mark.parametrize("D", [64, 128])
def test_one_to_two_tiles_per_sm(native_lib, D):
    """Pairs that all find an SM stay where the longest tile would lose its own; pairs that need a second round
    do not, unless the light ones make it."""
    ask = lambda heads, rows, keys, **kw: form(native_lib, 1, heads, heads, rows, keys, D, **kw)
    narrow_64 = NARROW if D == 64 else PAIRS
    # three tiles a head: 74 heads fill 148 SMs with pairs
    assert [ask(h, 384, 384) for h in (50, 59, 60, 74, 75, 98)] == [narrow_64] * 2 + [PAIRS] * 2 + [NARROW] * 2
    assert [ask(h, 384, 2000) for h in (50, 60, 74, 75, 98)] == [narrow_64] * 3 + [NARROW] * 2
    assert [ask(h, 384, 1200, page=16) for h in (50, 60, 74, 75, 98)] == [NARROW, PAIRS, PAIRS, NARROW, NARROW]
    # two, four: an SM for every pair always
    assert [ask(h, 256, 256) for h in (75, 90, 148)] == [narrow_64] * 3
    assert [ask(h, 256, 256, page=16) for h in (75, 90, 148)] == [NARROW] + [narrow_64] * 2
    assert [ask(h, 512, 512, page=16) for h in (45, 74)] == [NARROW] * 2
    assert [ask(h, 896, 1496) for h in (36, 40)] == [PAIRS if D == 128 else NARROW, NARROW]
    # the persistent kernel
    soft = lambda heads, rows, keys: ask(heads, rows, keys, softcap=True)
    assert [soft(h, 384, 384) for h in (50, 59, 60, 74, 75, 98)] == [NARROW] * 2 + [PAIRS] * 2 + [NARROW] * 2
    assert [soft(h, 384, 3384) for h in (60, 74, 75, 98)] == [PAIRS] * 2 + [NARROW] * 2
    assert [soft(h, 256, 256) for h in (75, 90, 148)] == [NARROW] + [narrow_64] * 2
    assert [soft(h, 512, 512) for h in (45, 74)] == [NARROW] * 2
    # (seven, causal: the light pairs of 40 heads fit behind the long ones, with more keys in front they do not)
    assert [soft(40, 896, 896 + more) for more in (0, 600)] == [PAIRS, NARROW]


def test_softcap_tiles_with_an_sm_each(native_lib):
    """Where a head has one tile, both forms give it an SM: the one with the deeper ring."""
    ask = lambda heads, rows, keys, D: form(native_lib, 1, heads, heads, rows, keys, D, softcap=True)
    assert [ask(h, 100, keys, 128) for h in (1, 148) for keys in (100, 1000, 8000)] == [PAIRS] * 6
    assert [ask(149, 100, keys, 128) for keys in (100, 600)] == [NARROW] * 2
    assert [ask(h, 100, 1000, 64) for h in (1, 148, 149)] == [NARROW] * 3
    assert [ask(h, 256, 1000, 128) for h in (1, 74)] == [NARROW] * 2


FAKE_RUNTIME = r"""
static int current, asked;
extern "C" {
void fake_set(int dev) { current = dev; }
int fake_asked() { return asked; }
int cudaGetDevice(int* dev) { *dev = current; return 0; }
int cudaDeviceGetAttribute(int* value, int attribute, int dev) { ++asked; *value = dev == 0 ? 148 : 4000; return 0; }
}
"""
ASK = """
import ctypes as C, sys
fake, lib = C.CDLL(sys.argv[1], mode=C.RTLD_GLOBAL), C.CDLL(sys.argv[2])
args = C.create_string_buffer(bytes.fromhex(sys.argv[3]))
for dev in (0, 1, 0, 1):
    fake.fake_set(dev)
    print(lib.lf_prefill_form(args, 0))
print(fake.fake_asked())
"""


def test_number_of_sms_is_the_current_devices(native_lib, tmp_path):
    """Two devices of different size behind a stand-in for the CUDA runtime's two queries: each is asked once,
    and a thread that changes device gets the form for the one it is on."""
    shim = tmp_path / "fake.so"
    (tmp_path / "fake.cpp").write_text(FAKE_RUNTIME)
    subprocess.run(["g++", "-shared", "-fPIC", str(tmp_path / "fake.cpp"), "-o", str(shim)], check=True)
    args = bytes(call(8, 32, 8, 512, 512, 128)).hex()
    out = subprocess.run([sys.executable, "-c", ASK, str(shim), str(_native.LIB_PATH), args], check=True, text=True,
                         capture_output=True, env=dict(os.environ, LD_PRELOAD=str(shim)))
    assert [int(x) for x in out.stdout.split()] == [NARROW, SPLIT, NARROW, SPLIT, 2]
