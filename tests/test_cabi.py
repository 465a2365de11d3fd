"""The C-ABI library without a GPU: it builds, loads, exports every declared symbol, and
rejects bad arguments with error codes before any CUDA work."""
import ctypes as C
import random
import re
from pathlib import Path

import pytest
import torch

from loopfuse_b200 import _native

HEADER = Path(__file__).resolve().parents[1] / "include" / "lf_sm100.h"


def declared_functions():
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return sorted(set(re.findall(r"\b(lf_[a-z0-9_]+)\s*\(", text)))


def test_exports_every_declared_symbol(native_lib):
    names = declared_functions()
    assert set(names) == set(_native.EXPORTS)
    for name in names:
        assert hasattr(native_lib, name), name


def test_strerror(native_lib):
    assert native_lib.lf_strerror(0) == b"ok"
    assert b"workspace" in native_lib.lf_strerror(-4)
    assert native_lib.lf_strerror(-999) == b"unknown status"


def test_workspace_bytes(native_lib):
    assert native_lib.lf_decode_workspace_bytes(64, 32, 1, 128, 1) == 0
    assert native_lib.lf_decode_workspace_bytes(64, 32, 1, 128, 4) == 64 * 32 * 4 * 130 * 4
    assert native_lib.lf_decode_workspace_bytes(64, 8, 4, 128, 8) == 64 * 8 * 4 * 8 * 130 * 4


def test_argument_validation_needs_no_gpu(native_lib):
    a = _native.LfPrefillArgs()
    assert native_lib.lf_prefill_bf16(C.byref(a), None) == -1       # null pointers
    a.q = a.k = a.v = a.out = 0x1000
    a.B, a.Hq, a.Hkv, a.Sq, a.Skv, a.D = 1, 4, 3, 128, 128, 128
    assert native_lib.lf_prefill_bf16(C.byref(a), None) == -1       # Hq % Hkv
    a.Hkv = 4
    a.D = 96
    assert native_lib.lf_prefill_bf16(C.byref(a), None) == -2       # unsupported head dim
    a.D = 128
    a.q = 0x1008
    assert native_lib.lf_prefill_bf16(C.byref(a), None) == -3       # misaligned pointer

    d = _native.LfDecodeArgs()
    assert native_lib.lf_decode_bf16(C.byref(d), None) == -1
    d.q = d.k = d.v = d.out = 0x1000
    d.B, d.Hkv, d.G, d.Skv, d.D = 2, 2, 3, 512, 128
    assert native_lib.lf_decode_bf16(C.byref(d), None) == -2        # G not in {1,2,4,8}
    d.G = 4
    d.splits = 2
    for i, s in enumerate((8192, 4096, 128)):
        d.q_stride[i] = d.o_stride[i] = s
        d.k_stride[i] = d.v_stride[i] = s
    assert native_lib.lf_decode_bf16(C.byref(d), None) == -4        # no workspace
    d.splits = 33
    assert native_lib.lf_decode_bf16(C.byref(d), None) == -7        # more than 32 splits
    d.splits = 2
    assert native_lib.lf_decode_paged_bf16(C.byref(d), None) == -1  # no block table


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_native, "_lib", None)
    monkeypatch.setattr(_native, "LIB_PATH", tmp_path / "nope.so")
    try:
        _native.load()
    except RuntimeError as e:
        assert "no fallback" in str(e)
    else:
        raise AssertionError("load() must raise when the library is missing")


def test_build_fingerprint_covers_every_included_file():
    """Every file a .cu under csrc/ #includes from the source tree is part of the rebuild
    fingerprint, so editing any of them rebuilds the library."""
    import re
    from loopfuse_b200 import build as B
    covered = {p.resolve() for p in B.fingerprint_files()}
    seen, todo = set(), [p for p in B.CSRC.glob("*.cu")]
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        for inc in re.findall(r'#include\s+"([^"]+)"', f.read_text()):
            target = (f.parent / inc).resolve()
            assert target.exists(), f"{f.name} includes missing {inc}"
            assert target in covered, f"{target} is not in the build fingerprint"
            todo.append(target)
    assert any(p.name == "lf_prefill_wide.cuh" for p in seen)


def decode_call(B, Hkv, G, Skv, D, page, splits, workspace_bytes):
    """The arguments of a decode call on made-up addresses, for what only looks at them."""
    a = _native.LfDecodeArgs()
    a.q = a.k = a.v = a.out = a.block_table = 0x1000
    a.B, a.Hkv, a.G, a.Skv, a.D, a.splits = B, Hkv, G, Skv, D, splits
    a.page_size, a.n_pages = page, 1 if page else 0
    a.workspace, a.workspace_bytes = (0x1000 if workspace_bytes else None), workspace_bytes
    return a


def test_announced_splits_and_workspace_are_what_a_call_takes(native_lib):
    """lf_decode_auto_splits, lf_decode_workspace_bytes, then a call with splits = 0 or that count:
    accepted; and the count is a power of two unless small pages ask for more than 16."""
    rng = random.Random(1)
    cases = [(2, 8, 4, 1100, 128, 0), (3, 1, 1, 2055, 128, 0), (2, 4, 4, 7369, 128, 0)]
    for _ in range(4000):
        length = int(2 ** rng.uniform(0, 16))
        cases.append((int(2 ** rng.uniform(0, 8)), rng.choice((1, 2, 3, 8, 32)),
                      rng.choice((1, 2, 4, 8)), length, rng.choice((64, 128)),
                      rng.choice((0, 0, 1, 3, 16, 24, 64))))
    for B, Hkv, G, Skv, D, page in cases:
        auto = native_lib.lf_decode_auto_splits(B, Hkv, G, Skv, D, page)
        assert auto in (1, 2, 4, 8, 16) or (page and 16 < auto <= 32), (B, Hkv, Skv, page, auto)
        need = native_lib.lf_decode_workspace_bytes(B, Hkv, G, D, auto)
        launches = [native_lib.lf_decode_launches(
            C.byref(decode_call(B, Hkv, G, Skv, D, page, n, need)), page > 0) for n in (0, auto)]
        assert launches[0] == launches[1] and launches[0] in (1, 2), (B, Hkv, G, Skv, D, page)
        n = rng.randint(2, 32)
        need = native_lib.lf_decode_workspace_bytes(B, Hkv, G, D, n)
        rc = native_lib.lf_decode_launches(C.byref(decode_call(B, Hkv, G, Skv, D, page, n, need)),
                                           page > 0)
        assert rc in (1, 2) or (page and rc == -7), (B, Hkv, G, Skv, D, page, n)
        if Skv > 64:            # (more than one split has tokens: its partials need room)
            a = decode_call(B, Hkv, G, Skv, D, page, n, 0)
            assert native_lib.lf_decode_launches(C.byref(a), page > 0) == -4


def test_many_waves_are_halved_only_where_it_pays(native_lib):
    auto = native_lib.lf_decode_auto_splits
    assert auto(64, 32, 1, 2048, 128, 0) == 2       # 256-byte rows, long caches
    assert auto(64, 32, 1, 2048, 64, 0) == 1
    assert auto(64, 32, 1, 1000, 128, 0) == 1
    assert auto(64, 32, 1, 2048, 128, 16) == 1


def test_splits_go_through_the_workspace_where_no_cluster_can_hold_them(native_lib):
    """Where the device does not say that it can hold a cluster of the splits, the combine kernel
    merges them (here: there is no device to say so)."""
    if torch.cuda.is_available():
        pytest.skip("a device is there")
    need = native_lib.lf_decode_workspace_bytes(1, 8, 4, 128, 16)
    for page in (0, 16):
        a = decode_call(1, 8, 4, 8190, 128, page, 16, need)
        assert native_lib.lf_decode_launches(C.byref(a), page > 0) == 2
        a.splits = 1
        assert native_lib.lf_decode_launches(C.byref(a), page > 0) == 1
