"""The forms of the prefill kernels, as far as they can be checked without a GPU."""
import re

import pytest

from loopfuse_b200 import build as B


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
