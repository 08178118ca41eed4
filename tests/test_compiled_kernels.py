"""What the compiler made of the kernels, from the logs that the build leaves (ptxas -v)."""
import os
import re

import pytest

from _util import ROOT

BUILD = os.path.join(ROOT, "bf16_huffman_infer_b200", "build")
# gemv_kernel<Dec, NB, NG, kRing, kShard, kHalf, kFew, kShift>
NAME = re.compile(r"gemv_kernel.*ELi(\d)ELi(\d)ELb(\d)ELi(\d)ELb(\d)ELb(\d)ELb(\d)EE")


def _kernels():
    """(template arguments, registers, bytes spilled) of each fused kernel"""
    for log in ("bhi_gemv_huffman.log", "bhi_gemv_ans.log"):
        path = os.path.join(BUILD, log)
        if not os.path.exists(path):
            pytest.skip("no build log")
        for part in open(path).read().split("Compiling entry function '")[1:]:
            name = NAME.search(part[:part.index("'")])
            if name:
                spilled = re.search(r"(\d+) bytes spill stores", part)
                yield tuple(map(int, name.groups())), int(re.search(r"Used (\d+) registers", part).group(1)), int(spilled.group(1)) if spilled else 0


def test_register_shifts_have_what_they_hand_out():
    """A kernel whose sixteen decoding warps go up to 112 registers a thread needs 96 in all of its 640 threads at the launch;
    with fewer, the wait for them would have no end."""
    shifting = [(args, registers) for args, registers, _ in _kernels() if args[-1]]
    assert shifting
    for args, registers in shifting:
        assert args[1] == 4 and args[2] == 1 and registers == 96, (args, registers)
        assert 640 * registers >= 512 * 112 + 128 * 32
