"""Conversions under settings of the calling program: default devices, other element types, captures that follow."""
import pytest
import torch
import torch.nn.functional as F
from torch import nn

from _util import make_weight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _classes():
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight
    return HuffmanWeight, ANSWeight


@pytest.mark.parametrize("default", ["cuda:0", "meta"])
@pytest.mark.parametrize("home", ["cpu", DEV])
@pytest.mark.parametrize("to_cpu", [True, False])
def test_default_device(default, home, to_cpu):
    """Host tensors of a conversion are host tensors whatever torch's default device is (3 MB: in slabs)."""
    W = make_weight(1024, 1536, 0)
    for cls in _classes():
        with torch.device(default):
            weight = cls.compress(W.to(home), to_cpu=to_cpu)
        assert {b.device.type for b in weight.buffers()} == {"cpu" if to_cpu else "cuda"}
        assert torch.equal(weight.to(DEV).get_weight().cpu(), W)
