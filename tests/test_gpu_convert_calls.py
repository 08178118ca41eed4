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


@pytest.mark.parametrize("dtype", [torch.float16, torch.int16])
def test_codec_of_bits(dtype):
    """The code of a tensor whose bits are BF16 values, whatever type they are declared as."""
    W = make_weight(64, 256, 1).to(DEV)
    for cls in _classes():
        a, b = cls.get_lut_kwargs(cls.get_codec(W)), cls.get_lut_kwargs(cls.get_codec(W.view(dtype)))
        assert all(torch.equal(a[k], b[k]) for k in a)
