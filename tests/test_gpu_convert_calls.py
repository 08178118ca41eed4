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


@pytest.mark.parametrize("algo", ["huffman", "ans", "smallest"])
def test_capture_right_after_conversion(algo):
    """A layer converted on the device is captured without a call before: its folded tables are there."""
    from bf16_huffman_infer_b200 import CompressedLinear, convert
    linear = nn.Linear(1536, 512, dtype=torch.bfloat16, device=DEV).requires_grad_(False)
    linear.weight.copy_(make_weight(512, 1536, 2))
    x = make_weight(1, 1536, 3).to(DEV)
    want = F.linear(x, linear.weight, linear.bias)
    layer = convert(linear, "layer", algo=algo)
    assert isinstance(layer, CompressedLinear)
    if algo != "ans":
        assert "_prepared" in layer.weight.__dict__ or layer.weight.algo == "ans"
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph):
        y = layer(x)
    graph.replay()
    torch.cuda.synchronize()
    assert ((y - want).double().norm() / want.double().norm()).item() < 2.0 ** -8
