"""The one-operator forward call: leading dimensions, bias in the kernel's epilogue against a separate addition, biases it
does not take, strided inputs, wrong widths."""
import pytest
import torch
import torch.nn.functional as F
from torch import nn

from _util import make_input, make_weight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("algo,tables", [("huffman", "limit6"), ("huffman", "escape"), ("ans", None)])
@pytest.mark.parametrize("M,K,lead", [(1, 384, (1,)), (130, 512, (2, 1, 3)), (1021, 4096, (8, 1)), (257, 12288, (4,))])
def test_forward_call(algo, tables, M, K, lead):
    from bf16_huffman_infer_b200 import ANSWeight, CompressedLinear, HuffmanWeight, set_huffman_tables
    previous = set_huffman_tables(tables or "limit6")
    try:
        weight = (ANSWeight if algo == "ans" else HuffmanWeight).compress(make_weight(M, K, 1).to(DEV), to_cpu=False)
    finally:
        set_huffman_tables(previous)
    rows = 1
    for d in lead:
        rows *= d
    x = make_input(rows, K, 2).view(*lead, K).to(DEV)
    bias = make_weight(1, M, 3)[0].to(DEV)
    with torch.no_grad():
        plain = CompressedLinear(weight, None)(x)
        assert plain.shape == lead + (M,)
        assert torch.equal(plain, weight._mv(x.flatten(0, -2)).view(plain.shape))
        assert torch.equal(F.linear(x, weight), plain)
        wide = torch.stack([x, x], dim=-1)[..., 0]                           # the same values, two elements apart
        assert torch.equal(CompressedLinear(weight, None)(wide), plain)
        for b in (bias, bias.float(), torch.stack([bias, bias], dim=-1)[:, 0]):
            want = plain.clone()
            want += b
            assert torch.equal(CompressedLinear(weight, nn.Parameter(b))(x), want)
        with pytest.raises((RuntimeError, AssertionError)):
            F.linear(x[..., :-128], weight)
        with pytest.raises((RuntimeError, AssertionError)):
            F.linear(x.float(), weight)
    trained = nn.Parameter(bias.clone())
    CompressedLinear(weight, trained)(x).float().sum().backward()
    assert trained.grad is not None and torch.equal(trained.grad, torch.full_like(bias, rows))
