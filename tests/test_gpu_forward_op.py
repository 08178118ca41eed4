"""The one-operator forward call: leading dimensions, bias in the kernel's epilogue against a separate addition, biases it
does not take, strided inputs, wrong widths."""
import pytest
import torch
import torch.nn.functional as F
from torch import nn

from _util import make_input, make_weight, rel_err

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


@pytest.mark.parametrize("algo,tables", [("huffman", "limit6"), ("huffman", "escape"), ("huffman", "reference"), ("ans", None)])
@pytest.mark.parametrize("M,K", [(3, 128), (130, 4736), (1021, 4096), (260, 12288), (64, 16384)])
def test_nine_to_thirty_two_rows(algo, tables, M, K):
    """More products per decoded word: counts around the groups of eight, X in segments that end mid-way, records too long
    for shared memory, the bias inside the sum; gradients take the dense matrix."""
    from bf16_huffman_infer_b200 import ANSWeight, CompressedLinear, HuffmanWeight, set_huffman_tables
    W, bias = make_weight(M, K, 4), make_weight(1, M, 5)[0]
    previous = set_huffman_tables(tables or "limit6")
    try:
        weight = (ANSWeight if algo == "ans" else HuffmanWeight).compress_split_n(W.to(DEV), n=3 if K == 12288 else 1, to_cpu=False)
    finally:
        set_huffman_tables(previous)
    layer = CompressedLinear(weight, nn.Parameter(bias.to(DEV)))
    for rows in (9, 16, 17, 24, 25, 32):
        x = make_input(rows, K, rows)
        with torch.no_grad():
            y = layer(x.view(rows, 1, K).to(DEV))
        assert y.shape == (rows, 1, M)
        ref = x.double() @ W.double().T + bias.double()
        assert rel_err(y.view(rows, M).float().cpu().numpy(), ref.numpy()) <= 1e-2, rows
    xg = make_input(12, K, 1).to(DEV).requires_grad_()
    layer(xg).float().sum().backward()
    assert xg.grad is not None and layer.bias.grad is not None


def test_unaligned_activations():
    """Activations that start 4 bytes past a 16-byte boundary: X is staged by plain stores, whole and in segments."""
    from bf16_huffman_infer_b200 import CompressedLinear, HuffmanWeight
    for M, K, rows in ((260, 4096, 1), (260, 12288, 8), (260, 4096, 20)):
        W = make_weight(M, K, 6)
        layer = CompressedLinear(HuffmanWeight.compress(W.to(DEV), to_cpu=False), None)
        x = make_input(rows, K, 7)
        flat = torch.empty(rows * K + 8, dtype=torch.bfloat16, device=DEV)
        shifted = flat[2:2 + rows * K].view(rows, K).copy_(x)
        with torch.no_grad():
            y = layer(shifted)
        assert rel_err(y.float().cpu().numpy(), (x.double() @ W.double().T).numpy()) <= 1e-2


@pytest.mark.parametrize("algo,tables", [("huffman", "reference"), ("ans", None)])
@pytest.mark.parametrize("M", [1, 598, 1187])
def test_one_unit_rings(algo, tables, M):
    """Two rows over 18944 columns in four chunks: X stays resident beside record rings that take a single unit."""
    from bf16_huffman_infer_b200 import ANSWeight, CompressedLinear, HuffmanWeight, set_huffman_tables
    K, W = 18944, make_weight(M, 18944, 7)
    previous = set_huffman_tables(tables or "limit6")
    try:
        weight = (ANSWeight if algo == "ans" else HuffmanWeight).compress(W.to(DEV), to_cpu=False)
    finally:
        set_huffman_tables(previous)
    x = make_input(2, K, 8).to(DEV)
    y = CompressedLinear(weight, None)(x)
    want = x.float() @ W.to(DEV).float().T
    assert ((y.float() - want).norm() / want.norm()).item() < 4e-3
