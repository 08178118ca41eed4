"""Layers whose rows differ in scale: records of very different lengths in one unit.  Units that fit their ring whole, quad by
quad and not at all stand side by side, and the results do not depend on which is which."""
import pytest
import torch

from _util import make_input, make_weight, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("algo,tables", [("huffman", "limit6"), ("huffman", "escape"), ("huffman", "reference"), ("ans", None)])
@pytest.mark.parametrize("M,K", [(1021, 4096), (302, 12288), (2045, 5120), (262, 18944), (150, 28672), (9001, 1536)])
@pytest.mark.parametrize("sigma", [0.35, 0.8, 2.5])
def test_rows_of_different_scale(algo, tables, M, K, sigma):
    from bf16_huffman_infer_b200 import ANSWeight, CompressedLinear, HuffmanWeight, set_huffman_tables
    gen = torch.Generator().manual_seed(M)
    W = (make_weight(M, K, 1).float() * torch.exp(sigma * torch.randn(M, 1, generator=gen))).bfloat16()
    previous = set_huffman_tables(tables or "limit6")
    try:
        weight = (ANSWeight if algo == "ans" else HuffmanWeight).compress(W.to(DEV), to_cpu=False)
    finally:
        set_huffman_tables(previous)
    assert torch.equal(weight.get_weight().cpu(), W)
    layer = CompressedLinear(weight, None)
    for rows in (1, 2, 4, 8, 16, 20):
        x = make_input(rows, K, rows)
        with torch.no_grad():
            y = layer(x.to(DEV)) if rows <= 8 else weight._forward(x.to(DEV), None)
        if rows > 8 and y.numel() == 0:
            continue                                           # left to the dense matrix
        y = y.float().cpu()
        ref = x.double() @ W.double().T
        for part in (slice(0, M // 2), slice(M // 2, M)):          # scaled row by row, so that small rows count as much
            scale = ref[:, part].abs().amax(0, keepdim=True).clamp(min=1e-30)
            assert rel_err((y[:, part] / scale).numpy(), (ref[:, part] / scale).numpy()) <= 1e-2, rows
