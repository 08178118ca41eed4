"""Layers with one exponent value: codes of one bit, half of whose windows the folded table does not resolve."""
import pytest
import torch
import torch.nn.functional as F

from _util import make_input, make_weight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _time(call):
    times = []
    for _ in range(6):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for _ in range(4):
            call()
        end.record()
        torch.cuda.synchronize()
        times.append(start.elapsed_time(end))
    return min(times)


@pytest.mark.parametrize("tables", ["limit6", "escape", "reference"])
def test_one_exponent(tables):
    """Decoded from shared memory as any other layer: from global memory, symbol by symbol, it takes several times as long."""
    from bf16_huffman_infer_b200 import CompressedLinear, HuffmanWeight, set_huffman_tables
    M, K = 4096, 4096
    sign = torch.randint(0, 2, (M, K), generator=torch.Generator().manual_seed(0)).bfloat16() * 2 - 1
    previous = set_huffman_tables(tables)
    try:
        for W in (0.5 * sign, torch.zeros(M, K, dtype=torch.bfloat16)):
            weight = HuffmanWeight.compress(W.to(DEV), to_cpu=False)
            assert torch.equal(weight.get_weight().cpu(), W)
            for rows in (1, 8, 16):
                x = make_input(rows, K, rows).to(DEV)
                y = CompressedLinear(weight, None)(x)
                want = F.linear(x.float(), W.to(DEV).float())
                assert ((y - want).norm() / want.norm().clamp(min=1e-9)).item() < 2.0 ** -8
        usual = HuffmanWeight.compress(make_weight(M, K, 1).to(DEV), to_cpu=False)
    finally:
        set_huffman_tables(previous)
    assert _time(weight.get_weight) < 2.5 * _time(usual.get_weight)
