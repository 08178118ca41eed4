"""The fused kernel reads its tables at a fixed place of shared memory and decodes without them where that is not the place;
the status word tells which it was."""
import ctypes

import pytest
import torch

from _util import Abi, make_input, make_weight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("algo,tables", [("huffman", "limit6"), ("huffman", "escape"), ("ans", None)])
@pytest.mark.parametrize("M,K", [(256, 4096), (4096, 4096), (300, 12288)])
def test_tables_lie_where_they_are_read(algo, tables, M, K):
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight, set_huffman_tables
    abi, status = Abi(), ctypes.c_int(-1)
    previous = set_huffman_tables(tables or "limit6")
    try:
        weight = (ANSWeight if algo == "ans" else HuffmanWeight).compress(make_weight(M, K, 0).to(DEV), to_cpu=False)
    finally:
        set_huffman_tables(previous)
    abi.check(abi.lib.bhi_debug_status(ctypes.byref(status)))            # what earlier calls left
    weight.get_weight()
    for rows in (1, 8, 16, 32):
        weight._forward(make_input(rows, K, rows).to(DEV), None)
        abi.check(abi.lib.bhi_debug_status(ctypes.byref(status)))
        assert status.value == 0, rows


@pytest.mark.parametrize("bits", [8, 12, 13, 15])
def test_encoder_of_fine_models(bits):
    """The per-stream rANS encoder against the slow codec, over the precisions that a model can have."""
    from bf16_huffman_infer_b200 import ops
    from bf16_huffman_infer_b200.ans import RANSEncoder
    gen = torch.Generator().manual_seed(bits)
    data = (torch.randn(6, 500, generator=gen) * 3 + 120).round().clamp(0, 255).to(torch.uint8)
    codec = RANSEncoder(torch.bincount(data.flatten().long(), minlength=256).tolist(), precision=bits)
    freq, cum = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (codec.freq, codec.cum))
    words = torch.zeros(6, 500 * 8, dtype=torch.int32, device=DEV)
    counts = torch.zeros(6, dtype=torch.int32, device=DEV)
    ops.ans_encode(data.to(DEV), freq, cum, words, counts)
    for row, stream, n in zip(data.tolist(), words.cpu().tolist(), counts.tolist()):
        blob = codec.compress(row)                                        # words in emission order, then two of the state
        want = [int.from_bytes(blob[i:i + 4], "big") for i in range(0, len(blob), 4)][::-1]
        want = want[1:] if want[0] == 0 else want                        # the state's high word may be empty
        assert [w & 0xFFFFFFFF for w in stream[:n]] == want
