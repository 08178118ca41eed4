"""X that passes through its ring, filled by a warpgroup that has given registers back: the ordinary and the row-sharded kernel
(one rank), eight rows, and 9 to 32."""
import pytest
import torch

from _util import Abi, gemv_arguments, make_input, make_weight, rel_err
from test_gpu_exchange import Exchange, _launch, _status

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("algo,tables", [("huffman", "limit6"), ("huffman", "escape"), ("ans", None)])
@pytest.mark.parametrize("M,K", [(300, 12288), (1023, 18944), (5, 28672)])
def test_rows_through_the_ring(algo, tables, M, K):
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight, set_huffman_tables
    abi = Abi()
    _status(abi)                                                          # what earlier calls left
    W = make_weight(M, K, 2).to(DEV)
    previous = set_huffman_tables(tables or "limit6")
    try:
        weight = (HuffmanWeight if algo == "huffman" else ANSWeight).compress(W, to_cpu=False)
    finally:
        set_huffman_tables(previous)
    for rows in (8, 9, 16, 17, 24, 25, 32):
        x = make_input(rows, K, rows).to(DEV)
        y = weight._forward(x, None)
        assert y.shape == (rows, M)                                      # empty: left to the dense matrix, which none of these is
        assert rel_err(y.float().cpu().numpy(), (x.double() @ W.double().T).cpu().numpy()) <= 1e-2, rows
        assert torch.equal(y, weight._forward(x, None))
    w, x = weight.kwargs(), make_input(8, K, 8).to(DEV)
    y = torch.zeros(8, M, dtype=torch.bfloat16, device=DEV)
    counters = torch.zeros(2, 32, dtype=torch.int32, device=DEV)
    launches = torch.zeros(2, dtype=torch.int32, device=DEV)
    ex = Exchange(world=1, rank=0, row_base=0, M_total=M)
    ex.y[0], ex.ready[0], ex.done[0] = y.data_ptr(), counters[0].data_ptr(), counters[1].data_ptr()
    ex.launches = launches.data_ptr()
    for _ in range(2):
        _launch(abi, algo, w, x, ex)
    torch.cuda.synchronize()
    assert _status(abi) == 0 and launches.tolist() == [2, 0]
    assert torch.equal(abi.gemv(algo, w, x, prepared=algo == "huffman"), y)


@pytest.mark.parametrize("algo,tables,M,K,rows,shift", [
    ("huffman", "limit6", 3584, 4096, 17, 0), ("huffman", "limit6", 520, 8576, 24, 0), ("huffman", "limit6", 520, 8576, 25, 1),
    ("ans", None, 520, 16256, 5, 0), ("ans", None, 4096, 12288, 8, 0), ("ans", None, 2368, 4096, 9, 0), ("ans", None, 2372, 4096, 9, 1),
    ("ans", None, 2600, 8576, 16, 0), ("ans", None, 2600, 8576, 9, 1), ("ans", None, 520, 4096, 17, 1),
    ("huffman", "escape", 2960, 12288, 25, 1), ("huffman", "escape", 2964, 12288, 25, 0), ("huffman", "escape", 4143, 12288, 32, 1),
    ("huffman", "escape", 4140, 12288, 32, 0), ("huffman", "escape", 3584, 6144, 32, 1), ("huffman", "escape", 3584, 18944, 32, 0),
    ("huffman", "escape", 3584, 12288, 24, 1),
    ("huffman", "escape", 3630, 9856, 25, 1), ("huffman", "escape", 3630, 7680, 25, 0), ("huffman", "escape", 3630, 6656, 25, 1), ("huffman", "limit6", 3584, 12288, 32, 1),
])
def test_which_launches_shift_registers(algo, tables, M, K, rows, shift):
    """Some forms decode slower with the shift's registers than without them; on either side the results are right."""
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight, set_huffman_tables
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are for 148 SMs")
    W = make_weight(M, K, 4).to(DEV)
    previous = set_huffman_tables(tables or "limit6")
    try:
        weight = (HuffmanWeight if algo == "huffman" else ANSWeight).compress(W, to_cpu=False)
    finally:
        set_huffman_tables(previous)
    x = make_input(rows, K, rows).to(DEV)
    y = weight._forward(x, None)
    assert gemv_arguments(lambda: weight._forward(x, None))[-1] == shift
    assert rel_err(y.float().cpu().numpy(), (x.double() @ W.double().T).cpu().numpy()) <= 1e-2
    assert torch.equal(y, weight._forward(x, None))
