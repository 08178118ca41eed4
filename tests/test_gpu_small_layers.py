"""Layers at the edges of the launch forms for small layers (half of each SM, one or two chunks) and of the product forms (up to
four rows of X, up to eight), against a double-precision product of the decoded weights."""
import ctypes

import pytest
import torch

from _util import Abi, gemv_arguments, make_input, make_weight, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _weight(algo, W, bits=8):
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight, set_ans_precision
    previous = set_ans_precision(bits)
    try:
        return (ANSWeight if algo == "ans" else HuffmanWeight).compress(W.to(DEV), to_cpu=False)
    finally:
        set_ans_precision(previous)


@pytest.mark.parametrize("algo,bits", [("huffman", 8), ("ans", 8), ("ans", 12)])
@pytest.mark.parametrize("M,K", [(1, 1024), (5, 1152), (593, 1024), (1184, 2048), (1185, 2048), (2365, 1024), (2368, 4096), (2372, 1024),
                                 (591, 6144), (1184, 6144), (1185, 6144), (300, 12288)])
def test_edges_of_small_layers(algo, bits, M, K):
    abi, status = Abi(), ctypes.c_int(-1)
    abi.check(abi.lib.bhi_debug_status(ctypes.byref(status)))            # what earlier calls left
    W = make_weight(M, K, M).to(DEV)
    weight = _weight(algo, W, bits)
    bias = make_input(1, M, 3).flatten().to(DEV)
    for rows in (1, 2, 3, 4, 5, 8):
        x = make_input(rows, K, rows).to(DEV)
        ref = (x.double() @ W.double().T).cpu().numpy()
        aside = torch.cat([x.flatten()[:2], x.flatten()])[2:].view(rows, K)          # 4-byte aligned only: X is copied by loads
        for given in (x, aside):
            y = weight._forward(given, None)
            assert rel_err(y.float().cpu().numpy(), ref) <= 1e-2, rows
            assert torch.equal(y, weight._forward(given, None))
        # a bias is added to the rounded product and rounded again, as torch adds it
        assert torch.equal(weight._forward(x, bias), y + bias)
    abi.check(abi.lib.bhi_debug_status(ctypes.byref(status)))
    assert status.value == 0


@pytest.mark.parametrize("algo", ["huffman", "ans"])
@pytest.mark.parametrize("M,K", [(512, 2048), (1024, 4096)])
def test_without_launch_overlap(algo, M, K):
    """Half of each SM is left to the next kernel only where that one may come early; the results are the same either way."""
    from bf16_huffman_infer_b200 import ops
    W = make_weight(M, K, M).to(DEV)
    weight = _weight(algo, W)
    for rows in (1, 2, 8):
        x = make_input(rows, K, rows).to(DEV)
        ref = (x.double() @ W.double().T).cpu().numpy()
        previous = ops.set_launch_overlap(True)
        try:
            beside = weight._forward(x, None)
            if rows == 1:
                assert gemv_arguments(lambda: weight._forward(x, None))[5] == 1
            ops.set_launch_overlap(False)
            alone = weight._forward(x, None)
            assert gemv_arguments(lambda: weight._forward(x, None))[5] == 0
        finally:
            ops.set_launch_overlap(previous)
        for y in (beside, alone):
            assert rel_err(y.float().cpu().numpy(), ref) <= 1e-2


@pytest.mark.parametrize("algo", ["huffman", "ans"])
def test_chains_of_small_layers(algo):
    """Each layer reads what the one before it wrote, while its own tables and records arrive beside that one: eagerly, in a
    graph, and with the launches of another stream in between."""
    from bf16_huffman_infer_b200 import CompressedLinear
    K, depth = 1024, 12
    layers = []
    for i in range(depth):
        layers.append(CompressedLinear(_weight(algo, make_weight(K, K, i, 1.0 / 32).to(DEV)), None))
    x = make_input(2, K, 9).to(DEV)

    def chain():
        out = [x]
        for layer in layers:
            out.append(layer(out[-1]))
        return out

    with torch.no_grad():
        want = chain()
        torch.cuda.synchronize()
        for got, layer, y in zip(want, layers, want[1:]):
            ref = got.double() @ layer.weight.get_weight().double().T
            assert rel_err(y.float().cpu().numpy(), ref.cpu().numpy()) <= 1e-2
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            again = chain()
        again_here = chain()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            replayed = chain()
        for y in replayed[1:]:
            y.zero_()
        for _ in range(5):
            graph.replay()
        torch.cuda.synchronize()
    for a, b, c, d in zip(want, again, again_here, replayed):
        assert torch.equal(a, b) and torch.equal(a, c) and torch.equal(a, d)


@pytest.mark.parametrize("algo", ["huffman", "ans"])
@pytest.mark.parametrize("K,depth", [(1024, 12), (4096, 6)])
def test_chains_of_unaligned_inputs(algo, K, depth):
    """X is what the layer before wrote, 4 bytes past an aligned address, so it comes by plain loads; the bias is a layer's
    output too.  (4096 rows are past the launch form of small layers.)"""
    layers = [_weight(algo, make_weight(K + 2, K, i, K ** -0.5).to(DEV)) for i in range(depth)]
    x = make_input(1, K, 9).to(DEV)

    def chain():
        out = [x]
        for i, w in enumerate(layers):
            y = w._forward(out[-1], out[-1].flatten().new_zeros(K + 2) if i == 0 else last.flatten())
            last = y
            out.append(y.flatten()[2:].view(1, K))
        return out

    want = chain()
    torch.cuda.synchronize()
    bias = torch.zeros(K + 2, dtype=torch.bfloat16, device=DEV)
    for i, w in enumerate(layers):
        assert want[i].data_ptr() % 16 == (4 if i else 0)
        y = w._forward(want[i].clone(), None)[0] + bias
        assert torch.equal(y[2:], want[i + 1][0])
        bias = y
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = chain()
    for _ in range(20):
        for y in replayed[1:]:
            y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(want, replayed))


@pytest.mark.parametrize("sigma", [0.8, 2.5])
@pytest.mark.parametrize("algo", ["huffman", "ans"])
def test_small_layers_of_uneven_rows(algo, sigma):
    """Records too long for the ring of half an SM come quad by quad or from global memory."""
    for M, K in ((700, 4096), (2300, 3584)):
        W = (make_weight(M, K, 1).float() * torch.exp(sigma * torch.randn(M, 1, generator=torch.Generator().manual_seed(M)))).bfloat16().to(DEV)
        weight = _weight(algo, W)
        for rows in (1, 4, 8):
            x = make_input(rows, K, rows).to(DEV)
            ref = x.double() @ W.double().T
            scale = ref.abs().amax(0, keepdim=True).clamp(min=1e-30)               # row by row, so that small rows count as much
            y = weight._forward(x, None).double()
            assert rel_err((y / scale).cpu().numpy(), (ref / scale).cpu().numpy()) <= 1e-2, rows


@pytest.mark.parametrize("algo,bits,M,K,half", [("ans", 8, 2368, 2048, 1), ("ans", 8, 1024, 4096, 1), ("ans", 8, 2372, 2048, 0), ("ans", 8, 1536, 4096, 0),
                                                ("ans", 8, 1024, 6144, 0), ("ans", 8, 600, 5120, 0),
                                                ("ans", 8, 296, 3584, 0), ("ans", 8, 297, 3584, 1), ("ans", 12, 296, 3584, 1), ("ans", 12, 600, 5120, 1),
                                                ("ans", 12, 2368, 2048, 1), ("ans", 12, 1024, 4096, 1), ("ans", 12, 1536, 4096, 0),
                                                ("huffman", 8, 2368, 4096, 1), ("huffman", 8, 2368, 4864, 0)])
def test_which_layers_are_small(algo, bits, M, K, half):
    """The line is drawn by the quads of an SM, for 8-bit rANS by their columns too; on either side the results are right."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are for 148 SMs")
    W = make_weight(M, K, M).to(DEV)
    weight = _weight(algo, W, bits)
    x = make_input(2, K, 5).to(DEV)
    y = weight._forward(x, None)
    assert gemv_arguments(lambda: weight._forward(x, None))[5] == half
    assert rel_err(y.float().cpu().numpy(), (x.double() @ W.double().T).cpu().numpy()) <= 1e-2


@pytest.mark.parametrize("algo", ["huffman", "ans"])
@pytest.mark.parametrize("M,K", [(1, 1152), (9, 1152), (1030, 4096), (5, 6144), (3000, 2176)])
def test_infinities_and_nans(algo, M, K):
    """Products with rows past the batch, absent quads, the other half and, for an odd number of blocks, what lies behind a row are
    discarded: an infinity or a NaN of X shows in its own row only, one of the weight in its own column only."""
    W = make_weight(M, K, 7)
    if M > 4:
        W[2, 7], W[3, K - 1], W[4, 130] = float("inf"), float("nan"), float("-inf")
    W = W.to(DEV)
    weight = _weight(algo, W)
    for rows in (1, 2, 3, 4, 5, 8):
        x = make_input(rows, K, rows).to(DEV)
        clean = weight._forward(x, None)
        odd = [r for r in (0, 1, 3, 7) if r < rows][-2:] if rows > 1 else []
        for i, r in enumerate(odd):
            x[r, 0 if i else K - 1] = float("nan") if i else float("inf")
        y = weight._forward(x, None)
        kept = [r for r in range(rows) if r not in odd]
        assert torch.equal(y[kept].view(torch.int16), clean[kept].view(torch.int16))
        ref = x.double() @ W.double().T
        assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf())
        assert torch.equal(y[y.isinf()].sign().double(), ref[ref.isinf()].sign())
        ok = torch.where(ref.isfinite(), ref, torch.zeros_like(ref))
        got = torch.where(ref.isfinite(), y.double(), torch.zeros_like(ref))
        assert rel_err(got.cpu().numpy(), ok.cpu().numpy()) <= 1e-2
