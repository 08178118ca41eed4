"""Calls of a compressed layer that a layer over the dense matrix answers: derivatives other than by backward, batching,
tracing, unusual biases and shapes."""
import pytest
import torch
import torch.autograd.forward_ad as fwad
import torch.nn.functional as F
from torch import nn

from _util import make_input, make_weight

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
M, K = 130, 512


@pytest.fixture(scope="module", params=["huffman", "ans"])
def coded(request):
    """(dense matrix, compressed weight, bias)"""
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight
    W = make_weight(M, K, 0).to(DEV)
    cls = HuffmanWeight if request.param == "huffman" else ANSWeight
    return W, cls.compress(W, to_cpu=False), make_weight(1, M, 1)[0].to(DEV)


def _layer(weight, bias):
    from bf16_huffman_infer_b200 import CompressedLinear
    return CompressedLinear(weight, None if bias is None else nn.Parameter(bias.clone(), requires_grad=False))


def _close(y, want):
    """BF16 roundings of FP32 sums in two orders: each output within one BF16 step (2^-8 of it) and the sums' own error."""
    return bool(((y - want).double().norm() / want.double().norm()) < 2.0 ** -8)


@pytest.mark.parametrize("rows", [9, 12, 32])
def test_forward_mode_nine_to_thirty_two_rows(coded, rows):
    W, weight, bias = coded
    layer = _layer(weight, bias)
    x, t = make_input(rows, K, 1).to(DEV), make_input(rows, K, 2).to(DEV)
    with fwad.dual_level():
        y = fwad.unpack_dual(layer(fwad.make_dual(x, t)))
        assert y.tangent is not None
        assert _close(y.primal, F.linear(x, W, bias)) and _close(y.tangent, F.linear(t, W))
    y, tangent = torch.func.jvp(layer, (x,), (t,))
    assert _close(y, F.linear(x, W, bias)) and _close(tangent, F.linear(t, W))
    assert _close(torch.func.vmap(layer)(torch.stack([x, t])), F.linear(torch.stack([x, t]), W, bias))


def test_trace_of_nine_rows_runs_with_more(coded):
    W, weight, bias = coded
    x = make_input(12, K, 1).to(DEV)
    more = make_input(40, K, 2).to(DEV)
    with torch.no_grad():
        traced = torch.jit.trace(_layer(weight, bias), (x,), check_trace=False)
        assert _close(traced(x), F.linear(x, W, bias)) and _close(traced(more), F.linear(more, W, bias))


@pytest.mark.parametrize("rows", [4, 12, 40])
def test_biases_of_other_shapes(coded, rows):
    """What an in-place addition (up to 8 rows) or F.linear (more) takes is taken, and what they refuse is refused."""
    W, weight, bias = coded
    x = make_input(rows, K, 1).to(DEV)
    plain = F.linear(x, W)
    takes = [bias, bias.float(), bias[:1], bias[:1].expand(M)] if rows <= 8 else [bias, bias[:1], bias[0], bias.expand(rows, M)]
    refuses = [bias[0], bias[None], bias[1:], bias[None].float(), bias.expand(rows, M), bias.cpu()] if rows <= 8 else \
        [bias[1:], bias.float(), bias.cpu()]
    with torch.no_grad():
        for b in takes:
            layer = _layer(weight, None)
            layer.bias = b
            assert _close(layer(x), plain + b), (b.shape, b.dtype)
        for b in refuses:
            layer = _layer(weight, None)
            layer.bias = b
            with pytest.raises((RuntimeError, IndexError)):
                layer(x)


def test_tangent_of_the_bias(coded):
    W, weight, bias = coded
    x, t = make_input(4, K, 1).to(DEV), make_weight(1, M, 2)[0].to(DEV)
    layer = _layer(weight, None)
    with fwad.dual_level():
        layer.bias = fwad.make_dual(bias, t)
        assert torch.equal(fwad.unpack_dual(layer(x)).tangent, t.expand(4, M))


@pytest.mark.parametrize("rows", [4, 12, 40])
def test_overrides_of_linear_see_the_call(coded, rows):
    from torch.overrides import TorchFunctionMode
    W, weight, bias = coded
    layer, x = _layer(weight, bias), make_input(rows, K, 1).to(DEV)
    seen = []

    class Watch(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    class Own(type(weight)):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(func)
            return super().__torch_function__(func, types, args, kwargs)

    with torch.no_grad():
        want = layer(x)
        with Watch():
            assert torch.equal(layer(x), want)
        assert seen.count(F.linear) >= 1
        seen.clear()
        assert torch.equal(_layer(Own(**weight.kwargs()), bias)(x), want)
        assert F.linear in seen


@pytest.mark.parametrize("rows", [4, 12])
def test_many_leading_dimensions(coded, rows):
    W, weight, bias = coded
    x = make_input(rows, K, 1).to(DEV).view(*[1] * 22, rows, K)
    with torch.no_grad():
        y = _layer(weight, bias)(x)
    assert y.shape == x.shape[:-1] + (M,) and _close(y, F.linear(x, W, bias))


@pytest.mark.parametrize("path", [0, 2])
def test_both_automatic_paths_take_more_rows(coded, path):
    from _util import Abi
    W, weight, bias = coded
    abi = Abi()
    previous = abi.set_path(path)
    try:
        x = make_input(12, K, 1).to(DEV)
        y = weight._forward(x, bias)
        assert y.shape == (12, M) and _close(y, F.linear(x, W, bias))
    finally:
        abi.set_path(previous)
