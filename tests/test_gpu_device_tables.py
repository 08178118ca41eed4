"""Code tables made on the device from a layer's histogram, against the host's builders (which the golden vectors pin)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _histograms(most: int):
    """Up to ``most`` symbols: one, two, as many as there may be and one more; equal counts, ties, geometric and random ones."""
    rng = np.random.default_rng(most)
    for n in sorted({1, 2, 3, 5, 17, most // 2 + 1, most - 1, most, most + 1}):
        if not 1 <= n <= 256:
            continue
        symbols = [np.arange(n), np.sort(rng.choice(256, n, replace=False)), np.arange(256 - n, 256)]
        counts = [np.full(n, 7), np.arange(1, n + 1) // 2 + 1, np.maximum(1, (2.0 ** 36 * 0.5 ** np.arange(n)).astype(np.int64)),
                  rng.integers(1, 10, n), rng.integers(1, 2 ** 30, n), np.where(np.arange(n) == n // 2, 2 ** 37, 1)]
        for i, c in enumerate(counts):
            hist = np.zeros(256, dtype=np.int64)
            hist[symbols[i % 3]] = c
            yield n, hist


@pytest.mark.parametrize("limit", [1, 3, 6, 8])
def test_limited_codes(limit):
    from bf16_huffman_infer_b200 import ops
    from bf16_huffman_infer_b200.huffman import LUTHuffmanEncoder
    for n, hist in _histograms(1 << limit):
        t = [torch.full((256,), 99, dtype=torch.uint8, device=DEV) for _ in range(5)]
        values, status = torch.full((256,), -1, dtype=torch.int32, device=DEV), torch.full((1,), -1, dtype=torch.int64, device=DEV)
        ops.huffman_limit_tables(torch.from_numpy(hist).to(DEV), limit, *t, values, status)
        assert status.item() == (n > 1 << limit)
        if n > 1 << limit:
            assert not any(x.any() for x in (*t, values))                # nothing unwritten for the pass that follows
            continue
        codec = LUTHuffmanEncoder()
        codec.build_lut(hist, method=f"limit{limit}")
        for got, want in zip(t, (codec.LUT1, codec.LUT2, codec.LUT3, codec.LUT4, codec.code_lengths)):
            assert (got.cpu().numpy() == want).all(), (n, hist)
        assert (values.cpu().numpy().view(np.uint32) == codec.code_values).all(), (n, hist)


@pytest.mark.parametrize("bits", [8, 10, 12])
def test_rans_models(bits):
    from bf16_huffman_infer_b200 import ANSWeight, ops
    from bf16_huffman_infer_b200.ans import RANSEncoder
    for n, hist in _histograms(256):
        freq, cum = (torch.full((256,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
        lut, status = torch.full((1 << bits,), -1, dtype=torch.int32, device=DEV), torch.full((1,), -1, dtype=torch.int64, device=DEV)
        ops.ans_tables(torch.from_numpy(hist).to(DEV), freq, cum, lut, status)
        codec = RANSEncoder(hist.tolist(), precision=bits)
        wide = max(codec.freq) > 0xFFF
        assert status.item() == wide
        assert freq.tolist() == codec.freq and cum.tolist() == codec.cum, (n, hist)
        if not wide:
            assert torch.equal(lut.cpu(), ANSWeight.get_lut_kwargs(codec)["LUT"])


@pytest.mark.parametrize("home", ["cpu", DEV])
def test_layers_that_the_device_cannot_serve(home):
    """More than 64 exponents under a limit of 6 bits: the escape-byte code, as the host's builder falls back to it; and a
    12-bit model of one exponent is refused as before."""
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight, set_ans_precision
    from bf16_huffman_infer_b200.huffman import LUTHuffmanEncoder
    gen = torch.Generator().manual_seed(0)
    exps = torch.randint(40, 140, (64, 1024), generator=gen)
    W = (exps << 7).to(torch.int16).view(torch.bfloat16).to(home)
    weight = HuffmanWeight.compress(W, to_cpu=home == "cpu")
    codec = LUTHuffmanEncoder()
    codec.build_lut(np.bincount(exps.flatten().numpy(), minlength=256), method="limit6")
    assert (weight.code_lengths.cpu().numpy() == codec.code_lengths).all() and int(weight.code_lengths.max()) > 6
    assert torch.equal(weight.to(DEV).get_weight().cpu(), W.cpu())
    ones = torch.ones(8, 1024, dtype=torch.bfloat16, device=home)
    previous = set_ans_precision(12)
    try:
        with pytest.raises(ValueError):
            ANSWeight.compress(ones, to_cpu=home == "cpu")
    finally:
        set_ans_precision(previous)


@pytest.mark.parametrize("home", ["cpu", DEV])
@pytest.mark.parametrize("algo", ["huffman", "ans"])
def test_weight_classes_with_tables_of_their_own(algo, home):
    """compress() of a derived class takes the tables that its get_lut_kwargs returns."""
    from _util import make_weight
    from bf16_huffman_infer_b200 import ANSWeight, HuffmanWeight
    base = ANSWeight if algo == "ans" else HuffmanWeight
    asked = []

    class Mine(base):
        @classmethod
        def get_lut_kwargs(cls, codec):
            tables = super().get_lut_kwargs(codec)
            if algo == "huffman":
                tables["LUT4"][:] = 9                                    # which codes of at most 8 bits do not reach
            asked.append({k: v.clone() for k, v in tables.items()})
            return tables

    W = make_weight(64, 1024, 3).to(home)
    weight = Mine.compress(W, to_cpu=home == "cpu")
    assert type(weight) is Mine and len(asked) == 1
    for name, table in asked[0].items():
        assert torch.equal(getattr(weight, name).cpu(), table), name
    assert torch.equal(weight.to(DEV).get_weight().cpu(), W.cpu())
    for name, table in base.compress(W, to_cpu=False).kwargs().items():
        if name != "LUT4":
            assert torch.equal(getattr(weight, name), table), name
