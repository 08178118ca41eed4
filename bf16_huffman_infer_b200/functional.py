"""Compressed-weight containers, the ``F.linear`` hook and model surgery.

Public surface and behaviour follow the reference's ``bf16_huffman_infer/functional.py``
(``HuffmanWeight`` :66-242, ``ANSWeight`` :245-310, ``CompressedLinear`` :313-320, ``convert``
:323-375, ``convert_all_linear`` :378-387, ``linear_huffman`` :390-411, ``mv_ans`` / ``linear_ans``
:414-466).  The tensors a weight holds (``rem``, ``exp``, ``offsets`` and the tables) are laid out
exactly as the reference lays them out, byte for byte.

What is different underneath: a layer is encoded by two CUDA passes over the BF16 weight (size
pass, prefix sum of the record sizes, emit pass) instead of expanding every symbol to 32
characters and assembling the format with tensor ops; the per-stream operators the reference
uses for that are still available (``compress_groups``) and produce the same words.
"""
from __future__ import annotations

from typing import Callable, Dict, List, Optional, Sequence, Tuple

import os

import numpy as np
import torch
import torch.nn.functional as F
from torch import Tensor, nn
from torch.autograd import forward_ad
from tqdm import tqdm

from . import ops, transfer
from .ans import RANSEncoder
from .huffman import LUTHuffmanEncoder
from .utils import get_block_size_n, split_bf16

OP_PER_LANE = 1
ANS_PRECISION = 8
SLAB_ROWS = 4096          # rows encoded per slab; 64 padding words follow every slab
FUSED_MAX_ROWS = 8        # up to here: fused decode + GEMV, as the reference
FUSED_MORE_ROWS = 32      # up to here without gradients: the same kernel with more products per decoded word; beyond, or with
                          # gradients: decode, then a library GEMM (as the reference)
# Rows up to which mm_huffman_prepared / mm_ans (at most 128) are used instead: up to 32 the same kernel again, beyond, the
# products that keep their sums in tensor memory.  Off by default: beyond 32 rows those are slower than decode + library GEMM
# (python -m bf16_huffman_infer_b200.examples.linear_bench), but need no dense scratch.  BHI_TENSOR_ROWS=128 turns them on.
TENSOR_MAX_ROWS = int(os.environ.get("BHI_TENSOR_ROWS", "0"))
# Which prefix code HuffmanWeight.compress builds (huffman.py; every choice yields tables of the reference's
# format, readable by any decoder of it, the reference's included):
#   "limit6"    (default) optimal code with no length above 6 bits: the fused kernel decodes it symbol by symbol in
#               tables that hold a copy per lane, free of bank conflicts and of exceptions (fastest; about 4 %
#               larger than "escape" on N(0, s) weights; falls back to "escape" beyond 64 distinct exponents);
#   "escape"    escape-byte code, near-entropy on every histogram (smallest);
#   "reference" the reference's own builder, bit for bit (and so its compressed bytes); on some histograms its
#               repair loop lengthens the frequent codes by 2 bits.
# See set_huffman_tables() and convert_all_linear(huffman_tables=...).
HUFFMAN_TABLES = os.environ.get("BHI_HUFFMAN_TABLES", "limit6")


def set_huffman_tables(method: str) -> str:
    """Choose the table builder used by later ``HuffmanWeight.compress`` calls; returns the previous choice."""
    global HUFFMAN_TABLES
    assert method in ("reference", "escape") or (method.startswith("limit") and method[5:].isdigit()), method
    previous, HUFFMAN_TABLES = HUFFMAN_TABLES, method
    return previous


def set_ans_precision(bits: int) -> int:
    """Probability precision (8..12 bits) of the rANS models built by later ``ANSWeight.compress`` calls; returns the
    previous value.  8 is the reference's constant (``functional.py:16``) and what its kernels read; a finer model
    codes the exponents in fewer words but needs a ``2^bits``-word table per weight, which only this package's kernels
    accept (the record and table-word formats are unchanged)."""
    global ANS_PRECISION
    if not 8 <= int(bits) <= 12:
        raise ValueError("rANS precision must be in [8, 12]")
    previous, ANS_PRECISION = ANS_PRECISION, int(bits)
    return previous


__all__ = [
    "linear_huffman",
    "linear_ans",
    "HuffmanWeight",
    "ANSWeight",
    "CompressedLinear",
    "FusedCompressedLinear",
    "convert_all_linear",
    "convert",
    "fuse_sibling_linears",
    "set_huffman_tables",
    "set_ans_precision",
]

# projections that read the same input inside one block of the usual decoder architectures
SIBLING_GROUPS = (("q_proj", "k_proj", "v_proj"), ("gate_proj", "up_proj"))


def _work_device(a: Tensor) -> torch.device:
    if a.is_cuda:
        return a.device
    if not torch.cuda.is_available():
        raise RuntimeError("bf16_huffman_infer_b200 needs a CUDA device: there is no CPU implementation")
    return torch.device("cuda", torch.cuda.current_device())


def _exp_histogram(a: Tensor) -> Tensor:
    """256 exponent counts of a BF16 tensor, or of the bits of one with 16-bit elements (int64, on the CPU)."""
    a = a.detach().contiguous()
    if a.is_cuda and a.dtype == torch.bfloat16 and a.numel() % 128 == 0 and 0 < a.numel() < 2 ** 38 and a.data_ptr() % 4 == 0:
        counts = torch.zeros(256, dtype=torch.int64, device=a.device)
        ops.split_histogram(a.view(-1, 128), 1, 0, torch.empty(0, dtype=torch.uint8, device=a.device), counts)
        return counts.cpu()
    bits = a.view(torch.int16).flatten()
    exp = ((bits >> 7) & 0xFF).to(torch.int64)
    return torch.bincount(exp, minlength=256).cpu()


def _record_offsets(words_per_row: Tensor) -> Tuple[Tensor, int]:
    """Word offset of every record from the per-record row counts ``[S, M]``.

    Records are stored chunk-major with rows ascending; after every slab of ``SLAB_ROWS`` rows (and
    after the last, partial slab of a chunk) 64 zero words are inserted, because a Huffman
    decoder may look one record row past the end of a record (reference ``functional.py:177``,
    ``:204-231``).
    """
    S, M = words_per_row.shape
    if words_per_row.is_cuda:
        offsets, total = _record_offsets_async(words_per_row)
        return offsets, _checked_total(int(total.item()))
    sizes = words_per_row.to(torch.int64) * 64
    pad = torch.zeros(M, dtype=torch.int64, device=sizes.device)
    pad[SLAB_ROWS - 1::SLAB_ROWS] = 64
    pad[M - 1] = 64
    sizes = (sizes + pad[None, :]).flatten()
    ends = torch.cumsum(sizes, 0)
    total = _checked_total(int(ends[-1].item()))
    return (ends - sizes).to(torch.int32).view(S, M), total


def _record_offsets_async(words_per_row: Tensor, total: Optional[Tensor] = None) -> Tuple[Tensor, Tensor]:
    """Same on the device, without waiting for it: offsets, and the total as an i64 tensor of one value (``total``, if given)."""
    offsets = torch.empty_like(words_per_row)
    if total is None:
        total = torch.empty(1, dtype=torch.int64, device=words_per_row.device)
    ops.record_offsets(words_per_row, SLAB_ROWS, offsets, total)
    return offsets, total


def _checked_total(total: int) -> int:
    if total >= 2 ** 31:
        raise RuntimeError("compressed exponent plane exceeds 2^31 words; split the layer")
    return total


class _Ingested:
    """A dense layer on the device with what its one pass over the weight yields: the sign/mantissa plane and the
    exponent counts.  A weight in host memory is passed over slab by slab while the rest is still on its way."""

    def __init__(self, a: Tensor, split_k: int, to_cpu: bool):
        assert a.dim() == 2 and a.dtype == torch.bfloat16
        assert a.size(1) % split_k == 0 and (a.size(1) // split_k) % 128 == 0, a.shape
        a = a.detach()
        dev = _work_device(a)
        M, K = a.shape
        self.split_k = split_k
        self.host_rem: Optional[Tensor] = None
        self.rem = torch.empty(split_k, M, K // split_k, dtype=torch.uint8, device=dev)
        counts = torch.zeros(256, dtype=torch.int64, device=dev)
        if a.is_cuda:
            self.w = a.contiguous()
            ops.split_histogram(self.w, split_k, 0, self.rem, counts)
        else:
            self.w = torch.empty(M, K, dtype=torch.bfloat16, device=dev)
            if to_cpu:
                self.host_rem = torch.empty(split_k, M, K // split_k, dtype=torch.uint8, device="cpu")

            def arrived(lo: int, hi: int) -> None:
                ops.split_histogram(self.w[lo:hi], split_k, lo, self.rem, counts)
                if to_cpu:
                    # the pages that will take the plane on its way back are faulted in while the link is busy with the
                    # next slab (the faults are half the time of a copy into new memory)
                    self.host_rem[:, lo:hi].zero_()

            transfer.upload_rows(a, self.w, arrived)
        self.counts = counts

    @property
    def histogram(self) -> Tensor:
        return self.counts.cpu()


class _Plan:
    """One coder's measure of a layer: its tables and where every record will lie.  ``result`` (i64 ``[2]``, on the device) gets
    the words of the exponent plane and, from tables that were made on the device, whether they serve the layer."""

    def __init__(self, cls, layer: _Ingested, result: Tensor, on_device: bool = True):
        self.cls, self.layer = cls, layer
        # (a class derived from these may have its own get_lut_kwargs, which the host's way asks)
        made = cls._device_tables(layer.counts, result[1:]) if on_device and cls in (HuffmanWeight, ANSWeight) else None
        self.on_device = made is not None
        if made is None:
            codec = cls._codec_of(layer.histogram)
            made = cls.get_lut_kwargs(codec), cls._encoder_tables(codec, layer.w.device)
        self.luts, self.tables = made                                  # luts: where they were made
        rows = torch.empty(layer.rem.shape[:2], dtype=torch.int32, device=layer.w.device)
        cls._size_pass(layer, self.tables, rows)
        self.offsets, _ = _record_offsets_async(rows, result[:1])

    def finish(self, total: int, to_cpu: bool) -> "HuffmanWeight":
        layer, dev = self.layer, self.layer.w.device
        exp = torch.zeros(_checked_total(total), dtype=torch.int32, device=dev)
        self.cls._emit_pass(layer, self.tables, self.offsets, exp)
        if to_cpu:
            home = _tables_home(self.luts) if self.on_device else lambda: self.luts          # under way before the downloads, which wait for the stream
            rem, exp, offsets = transfer.download(layer.rem, layer.host_rem), transfer.download(exp), transfer.download(self.offsets)
            return self.cls(rem=rem, exp=exp, offsets=offsets, **home())
        luts = self.luts if self.on_device else _tables_to(self.luts, dev)
        weight = self.cls(rem=layer.rem, exp=exp, offsets=self.offsets, **luts)          # while the records are being written
        # the buffers must be complete in memory before a fused kernel with launch overlap reads them
        torch.cuda.current_stream(dev).synchronize()
        return weight


def _tables_to(tables: Dict[str, Tensor], dev: torch.device) -> Dict[str, Tensor]:
    """Small host tensors on the device, each in memory of its own, through one copy."""
    raw = [np.ascontiguousarray(t.numpy()).reshape(-1).view(np.uint8) for t in tables.values()]
    packed = torch.from_numpy(np.concatenate(raw)).to(dev)
    out, at = {}, 0
    for (name, t), r in zip(tables.items(), raw):
        out[name] = packed[at:at + r.size].view(t.dtype).view(t.shape).clone()
        at += r.size
    return out


def _tables_home(tables: Dict[str, Tensor]) -> Callable[[], Dict[str, Tensor]]:
    """The way back: the copy is enqueued here, and the tables are taken from it once the stream has been waited for."""
    packed = torch.cat([t.view(torch.uint8) for t in tables.values()])
    here = torch.empty(packed.shape, dtype=torch.uint8, device="cpu", pin_memory=True)
    here.copy_(packed, non_blocking=True)

    def taken() -> Dict[str, Tensor]:
        parts = here.split([t.numel() * t.element_size() for t in tables.values()])
        return {name: part.clone().view(t.dtype) for (name, t), part in zip(tables.items(), parts)}

    return taken


def _compress(a: Tensor, split_k: int, coders: Sequence[type], to_cpu: bool) -> "HuffmanWeight":
    """``a`` by the coder that stores it in the fewest bytes (the first of those that tie).  The sizes are known after
    the size pass, so only the coder that is kept writes its records."""
    layer = _Ingested(a, split_k, to_cpu)
    results = torch.zeros(len(coders), 2, dtype=torch.int64, device=layer.w.device)
    plans: List[_Plan] = [_Plan(c, layer, r) for c, r in zip(coders, results)]
    totals, unserved = zip(*results.tolist())
    if any(unserved):
        plans = [_Plan(p.cls, layer, r, on_device=False) if bad else p for p, r, bad in zip(plans, results, unserved)]
        totals, _ = zip(*results.tolist())
    for t in totals:
        _checked_total(t)
    sizes = [4 * t + sum(v.nelement() * v.element_size() for v in p.luts.values()) for p, t in zip(plans, totals)]
    best = min(range(len(plans)), key=sizes.__getitem__)
    return plans[best].finish(totals[best], to_cpu)


def mv_huffman(
    A_rem: Tensor, A_exp: Tensor, X: Tensor, offsets: Tensor,
    LUT1: Tensor, LUT2: Tensor, LUT3: Tensor, LUT4: Tensor, code_lengths: Tensor,
) -> Tensor:
    """``X @ W.T`` for at most 8 rows of ``X`` from the Huffman-coded ``W`` (reference ``functional.py:28-63``)."""
    if A_rem.dim() == 2:
        A_rem = A_rem[None, :, :]
    if offsets.dim() == 1:
        offsets = offsets[None, :]
    split_k, M, N = A_rem.shape
    X = X.view(-1, split_k, N)
    assert N % 128 == 0
    assert X.dtype == torch.bfloat16
    assert A_rem.device.type == A_exp.device.type == X.device.type == "cuda"
    assert A_rem.device == A_exp.device == X.device
    Y = torch.empty((X.size(0), M), dtype=torch.bfloat16, device=A_rem.device)
    ops.gemv_bf16_huffman(
        A_rem.contiguous(), A_exp.contiguous(), X.contiguous(), Y, offsets.contiguous(),
        LUT1.contiguous(), LUT2.contiguous(), LUT3.contiguous(), LUT4.contiguous(), code_lengths.contiguous(),
    )
    return Y


def mv_huffman_prepared(A_rem: Tensor, A_exp: Tensor, X: Tensor, offsets: Tensor, prepared: Tensor) -> Tensor:
    """:func:`mv_huffman` with the tables already folded (see :meth:`HuffmanWeight.prepared`)."""
    if A_rem.dim() == 2:
        A_rem = A_rem[None, :, :]
    split_k, M, N = A_rem.shape
    X = X.view(-1, split_k, N)
    assert N % 128 == 0
    assert X.dtype == torch.bfloat16
    assert A_rem.device == A_exp.device == X.device and A_rem.device.type == "cuda"
    Y = torch.empty((X.size(0), M), dtype=torch.bfloat16, device=A_rem.device)
    ops.gemv_bf16_huffman_prepared(A_rem.contiguous(), A_exp.contiguous(), X.contiguous(), Y, offsets.contiguous(), prepared)
    return Y


def mv_ans(A_rem: Tensor, A_exp: Tensor, X: Tensor, offsets: Tensor, LUT: Tensor) -> Tensor:
    """``X @ W.T`` for at most 8 rows of ``X`` from the rANS-coded ``W`` (reference ``functional.py:414-444``)."""
    if A_rem.dim() == 2:
        A_rem = A_rem[None, :, :]
    if offsets.dim() == 1:
        offsets = offsets[None, :]
    split_k, M, N = A_rem.shape
    X = X.view(-1, split_k, N)
    assert N % 128 == 0
    assert X.dtype == torch.bfloat16
    assert A_rem.device.type == A_exp.device.type == X.device.type == "cuda"
    assert A_rem.device == A_exp.device == X.device
    Y = torch.empty((X.size(0), M), dtype=torch.bfloat16, device=A_rem.device)
    ops.gemv_bf16_ans(A_rem.contiguous(), A_exp.contiguous(), X.contiguous(), Y, offsets.contiguous(), LUT.contiguous())
    return Y


def mm_huffman_prepared(A_rem: Tensor, A_exp: Tensor, X: Tensor, offsets: Tensor, prepared: Tensor) -> Tensor:
    """``X @ W.T`` for at most 128 rows of ``X`` from the Huffman-coded ``W``: rows of ``W`` are decoded
    into shared memory and multiplied there on the tensor cores.  Stands in for the reference's
    ``huffman_decode`` + ``F.linear`` pair (``functional.py:405-407``) in that range."""
    if A_rem.dim() == 2:
        A_rem = A_rem[None, :, :]
    split_k, M, N = A_rem.shape
    X = X.view(-1, split_k, N)
    assert N % 128 == 0
    assert X.dtype == torch.bfloat16
    assert A_rem.device == A_exp.device == X.device and A_rem.device.type == "cuda"
    Y = torch.empty((X.size(0), M), dtype=torch.bfloat16, device=A_rem.device)
    ops.linear_bf16_huffman_prepared(A_rem.contiguous(), A_exp.contiguous(), X.contiguous(), Y, offsets.contiguous(), prepared)
    return Y


def mm_ans(A_rem: Tensor, A_exp: Tensor, X: Tensor, offsets: Tensor, LUT: Tensor) -> Tensor:
    """Same for the rANS-coded ``W`` (stands in for ``ans_decode`` + ``F.linear``, reference
    ``functional.py:476-478``)."""
    if A_rem.dim() == 2:
        A_rem = A_rem[None, :, :]
    split_k, M, N = A_rem.shape
    X = X.view(-1, split_k, N)
    assert N % 128 == 0
    assert X.dtype == torch.bfloat16
    assert A_rem.device == A_exp.device == X.device and A_rem.device.type == "cuda"
    Y = torch.empty((X.size(0), M), dtype=torch.bfloat16, device=A_rem.device)
    ops.linear_bf16_ans(A_rem.contiguous(), A_exp.contiguous(), X.contiguous(), Y, offsets.contiguous(), LUT.contiguous())
    return Y


class HuffmanWeight(nn.Module):
    """A ``[M, K]`` BF16 weight with Huffman-coded exponents.

    Buffers: ``rem`` u8 ``[S, M, K/S]``, ``exp`` i32 ``[words]``, ``offsets`` i32 ``[S, M]``, ``LUT1..LUT4``
    and ``code_lengths`` u8 ``[256]``.  Passing an instance as the weight of ``F.linear`` dispatches to
    :func:`linear_huffman`.
    """

    algo = "huffman"

    def __init__(self, rem: Tensor, exp: Tensor, offsets: Tensor,
                 LUT1: Tensor, LUT2: Tensor, LUT3: Tensor, LUT4: Tensor, code_lengths: Tensor):
        super().__init__()
        self.rem = nn.Buffer(rem)
        self.exp = nn.Buffer(exp)
        self.offsets = nn.Buffer(offsets)
        self.LUT1 = nn.Buffer(LUT1)
        self.LUT2 = nn.Buffer(LUT2)
        self.LUT3 = nn.Buffer(LUT3)
        self.LUT4 = nn.Buffer(LUT4)
        self.code_lengths = nn.Buffer(code_lengths)

    # -- container protocol ---------------------------------------------------------------
    def kwargs(self) -> Dict[str, Tensor]:
        return dict(self.named_buffers())

    @property
    def shape(self) -> Tuple[int, int]:
        s, m, n = self.rem.shape
        return (m, s * n)

    def nbytes(self) -> int:
        return sum(b.nelement() * b.element_size() for b in self.buffers())

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        if func is not F.linear:
            return NotImplemented
        return linear_huffman(*args, **(kwargs or {}))

    def prepared(self) -> Tensor:
        """The decode tables folded for the fused kernels (built on first use on each device, so the
        first call has to happen outside CUDA-graph capture; warm-up iterations take care of that).
        Not a buffer: it is derived data and stays out of ``state_dict`` and size accounting."""
        d = self.__dict__
        b = d["_buffers"]
        t1, t2, t3, t4, cl = b["LUT1"], b["LUT2"], b["LUT3"], b["LUT4"], b["code_lengths"]
        # in-place loads (load_state_dict) bump the version; a tensor whose data was replaced has another address, because
        # the memory of the tables that were folded is held as long as the blob is
        src = (t1.data_ptr(), t2.data_ptr(), t3.data_ptr(), t4.data_ptr(), cl.data_ptr(),
               t1._version, t2._version, t3._version, t4._version, cl._version)
        if d.get("_prepared_src") != src:
            blob = torch.empty(ops.PREPARED_BYTES, dtype=torch.uint8, device=self.rem.device)
            ops.huffman_prepare(t1, t2, t3, t4, cl, blob)
            # codes of at most 6 bits go through the tables of single symbols
            ops.huffman_table_hint(blob, int(cl.max().item()) <= 6)
            d["_prepared"] = blob
            d["_prepared_tables"] = tuple(t.detach() for t in (t1, t2, t3, t4, cl))
            d["_prepared_src"] = src
        return d["_prepared"]

    derived = ("_prepared_src", "_prepared", "_prepared_tables")        # what prepared() keeps

    @classmethod
    def _drop_prepared(cls, state: Dict) -> Dict:
        for name in cls.derived:
            state.pop(name, None)
        return state

    def _apply(self, *args, **kwargs):
        super()._apply(*args, **kwargs)
        blob = self.__dict__.get("_prepared")
        if blob is not None and blob.device != self.rem.device:
            self._drop_prepared(self.__dict__)
        return self

    def __getstate__(self):
        """Copies and pickles fold their own tables (shallow_copy_model's, which share the buffers, share the fold too)."""
        return self._drop_prepared(self.__dict__.copy())

    def _plain(self) -> bool:
        """The buffers are as the operators take them (``compress`` makes no others)."""
        b = self.__dict__["_buffers"]
        rem, exp, off = b["rem"], b["exp"], b["offsets"]
        return rem.dim() == 3 and off.dim() == 2 and rem.is_contiguous() and exp.is_contiguous() and off.is_contiguous()

    def _forward(self, x: Tensor, bias: Optional[Tensor]) -> Tensor:
        b = self.__dict__["_buffers"]
        return ops.forward_huffman(x, b["rem"], b["exp"], b["offsets"], self.prepared(), bias)

    def _mv(self, x: Tensor) -> Tensor:
        return mv_huffman_prepared(self.rem, self.exp, x, self.offsets, self.prepared())

    def _mm(self, x: Tensor) -> Tensor:
        return mm_huffman_prepared(self.rem, self.exp, x, self.offsets, self.prepared())

    def get_weight(self) -> Tensor:
        """Dense BF16 ``[M, K]`` (reference ``functional.py:99-108``)."""
        b = self._buffers
        assert b["rem"].is_cuda
        return ops.dense_huffman(b["rem"], b["exp"], b["offsets"], self.prepared())

    # -- encoding -----------------------------------------------------------------------------
    @classmethod
    def get_codec(cls, a: Tensor) -> LUTHuffmanEncoder:
        """Code tables from the exponent histogram of ``a`` (reference ``functional.py:110-117``)."""
        return cls._codec_of(_exp_histogram(a.to(_work_device(a))))

    @classmethod
    def _codec_of(cls, histogram: Tensor) -> LUTHuffmanEncoder:
        codec = LUTHuffmanEncoder()
        codec.build_lut(histogram, method=HUFFMAN_TABLES)
        return codec

    @classmethod
    def get_lut_kwargs(cls, codec: LUTHuffmanEncoder) -> Dict[str, Tensor]:
        return {
            "LUT1": torch.from_numpy(codec.LUT1.copy()),
            "LUT2": torch.from_numpy(codec.LUT2.copy()),
            "LUT3": torch.from_numpy(codec.LUT3.copy()),
            "LUT4": torch.from_numpy(codec.LUT4.copy()),
            "code_lengths": torch.from_numpy(codec.code_lengths.copy()),
        }

    @classmethod
    def compress_groups(cls, x: Tensor, codec: LUTHuffmanEncoder) -> Tuple[Tensor, Tensor]:
        """Per-stream operator path: ``x`` u8 ``[rows, 64, n]`` -> (words i32 ``[rows*64, n]``, rows' word counts).

        Same result as reference ``functional.py:129-159`` (character expansion by the
        ``huffman_encode`` operator, then LSB-first packing), kept for operator compatibility and
        as a cross-check of :meth:`compress_split_n`.
        """
        dev = x.device
        rows, groups, n = x.shape
        flat = x.reshape(rows * groups, n).contiguous()
        chars = torch.full((rows * groups, n * 32), ord("0"), dtype=torch.uint8, device=dev)
        bits = torch.zeros(rows * groups, dtype=torch.int32, device=dev)
        table = torch.zeros(256, 32, dtype=torch.uint8)
        for sym, code in codec.huffman_codes.items():
            path = code[::-1]                      # stored reversed; the stream wants root first
            table[sym, :len(path)] = torch.tensor([ord(c) for c in path], dtype=torch.uint8)
        ops.huffman_encode(flat, table.to(dev), chars, bits)
        nbytes = (bits + 7) // 8
        row_words = (nbytes.view(rows, groups).amax(dim=1) + 3) // 4
        weights = (1 << torch.arange(8, device=dev, dtype=torch.int32))
        packed = ((chars.view(rows * groups, -1, 8).to(torch.int32) - ord("0")) * weights).sum(-1).to(torch.uint8)
        return packed.view(torch.int32), row_words.to(torch.int32)

    @classmethod
    def _device_tables(cls, counts: Tensor, status: Tensor) -> Optional[Tuple[Dict[str, Tensor], Dict[str, Tensor]]]:
        """The layer's tables and the encoder's, made from the histogram on its device; None where only the host builds them."""
        if not HUFFMAN_TABLES.startswith("limit") or not 1 <= int(HUFFMAN_TABLES[5:]) <= 8:
            return None
        luts = {k: torch.empty(256, dtype=torch.uint8, device=counts.device) for k in ("LUT1", "LUT2", "LUT3", "LUT4", "code_lengths")}
        values = torch.empty(256, dtype=torch.int32, device=counts.device)
        ops.huffman_limit_tables(counts, int(HUFFMAN_TABLES[5:]), *luts.values(), values, status)
        return luts, {"code_values": values, "code_lengths": luts["code_lengths"]}

    @classmethod
    def _encoder_tables(cls, codec, dev) -> Dict[str, Tensor]:
        return _tables_to({"code_values": torch.from_numpy(codec.code_values.view("int32")),
                           "code_lengths": torch.from_numpy(codec.code_lengths)}, dev)

    @classmethod
    def _size_pass(cls, layer: _Ingested, t: Dict[str, Tensor], rows: Tensor) -> None:
        ops.huffman_size_pass(layer.w, layer.split_k, t["code_lengths"], rows)

    @classmethod
    def _emit_pass(cls, layer: _Ingested, t: Dict[str, Tensor], offsets: Tensor, exp: Tensor) -> None:
        ops.huffman_emit_pass(layer.w, layer.split_k, t["code_lengths"], t["code_values"], offsets, layer.rem.new_empty(0), exp)

    @classmethod
    def compress_split_n(cls, a: Tensor, n: int = 2, to_cpu: bool = True):
        """Encode ``a`` with ``n`` K-chunks (reference ``functional.py:195-238``)."""
        return _compress(a, n, (cls,), to_cpu)

    @classmethod
    def compress(cls, a: Tensor, to_cpu: bool = True):
        """Encode with the format's own K-chunk choice (reference ``functional.py:240-242``)."""
        return cls.compress_split_n(a, n=get_block_size_n(a)[0], to_cpu=to_cpu)


class ANSWeight(HuffmanWeight):
    """A ``[M, K]`` BF16 weight with rANS-coded exponents (8-bit probabilities unless :func:`set_ans_precision` says otherwise).

    Buffers: ``rem``, ``exp``, ``offsets`` as for :class:`HuffmanWeight`, and ``LUT`` i32 ``[2^precision]`` holding
    ``sym << 24 | freq << 12 | (slot - cum[sym])`` per slot (reference ``functional.py:245-310``).
    """

    algo = "ans"

    def __init__(self, rem: Tensor, exp: Tensor, offsets: Tensor, LUT: Tensor):
        nn.Module.__init__(self)
        self.rem = nn.Buffer(rem)
        self.exp = nn.Buffer(exp)
        self.offsets = nn.Buffer(offsets)
        self.LUT = nn.Buffer(LUT if isinstance(LUT, Tensor) else torch.as_tensor(LUT))      # as_tensor moves to a default device

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        if func is not F.linear:
            return NotImplemented
        return linear_ans(*args, **(kwargs or {}))

    def _forward(self, x: Tensor, bias: Optional[Tensor]) -> Tensor:
        b = self.__dict__["_buffers"]
        return ops.forward_ans(x, b["rem"], b["exp"], b["offsets"], b["LUT"], bias)

    def _mv(self, x: Tensor) -> Tensor:
        return mv_ans(self.rem, self.exp, x, self.offsets, self.LUT)

    def _mm(self, x: Tensor) -> Tensor:
        return mm_ans(self.rem, self.exp, x, self.offsets, self.LUT)

    def get_weight(self) -> Tensor:
        b = self._buffers
        assert b["rem"].is_cuda
        return ops.dense_ans(b["rem"], b["exp"], b["offsets"], b["LUT"])

    @classmethod
    def get_codec(cls, a: Tensor) -> RANSEncoder:
        return cls._codec_of(_exp_histogram(a.to(_work_device(a))))

    @classmethod
    def _codec_of(cls, histogram: Tensor) -> RANSEncoder:
        return RANSEncoder(histogram.tolist(), precision=ANS_PRECISION)

    @classmethod
    def get_lut_kwargs(cls, codec: RANSEncoder) -> Dict[str, Tensor]:
        if max(codec.freq) > 0xFFF:
            raise ValueError("one exponent value holds the whole 12-bit model: its frequency does not fit the table word")
        freq, cum = np.array(codec.freq), np.array(codec.cum)
        sym = np.repeat(np.arange(256), freq)
        words = (sym << 24) | (freq[sym] << 12) | (np.arange(sym.size) - cum[sym])
        return {"LUT": torch.from_numpy(words.astype(np.uint32).view(np.int32))}

    @classmethod
    def compress_groups(cls, x: Tensor, codec: RANSEncoder) -> Tuple[Tensor, Tensor]:
        """Per-stream operator path (reference ``functional.py:297-310``): words i32 ``[rows*64, 8n]``, rows' word counts."""
        dev = x.device
        rows, groups, n = x.shape
        flat = x.reshape(rows * groups, n).contiguous()
        words = torch.zeros(rows * groups, n * 8, dtype=torch.int32, device=dev)
        counts = torch.zeros(rows * groups, dtype=torch.int32, device=dev)
        freq = torch.tensor(codec.freq, dtype=torch.int32, device=dev)
        cum = torch.tensor(codec.cum, dtype=torch.int32, device=dev)
        ops.ans_encode(flat, freq, cum, words, counts)
        return words, counts.view(rows, groups).amax(dim=1)

    @classmethod
    def _device_tables(cls, counts: Tensor, status: Tensor) -> Optional[Tuple[Dict[str, Tensor], Dict[str, Tensor]]]:
        freq, cum = (torch.empty(256, dtype=torch.int32, device=counts.device) for _ in range(2))
        lut = torch.empty(1 << ANS_PRECISION, dtype=torch.int32, device=counts.device)
        ops.ans_tables(counts, freq, cum, lut, status)
        return {"LUT": lut}, {"freq": freq, "cum": cum}

    @classmethod
    def _encoder_tables(cls, codec, dev) -> Dict[str, Tensor]:
        return _tables_to({"freq": torch.tensor(codec.freq, dtype=torch.int32, device="cpu"),
                           "cum": torch.tensor(codec.cum, dtype=torch.int32, device="cpu")}, dev)

    @classmethod
    def _size_pass(cls, layer: _Ingested, t: Dict[str, Tensor], rows: Tensor) -> None:
        t["stream_words"] = torch.empty(*rows.shape, 64, dtype=torch.uint8, device=rows.device)
        ops.ans_size_pass(layer.w, layer.split_k, t["freq"], t["cum"], rows, t["stream_words"])

    @classmethod
    def _emit_pass(cls, layer: _Ingested, t: Dict[str, Tensor], offsets: Tensor, exp: Tensor) -> None:
        ops.ans_emit_pass(layer.w, layer.split_k, t["freq"], t["cum"], offsets, t["stream_words"], layer.rem.new_empty(0), exp)


class CompressedLinear(nn.Module):
    """``nn.Linear`` replacement whose weight is a :class:`HuffmanWeight` / :class:`ANSWeight` (reference ``functional.py:313-320``)."""

    def __init__(self, weight: HuffmanWeight, bias: Optional[Tensor]) -> None:
        super().__init__()
        self.weight = weight
        self.bias = bias

    @property
    def out_features(self) -> int:
        return self.weight.shape[0]

    @property
    def in_features(self) -> int:
        return self.weight.shape[1]

    def forward(self, input: Tensor) -> Tensor:
        # nn.Module's own attribute lookup and F.linear's dispatch cost more than the checks below; whoever watches or
        # overrides F.linear (a function mode, a tensor subclass, a weight class of its own) still sees the call
        d = self.__dict__
        weight = d["_modules"]["weight"]
        bias = d["_parameters"].get("bias")
        if bias is None:
            bias = self.bias
        if type(input) is Tensor and type(weight) in (HuffmanWeight, ANSWeight) and not torch._C._is_torch_function_mode_enabled():
            return _linear_compressed(input, weight, bias)
        return F.linear(input, weight, bias)


def _linear_compressed(input: Tensor, weight: HuffmanWeight, bias: Optional[Tensor]) -> Tensor:
    assert input.dim() >= 2, input
    rows = input.numel() // max(input.size(-1), 1)
    if rows <= FUSED_MAX_ROWS and weight._plain():
        # one operator call; a bias that needs a derivative, or is not a whole BF16 vector on the layer's device, is added after it
        assert input.is_cuda and input.dtype == torch.bfloat16
        if input.requires_grad:
            input = input.detach()
        if not input.is_contiguous():
            input = input.contiguous()
        if bias is None:
            return weight._forward(input, None)
        if _takes_bias(bias, input) and not (bias.requires_grad and torch.is_grad_enabled()) and not _transformed():
            try:
                return weight._forward(input, bias)
            except RuntimeError:                     # nothing was launched; asked afterwards, the shape costs nothing here
                if _is_row(weight, bias):
                    raise
        output = weight._forward(input.flatten(0, -2), None)
        output += bias[None, :]
        return output.unflatten(0, input.shape[:-1])
    if FUSED_MAX_ROWS < rows <= FUSED_MORE_ROWS and rows > TENSOR_MAX_ROWS and _takes_more_rows(input, weight, bias):
        output = weight._forward(input.contiguous(), bias)
        if output.numel():
            return output
    if rows > max(FUSED_MAX_ROWS, min(TENSOR_MAX_ROWS, 128)):
        return F.linear(input, weight.get_weight(), bias)
    shape = input.shape
    input = input.flatten(0, -2)
    output = weight._mv(input) if rows <= FUSED_MAX_ROWS else weight._mm(input)
    if bias is not None:
        output += bias[None, :]
    return output.unflatten(0, shape[:-1])


def _takes_bias(bias: Tensor, input: Tensor) -> bool:
    """Whether the operators take the bias as it is, its shape aside; others are torch's to add."""
    return bias.dtype == torch.bfloat16 and bias.device == input.device and bias.is_contiguous()


def _is_row(weight: HuffmanWeight, bias: Tensor) -> bool:
    """A value for each output, which the operators want; torch's addition also takes one for all."""
    return bias.shape == weight.__dict__["_buffers"]["rem"].shape[1:2]


def _transformed() -> bool:
    """A tangent, a batch dimension or a gradient of torch.func may ride on a tensor, which the operators do not carry on."""
    return forward_ad._current_level >= 0 or torch._C._functorch.peek_interpreter_stack() is not None


def _takes_more_rows(input: Tensor, weight: HuffmanWeight, bias: Optional[Tensor]) -> bool:
    """Whether 9 to 32 rows can take the fused product, which has no derivatives, knows BF16 only and would bind a trace to
    its row limit."""
    if not (input.is_cuda and input.dtype == torch.bfloat16 and weight._plain()) or torch.is_autocast_enabled():
        return False
    if _transformed() or torch._C._get_tracing_state() is not None:
        return False
    if bias is not None and not (_takes_bias(bias, input) and _is_row(weight, bias)):
        return False
    return not (torch.is_grad_enabled() and (input.requires_grad or (bias is not None and bias.requires_grad)))


def linear_huffman(input: Tensor, weight: HuffmanWeight, bias: Optional[Tensor] = None) -> Tensor:
    """``F.linear`` on a Huffman-coded weight: fused decode+GEMV up to 8 rows (up to 32 without gradients), decode then
    GEMM beyond (reference ``functional.py:390-411``); optionally the fused tensor-core product up to ``TENSOR_MAX_ROWS``."""
    return _linear_compressed(input, weight, bias)


def linear_ans(input: Tensor, weight: ANSWeight, bias: Optional[Tensor] = None) -> Tensor:
    """Same for an rANS-coded weight (reference ``functional.py:447-466``)."""
    return _linear_compressed(input, weight, bias)


def _buffers_size(w: nn.Module) -> int:
    return sum(b.nelement() * b.element_size() for b in w.buffers())


_CODERS = {"huffman": (HuffmanWeight,), "ans": (ANSWeight,), "smallest": (HuffmanWeight, ANSWeight)}


def _compress_for(a: Tensor, algo: str) -> HuffmanWeight:
    """``a`` compressed as ``algo`` says, on the device it is on."""
    assert algo in _CODERS
    return _compress(a, get_block_size_n(a)[0], _CODERS[algo], to_cpu=not a.is_cuda)


def convert(linear: nn.Linear, name, disable_precision_check: bool = True, algo: str = "huffman"):
    """Compress one ``nn.Linear``; returns a :class:`CompressedLinear`, or ``linear`` itself when
    compression does not pay (ratio >= 1) or, if checking is enabled, when the fused output is off
    by 2 % or more on a random input (reference ``functional.py:323-375``).  The module comes back
    on the device ``linear`` was on."""
    home = linear.weight.device
    module = CompressedLinear(weight=_compress_for(linear.weight, algo), bias=linear.bias)

    ori_size = linear.weight.nelement() * linear.weight.element_size()
    ratio = _buffers_size(module.weight) / ori_size

    max_rtol = 0.0
    if not disable_precision_check:
        work = _work_device(linear.weight)
        linear.to(work)
        module.to(work)
        x = torch.randn(1, linear.in_features, dtype=torch.bfloat16, device=work)
        with torch.no_grad():
            y1 = linear(x)
            y2 = module(x)
        max_rtol = ((y2 - y1).abs() / y1.abs().clamp(min=1e-4)).max().item()
        linear.to(home)
        module.to(home)

    fallback = False
    if ratio >= 1:
        print(f"\nWarning! {name} ratio = {ratio:.2%}")
        fallback = True
    if not disable_precision_check and max_rtol >= 0.02:
        print(f"\nWarning! {name} output mismatch: max rtol = {max_rtol:.2f}")
        fallback = True
    if fallback:
        print("Fallback to regular nn.Linear")
        return linear
    if home.type == "cuda" and module.weight.algo == "huffman":
        module.weight.prepared()              # so that a layer converted on its device can be captured without a first call
    return module


class FusedCompressedLinear(nn.Module):
    """Several ``nn.Linear`` layers that read the same input, stored as ONE compressed weight (their
    rows concatenated) and computed by ONE fused launch.

    A 1024-row projection cannot fill a B200 on its own (7 rows per SM); stacking q/k/v (or
    gate/up) gives the kernel enough rows and saves the fixed cost of the extra launches.  The
    reference attacks the same problem with side streams (``cudastream_utils.py:7-47``).  Each
    original module is replaced by a :class:`_FusedSlice`; the first one in call order computes the
    stacked output, the others return their slice of it.
    """

    def __init__(self, weight: HuffmanWeight, bias: Optional[Tensor], splits):
        super().__init__()
        self.weight = weight
        self.bias = bias
        self.splits = list(splits)            # [(start, stop), ...] in stacking order
        self.sharded: Optional[nn.Module] = None   # set by tensor_parallel.shard_model_linears: computes the full output
        self._last_in = None
        self._last_out = None
        self._readers_left = 0                      # slices that have not picked up the last output yet

    def run(self, input: Tensor) -> Tensor:
        out = self.sharded(input) if self.sharded is not None else F.linear(input, self.weight, self.bias)
        self._last_in = (input.data_ptr(), input._version, tuple(input.shape))
        self._last_out = out
        self._readers_left = len(self.splits) - 1
        return out

    def cached(self, input: Tensor) -> Tensor:
        """The leader's output for this very input.  It is kept only until every other slice has read it once:
        a later tensor that happens to get the same address (and version 0) must not match a stale entry."""
        key = (input.data_ptr(), input._version, tuple(input.shape))
        if self._last_out is None or self._last_in != key:
            out = self.run(input)
            self._readers_left -= 1
        else:
            out = self._last_out
            self._readers_left -= 1
        if self._readers_left <= 0:
            self._last_in = self._last_out = None
        return out


class _FusedSlice(nn.Module):
    """Stands where one of the stacked layers was; ``leader`` recomputes, the others reuse."""

    def __init__(self, owner: FusedCompressedLinear, index: int, leader: bool):
        super().__init__()
        self.__dict__["_owner"] = owner       # not a submodule: the owner is registered once, on the leader
        if leader:
            self.fused = owner
        self.index = index
        self.leader = leader

    @property
    def out_features(self) -> int:
        a, b = self._owner.splits[self.index]
        return b - a

    def forward(self, input: Tensor) -> Tensor:
        owner = self._owner
        out = owner.run(input) if self.leader else owner.cached(input)
        a, b = owner.splits[self.index]
        return out[..., a:b]


def fuse_sibling_linears(model: nn.Module, groups=SIBLING_GROUPS, algo: str = "huffman", progress: bool = False) -> int:
    """Stack and compress sibling ``nn.Linear`` layers (same parent, same input width, all with or all
    without bias) named as in ``groups``.  Call before :func:`convert_all_linear`, which then handles
    the remaining layers.  Returns the number of groups fused."""
    todo = []
    for pname, parent in model.named_modules():
        for names in groups:
            mods = [getattr(parent, n, None) for n in names]
            if not all(isinstance(m, nn.Linear) for m in mods):
                continue
            if len({m.in_features for m in mods}) != 1 or len({m.bias is None for m in mods}) != 1:
                continue
            todo.append((pname, parent, names, mods))
    for pname, parent, names, mods in tqdm(todo, disable=not progress):
        home = mods[0].weight.device
        stacked = torch.cat([m.weight.detach() for m in mods], dim=0)
        bias = None if mods[0].bias is None else nn.Parameter(torch.cat([m.bias.detach() for m in mods]), requires_grad=False)
        weight = _compress_for(stacked, algo)
        if _buffers_size(weight) >= stacked.nelement() * stacked.element_size():
            continue                                      # does not pay: leave the layers alone
        bounds, at = [], 0
        for m in mods:
            bounds.append((at, at + m.out_features))
            at += m.out_features
        owner = FusedCompressedLinear(weight, bias, bounds).to(home)
        for i, n in enumerate(names):
            setattr(parent, n, _FusedSlice(owner, i, leader=(i == 0)))
    return len(todo)


def convert_all_linear(model: nn.Module, min_out_features: int = 4096, progress: bool = True,
                       algo: str = "huffman", fuse_siblings: bool = False, huffman_tables: Optional[str] = None) -> None:
    """Replace, in place, every ``nn.Linear`` with at least ``min_out_features`` outputs
    (reference ``functional.py:378-387``).  Not in the reference: ``fuse_siblings=True`` first stacks
    q/k/v and gate/up projections into single compressed weights (:class:`FusedCompressedLinear`);
    ``huffman_tables`` picks the table builder for this call (:func:`set_huffman_tables`)."""
    previous = set_huffman_tables(huffman_tables) if huffman_tables is not None else None
    try:
        if fuse_siblings:
            fuse_sibling_linears(model, algo=algo, progress=progress)
        targets = [name for name, mod in model.named_modules()
                   if isinstance(mod, nn.Linear) and mod.out_features >= min_out_features]
        for name in tqdm(targets, disable=not progress):
            model.set_submodule(name, convert(model.get_submodule(name), name, algo=algo))
    finally:
        if previous is not None:
            set_huffman_tables(previous)
