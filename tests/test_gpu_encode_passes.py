"""The one pass over a dense weight (sign/mantissa plane, exponent counts) and the scan of record sizes, on the device,
against the CPU oracle."""
import os
import sys

import numpy as np
import pytest
import torch

from _util import ROOT, bits_of, make_weight, tables_for

sys.path.insert(0, os.path.join(ROOT, "oracle"))
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,K,S", [(1, 128, 1), (3, 384, 3), (8193, 256, 2), (4096, 640, 1), (37, 12288, 3)])
def test_split_pass_and_record_offsets(M, K, S):
    """The one pass over a weight (plane and counts, in slabs of rows) and the device scan, against the oracle's layout."""
    from bf16_huffman_infer_b200 import ops
    W = make_weight(M, K, 3)
    Wb = bits_of(W)
    tabs = tables_for("huffman", oracle.histogram(Wb))
    rem, exp, offsets, L = oracle.compress(Wb, "huffman", tabs, split_k=S)
    Wd = W.to(DEV)
    plane = torch.empty(S, M, K // S, dtype=torch.uint8, device=DEV)
    counts = torch.zeros(256, dtype=torch.int64, device=DEV)
    cut = (M + 1) // 2
    for lo, hi in ((0, cut), (cut, M)):
        if hi > lo:
            ops.split_histogram(Wd[lo:hi], S, lo, plane, counts)
    assert (plane.cpu().numpy() == rem).all()
    assert (counts.cpu().numpy() == oracle.histogram(Wb)).all()
    rows = torch.from_numpy(np.ascontiguousarray(L).astype(np.int32)).view(S, M).to(DEV)
    off, total = torch.empty_like(rows), torch.empty(1, dtype=torch.int64, device=DEV)
    ops.record_offsets(rows, 4096, off, total)
    assert (off.cpu().numpy() == offsets).all() and total.item() == exp.size
