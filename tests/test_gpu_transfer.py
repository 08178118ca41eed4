"""Slab-wise copies between host and device: sizes around a slab, wide rows, strided and pinned sources."""
import pytest
import torch

from bf16_huffman_infer_b200 import transfer

pytestmark = pytest.mark.gpu
SLAB = transfer.SLAB_BYTES


@pytest.mark.parametrize("rows,cols", [(1, 128), (SLAB // 256 - 1, 128), (SLAB // 256 + 1, 128), (5 * SLAB // 7680, 3840), (2, SLAB // 2 + 64)])
def test_round_trip(rows, cols):
    src = torch.randint(-2 ** 15, 2 ** 15, (rows, cols), dtype=torch.int16).view(torch.bfloat16)
    for host in (src, src.pin_memory(), src.t().contiguous().t()):
        dst = torch.empty(rows, cols, dtype=torch.bfloat16, device="cuda:0")
        seen = []
        transfer.upload_rows(host, dst, lambda lo, hi: seen.append((lo, hi)))
        back = transfer.download(dst)
        assert torch.equal(back.view(torch.int16), src.view(torch.int16))
        assert seen[0][0] == 0 and seen[-1][1] == rows and all(a[1] == b[0] for a, b in zip(seen, seen[1:]))
