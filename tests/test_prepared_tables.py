"""The folded tables of a Huffman weight follow the tables they were folded from, whatever memory those lie in."""
import copy
import io

import pytest
import torch

from _util import make_weight

TABLES = ("LUT1", "LUT2", "LUT3", "LUT4", "code_lengths")


def _weight(value: int):
    from bf16_huffman_infer_b200 import HuffmanWeight
    return HuffmanWeight(torch.zeros(1, 1, 128, dtype=torch.uint8), torch.zeros(64, dtype=torch.int32),
                         torch.zeros(1, 1, dtype=torch.int32), *(torch.full((256,), value, dtype=torch.uint8) for _ in TABLES))


@pytest.fixture
def folds(monkeypatch):
    """Stands in for the device fold: the blob's first byte is that of the code lengths."""
    from bf16_huffman_infer_b200 import ops
    monkeypatch.setattr(ops, "huffman_prepare", lambda t1, t2, t3, t4, cl, blob: blob.fill_(int(cl[0])))
    monkeypatch.setattr(ops, "huffman_table_hint", lambda blob, complete: None)


def test_tables_in_reused_memory(folds):
    """A move to the host and back frees the tables and makes new ones, which may lie where the old ones were."""
    w, folded, size = _weight(0), [], 40 << 20       # blocks so large are given back and handed out again at once
    for value in range(6):
        for name in TABLES:
            w._buffers[name] = None
        for name in TABLES:
            w._buffers[name] = torch.full((size,), value, dtype=torch.uint8)
        folded.append(int(w.prepared()[0]))
    assert folded == list(range(6))


def test_tables_written_in_place(folds):
    w = _weight(3)
    assert int(w.prepared()[0]) == 3
    w.load_state_dict(_weight(5).state_dict())
    assert int(w.prepared()[0]) == 5


def test_copies_and_pickles_fold_their_own(folds):
    w = _weight(3)
    w.prepared()
    buffer = io.BytesIO()
    torch.save(w, buffer)
    buffer.seek(0)
    for other in (copy.deepcopy(w), torch.load(buffer, weights_only=False)):
        assert not [name for name in other.__dict__ if name.startswith("_prepared")]
        other.load_state_dict(_weight(7).state_dict())
        assert int(other.prepared()[0]) == 7
    assert int(w.prepared()[0]) == 3


def test_copies_that_share_the_buffers_share_the_fold(folds):
    from bf16_huffman_infer_b200.utils import shallow_copy_model
    model = torch.nn.Sequential(_weight(3), _weight(4))
    model[0].prepared()
    copied = shallow_copy_model(model)
    assert copied[0] is not model[0] and copied[0].LUT1 is model[0].LUT1
    assert copied[0].prepared() is model[0].prepared()
    assert "_prepared" not in vars(copied[1]) and int(copied[1].prepared()[0]) == 4


@pytest.mark.gpu
def test_move_load_move():
    from bf16_huffman_infer_b200 import HuffmanWeight, set_huffman_tables
    W = make_weight(64, 384, 0)
    weights = []
    for method in ("limit6", "escape", "reference"):
        previous = set_huffman_tables(method)
        weights.append(HuffmanWeight.compress(W))
        set_huffman_tables(previous)
    w = copy.deepcopy(weights[0]).cuda()
    for other in weights + weights[::-1]:
        w = w.cpu()
        for name, value in other.state_dict().items():
            if w._buffers[name].shape == value.shape:
                w._buffers[name].copy_(value)
            else:
                w._buffers[name] = value.clone()
        w = w.cuda()
        assert torch.equal(w.get_weight().cpu(), W)
