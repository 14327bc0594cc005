"""Partial tiles of batches above 128 rows where memory is short (host only: the allocator is a fake)."""
import pytest

torch = pytest.importorskip("torch")

from georefine_b200 import resident

ROW = 148 * 512      # one batch row of every slot


def _weight(sizes):
    w = object.__new__(resident.ResidentWeight)
    w.device, w.wide_scratch_sizes = torch.device("cpu"), sizes
    w.wide_scratch_bytes = sizes[0] if sizes else 0
    return w


@pytest.mark.parametrize("left,rows", [(384, 384), (383, 256), (256, 256), (255, 192), (192, 192), (191, 0), (0, 0)])
def test_narrower_passes_before_none(monkeypatch, left, rows):
    asked, empty = [], torch.empty

    def short(size, **kw):
        asked.append(size)
        if size > left * ROW:
            raise torch.cuda.OutOfMemoryError("no memory left")
        return empty(size, **kw)

    monkeypatch.setattr(torch, "empty", short)
    block = _weight([384 * ROW, 256 * ROW, 192 * ROW])._lent_scratch(False)
    assert (0 if block is None else block.numel()) == rows * ROW and asked == sorted(asked, reverse=True)
    assert _weight([])._lent_scratch(False) is None
