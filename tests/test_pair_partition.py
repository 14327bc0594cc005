"""The work partition of pairs of workers (4-bit window images): who gets it, what it covers, and that the validator holds an
image to the one its header names."""
import ctypes

import numpy as np
import pytest

from georefine_b200 import _native, resident

# rows x columns, workers -> partition of pairs?  (units = row blocks x chunks)
SHAPES = [((512, 2048), 4, 1), ((512, 2048), 6, 1), ((500, 2040), 6, 1),
          ((512, 2048), 8, 0),      # two whole workers a row block: clusters
          ((512, 2048), 10, 0),     # fewer than eight chunks a worker
          ((512, 2048), 5, 0),      # an odd number of workers
          ((640, 2048), 6, 0)]      # an odd number of row blocks


def _image(orc, shape, workers, layout="window4"):
    words = orc.synthetic_weight_words(*shape, 5)
    image, h = resident.build_image(words, workers, layout=layout)
    return words, image, h


@pytest.mark.parametrize("shape,workers,paired", SHAPES)
def test_partition(orc, shape, workers, paired):
    words, image, h = _image(orc, shape, workers)
    assert h.paired == paired and np.array_equal(resident.decode_image_host(image), words)
    items = (_native.BxrItem * h.items).from_buffer_copy(image[h.items_at:h.items_at + 32 * h.items].tobytes())
    at = np.frombuffer(image[h.worker_items_at:h.worker_items_at + 4 * (workers + 1)].tobytes(), dtype=np.uint32)
    covered, parts, slots = np.zeros((h.row_blocks, h.chunks), dtype=int), [[] for _ in range(h.row_blocks)], set()
    for it in items:
        covered[it.row_block, it.chunk_begin:it.chunk_end] += 1
        parts[it.row_block].append((it.chunk_begin, it.part, it.parts))
        if it.parts > 1:
            slots.add(it.slot)
    assert np.all(covered == 1) and slots == set(range(h.partial_slots))
    for p in parts:       # K order
        assert [part for _, part, _ in sorted(p)] == list(range(len(p))) and {n for _, _, n in p} == {len(p)}
    loads = [[(items[i].row_block, items[i].chunk_begin, items[i].chunk_end) for i in range(at[w], at[w + 1])] for w in range(workers)]
    sizes = [sum(e - b for _, b, e in load) for load in loads]
    assert max(sizes) - min(sizes) <= 1
    if paired:
        for even, odd in zip(loads[::2], loads[1::2]):
            assert [(rb + 1, b, e) for rb, b, e in even] == odd and all(rb % 2 == 0 for rb, _, _ in even)


def test_an_image_is_held_to_its_partition(orc):
    for shape, workers, paired in SHAPES[1:5]:     # (four workers for four row blocks: the two partitions coincide)
        _, image, h = _image(orc, shape, workers)
        for value in (1 - paired, 2 if paired else 1):
            bad = image.copy()
            other = resident.header_of(bad)
            other.paired = value
            bad[:ctypes.sizeof(other)] = np.frombuffer(bytes(other), dtype=np.uint8)
            with pytest.raises(ValueError):
                resident.validate_image(bad)


@pytest.mark.parametrize("layout", ["window", "rans"])
def test_other_layouts_keep_the_plain_partition(orc, layout):
    _, _, h = _image(orc, (512, 2048), 6, layout)
    assert h.paired == 0
