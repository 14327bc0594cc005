"""The cache of resident images and the rule by which their work is cut: an entry of another rule is never looked at."""
import hashlib
import json

import numpy as np

from georefine_b200 import codec, image_cache, resident


def _plain(image):
    """The image as a build without the partition of pairs cut it: the same blobs, the items of ascending shares."""
    from georefine_b200 import _native
    import ctypes

    old = image.copy()
    h = resident.header_of(old)
    items, at = [], [0]
    units = h.row_blocks * h.chunks
    for w in range(h.workers):
        u, end = units * w // h.workers, units * (w + 1) // h.workers
        while u < end:
            rb, c0 = divmod(u, h.chunks)
            c1 = min(h.chunks, c0 + end - u)
            items.append([rb, c0, c1])
            u += c1 - c0
        at.append(len(items))
    parts = {rb: sum(i[0] == rb for i in items) for rb in range(h.row_blocks)}
    assert len(items) == h.items
    seen, slot = {}, 0
    records = np.frombuffer(old[h.items_at:h.items_at + 32 * h.items].tobytes(), dtype=np.uint32).reshape(-1, 8).copy()
    fields = [name for name, _ in _native.BxrItem._fields_]
    for rec, (rb, c0, c1) in zip(records, items):
        values = {"row_block": rb, "chunk_begin": c0, "chunk_end": c1, "part": seen.setdefault(rb, 0), "parts": parts[rb]}
        seen[rb] += 1
        if parts[rb] > 1:
            values["slot"], slot = slot, slot + 1
        for name, value in values.items():
            rec[fields.index(name)] = value
    old[h.items_at:h.items_at + 32 * h.items] = records.reshape(-1).view(np.uint8)
    old[h.worker_items_at:h.worker_items_at + 4 * len(at)] = np.array(at, dtype=np.uint32).view(np.uint8)
    h.paired = 0
    old[:ctypes.sizeof(h)] = np.frombuffer(bytes(h), dtype=np.uint8)
    return old


def test_an_entry_cut_by_the_rule_before_is_not_served(orc, tmp_path, monkeypatch):
    words = orc.synthetic_weight_words(512, 2048, 5)
    frame = codec.encode(words)
    source, workers = hashlib.sha256(words.tobytes()).hexdigest(), 6
    new, h = resident.build_image(words, workers)
    assert h.paired == 1
    old = _plain(new)
    resident.validate_image(old)                                    # still a good image, for whoever holds one
    assert np.array_equal(resident.decode_image_host(old), words)
    # the entry that the build before wrote: its key knows the layout version alone
    material = {"schema": image_cache.SCHEMA, "cache_format": image_cache.CACHE_FORMAT, "layout_version": image_cache.layout_version(),
                "source_sha256": source, "shape": [512, 2048], "layout": "window4", "workers": workers}
    key = hashlib.sha256(json.dumps(material, sort_keys=True, separators=(",", ":")).encode()).hexdigest()
    (tmp_path / key[:2]).mkdir()
    (tmp_path / key[:2] / f"{key}.bxr").write_bytes(old.tobytes())
    (tmp_path / key[:2] / f"{key}.json").write_text(json.dumps({**material, "mode": 3, "image_bytes": int(old.size),
                                                                "image_sha256": hashlib.sha256(old.tobytes()).hexdigest()}))
    cache = image_cache.ImageCache(tmp_path)
    image, _, hit = image_cache.image_for_frame(frame, workers, cache=cache)
    assert not hit and np.array_equal(image, new) and cache.stats["quarantined"] == 0
    assert (tmp_path / key[:2] / f"{key}.bxr").read_bytes() == old.tobytes()      # and left to the build that wrote it
    assert image_cache.image_for_frame(frame, workers, cache=cache)[2]
    # another rule, another entry
    monkeypatch.setattr(image_cache, "partition_version", lambda: 3)
    assert cache.get(source, (512, 2048), "window4", workers) is None and cache.stats["quarantined"] == 0
