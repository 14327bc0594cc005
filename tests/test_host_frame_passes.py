"""The whole-frame passes of the host coder (csrc/bcx_frame.cpp) against the oracle and the stream-by-stream functions."""
import numpy as np
import pytest

from georefine_b200 import codec
from georefine_b200.gpu import checkpoints, index_frame

SHAPES = [(1, 1), (1, 7), (5, 1), (3, 16), (33, 65), (300, 999), (2, 70000)]     # the last two run on several threads


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("classes", [(1, 1), (16, 4), (64, 16)])
@pytest.mark.parametrize("kind", ["weights", "coarse", "constant", "noise"])
def test_frames_equal_the_oracle_and_decode_in_one_pass(orc, oracle_coder, shape, classes, kind):
    words = orc.synthetic_weight_words(*shape, 7)
    if kind == "coarse":
        words &= 0xFFF8                       # coded residuals win
    elif kind == "constant":
        words[:] = 0x3F80                     # every frequency is 0 or 65536
    elif kind == "noise":                     # more live symbols than the one pass takes in a context of a large enough tensor
        words = np.random.default_rng(5).integers(0, 65536, shape, dtype=np.uint16)
    frame = codec.encode(words, row_classes=classes[0], col_classes=classes[1])
    assert frame == oracle_coder.encode(words, row_classes=classes[0], col_classes=classes[1])
    assert np.array_equal(codec.decode(frame), words)
    f = codec.parse(frame)
    if f["mode"] == codec.MODE_WORDS:
        return
    for stride in (1, 48, 1024):
        i = index_frame(frame, stride)
        common = (f["rows"], f["columns"], shape, f["nr"], f["nc"], stride)
        states, offsets, main = checkpoints(f["main_stream"], i["main_freq"], *common)
        assert np.array_equal(i["main_states"], states) and np.array_equal(i["main_offsets"], offsets)
        if f["mode"] == codec.MODE_CONDITIONAL:
            states, offsets, _ = checkpoints(f["residual_stream"], i["residual_freq"], *common, main)
            assert np.array_equal(i["residual_states"], states) and np.array_equal(i["residual_offsets"], offsets)


@pytest.mark.parametrize("seed,mask", [(1, 0xFFFF), (2, 0xFFF8), (3, 0xFFE0), (4, 0x7F80)])
def test_residual_floor_is_below_the_stream_and_close(orc, seed, mask):
    words = orc.synthetic_weight_words(700, 700, seed) & np.uint16(mask)
    a, lib = codec._input(words), codec._lib()
    rc, cc = codec._labels(a, 16, 4)
    main, residual, floor = codec._both_frequencies(lib, a, rc, cc, 16, 4)
    for kind, table in ((0, main), (1, residual)):
        assert codec._encode_kind(lib, a, rc, cc, 16, 4, kind) == (table.tobytes(), codec._encode_under(lib, a, rc, cc, 16, 4, kind, table))
    stream = codec._encode_under(lib, a, rc, cc, 16, 4, 1, residual)
    # the bound gives away 0.0114 bits per word and what bytes before rare symbols cost
    assert floor <= len(stream) <= floor + 0.0114 / 8 * a.size + 64 + 0.02 * len(stream)


@pytest.mark.parametrize("choice,decoder", [(None, None), ("0", "bcx_decode"), ("1", "bcx_decode_compact")])
@pytest.mark.parametrize("mask", [0xFFFF, 0xFFF8])
def test_the_environment_chooses_the_stream_decoder(orc, monkeypatch, choice, decoder, mask):
    words = orc.synthetic_weight_words(300, 999, 3) & np.uint16(mask)
    frame = codec.encode(words)
    lib, called = codec._lib(), []

    class Watched:
        def __getattr__(self, name):
            called.append(name)
            return getattr(lib, name)

    monkeypatch.setattr(codec, "_lib", Watched)
    if choice is None:
        monkeypatch.delenv("GEOREFINE_CONTEXT_COMPACT_RANS", raising=False)
    else:
        monkeypatch.setenv("GEOREFINE_CONTEXT_COMPACT_RANS", choice)
    assert np.array_equal(codec.decode(frame), words)
    streams = 2 if mask != 0xFFFF else 1
    assert [name for name in called if name.startswith("bcx_decode")] == ([decoder] * streams if decoder else [])
    monkeypatch.setenv("GEOREFINE_CONTEXT_COMPACT_RANS", "2")
    with pytest.raises(codec.CodecError, match="must be 0 or 1"):
        codec.decode(frame)
