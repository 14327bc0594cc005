"""Frames whose tables give a main symbol a frequency that no word uses, so that it has no residual model: a producer that
smooths its tables makes them.  They are valid, and decode everywhere."""
import zlib

import numpy as np
import pytest

from georefine_b200 import codec


def smoothed_frame(orc, shape=(48, 512)):
    """A mode 128 frame (coded residuals) in which one context lends one slot to a main symbol that never occurs."""
    words = orc.synthetic_weight_words(*shape, 21) & np.uint16(0xFFF8)
    f = codec.parse(codec.encode(words))
    assert f["mode"] == codec.MODE_CONDITIONAL
    a, lib, rc, cc, nr, nc = codec._input(words), codec._lib(), f["rows"], f["columns"], f["nr"], f["nc"]
    main = np.frombuffer(f["main_table"], dtype="<u4").copy().reshape(nr * nc, 1024)
    residual = np.frombuffer(f["residual_table"], dtype="<u4").copy()
    unused = int(np.flatnonzero(~main.any(axis=0))[0])
    assert not residual.reshape(1024, 64)[unused].any()
    main[0, np.argmax(main[0])] -= 1
    main[0, unused] = 1
    streams = [codec._encode_under(lib, a, rc, cc, nr, nc, kind, t) for kind, t in ((0, main), (1, residual))]
    labels, tables = zlib.compress(rc.tobytes() + cc.tobytes(), 6), zlib.compress(main.tobytes() + residual.tobytes(), 6)
    head = codec._Head(codec.MODE_CONDITIONAL, nr, nc, *shape, (len(labels), len(tables), *map(len, streams)), f["digest"])
    return words, codec._sealed(head.pack(), labels, tables, *streams)


def test_host_decodes_and_indexes(orc):
    from georefine_b200 import gpu

    words, frame = smoothed_frame(orc)
    assert np.array_equal(codec.decode(frame), words)
    indexed = gpu.index_frame(frame, 128, keep_words=True)
    assert np.array_equal(indexed["words"], words)
    assert gpu._packed_tables(indexed, 128) is None       # bctx_decode_kernel's


def test_invalid_tables_are_still_refused(orc):
    from georefine_b200 import gpu

    indexed = gpu.index_frame(smoothed_frame(orc)[1], 128)
    indexed["main_freq"][1, 0] += 1
    with pytest.raises(codec.CodecError, match="invalid frequency tables"):
        gpu._packed_tables(indexed, 128)


@pytest.mark.gpu
def test_gpu_decodes_and_gathers(orc):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from georefine_b200.gpu import CudaContextTensor

    words, frame = smoothed_frame(orc)
    t = CudaContextTensor(frame, device="cuda:0", fused=False)
    assert np.array_equal(t.decode().view(torch.uint16).cpu().numpy(), words)
    ids = torch.tensor([47, 0, 5])
    assert np.array_equal(t.gather_rows(ids).view(torch.uint16).cpu().numpy(), words[ids.numpy()])
