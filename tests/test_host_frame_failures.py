"""The whole-frame passes of the host coder where memory or threads run out: an error, never the end of the process."""
import subprocess
import sys
from pathlib import Path

import pytest

SCRIPT = """
import resource, sys
import numpy as np
from georefine_b200 import codec

spare, rows = int(sys.argv[1]) << 20, 2048
a = codec._input(np.random.default_rng(0).integers(0, 65536, (rows, 2048), dtype=np.uint16))
rc, cc = codec._labels(a, 64, 16)
lib = codec._lib()
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + spare, resource.RLIM_INFINITY))
for name, call in (("frequencies", lambda: codec._both_frequencies(lib, a, rc, cc, 64, 16)), ("labels", lambda: codec._labels(a, 64, 16))):
    try:
        call()
        print(name, "done")
    except (codec.CodecError, MemoryError) as exc:
        print(name, type(exc).__name__)
"""


@pytest.mark.skipif(sys.platform != "linux", reason="address-space limits")
@pytest.mark.parametrize("spare", [1, 4, 10, 20, 40, 80, 1500])     # MB left: nothing, some shares' counts, some threads' stacks, everything
def test_workers_that_get_no_memory_report_it(spare):
    run = subprocess.run([sys.executable, "-c", SCRIPT, str(spare)], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, (run.returncode, run.stderr[-500:])
    assert [line.split()[0] for line in run.stdout.splitlines()] == ["frequencies", "labels"]
    if spare == 1500:
        assert run.stdout.split() == ["frequencies", "done", "labels", "done"]


@pytest.mark.parametrize("mask", [0xFFFF, 0xFFF8])
def test_frames_are_made_and_read_without_a_second_thread(orc, monkeypatch, mask):
    import threading

    import numpy as np

    from georefine_b200 import codec
    from georefine_b200.gpu import index_frame

    words = orc.synthetic_weight_words(300, 999, 3) & np.uint16(mask)
    assert words.size >= codec._BESIDE_WORDS
    want = codec.encode(words)

    def refused(self):
        raise RuntimeError("can't start new thread")

    monkeypatch.setattr(threading.Thread, "start", refused)
    frame = codec.encode(words)
    assert frame == want and np.array_equal(codec.decode(frame), words)
    assert np.array_equal(index_frame(frame, 128, keep_words=True)["words"], words)
    for at in (codec.HEADER.size + 5, len(frame) // 2, len(frame) - 1):
        broken = bytearray(frame)
        broken[at] ^= 1
        with pytest.raises(codec.CodecError, match="frame checksum mismatch"):
            codec.decode(bytes(broken))
