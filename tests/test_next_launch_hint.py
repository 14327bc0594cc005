"""Which blobs a launch asks the L2 for on behalf of the next one (bxr_leading_blobs, the rule the kernel follows), for every worker of plain and
of paired partitions: the leading ones of its share that follow one another in memory, eight of them where the share has them."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "georefine_b200" / "csrc"
MOST = 8


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    compiler = shutil.which("gcc") or shutil.which("cc")
    if compiler is None:
        pytest.skip("no C compiler")
    at = tmp_path_factory.mktemp("hint")
    (at / "rule.c").write_text('#include "bxr_format.h"\nuint32_t rule(uint32_t rb, uint32_t c, uint32_t w, uint32_t p, uint32_t i, uint32_t m, uint32_t* f)'
                               " { return bxr_leading_blobs(rb, c, w, p, i, m, f); }\n")
    subprocess.run([compiler, "-shared", "-fPIC", "-I", str(CSRC), str(at / "rule.c"), "-o", str(at / "rule.so")], check=True)
    return ctypes.CDLL(str(at / "rule.so")).rule


def _share(row_blocks, chunks, workers, paired, w):
    """The blobs of worker w's share in the order it walks them (one row block after another, chunk by chunk)."""
    if not paired:
        order, share, shares = [(rb, c) for rb in range(row_blocks) for c in range(chunks)], w, workers
    else:
        order, share, shares = [(2 * g + w % 2, c) for g in range(row_blocks // 2) for c in range(chunks)], w // 2, workers // 2
    return [rb * chunks + c for rb, c in order[len(order) * share // shares:len(order) * (share + 1) // shares]]


@pytest.mark.parametrize("row_blocks,chunks,workers,paired", [(40, 136, 148, 0), (40, 136, 148, 1), (272, 40, 148, 0), (272, 40, 148, 1), (7, 9, 63, 0), (5, 16, 37, 0),
                                                              (4, 16, 4, 1), (4, 16, 4, 0), (3, 2, 12, 0), (30, 3, 8, 0), (30, 3, 8, 1), (1, 1, 1, 0), (2, 1, 148, 0)])
def test_leading_blobs(rule, row_blocks, chunks, workers, paired):
    first = ctypes.c_uint32()
    for w in range(workers):
        share = _share(row_blocks, chunks, workers, paired, w)
        run = next((i for i, b in enumerate(share) if b != share[0] + i), len(share))
        n = rule(row_blocks, chunks, workers, paired, w, MOST, ctypes.byref(first))
        assert n == min(run, MOST) if paired else n == min(len(share), MOST)       # (a plain share is one stretch of memory)
        assert n <= run and (not n or first.value == share[0])


def test_the_kernel_follows_the_rule():
    text = (CSRC / "bxq_kernels.cuh").read_text()
    assert "bxr_leading_blobs(args.next_row_blocks, args.next_chunks, args.next_workers, args.next_paired, w2, kWideNextBlobs, &first)" in text
