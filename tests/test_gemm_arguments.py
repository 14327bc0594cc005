"""grb_bxr_gemm checks what it is given before anything is launched (no GPU needed)."""
import ctypes

import pytest

UNSUPPORTED, WORKSPACE = 2, 3
MAGIC, WINDOW, WINDOW4 = 0x31525842, 2, 3


@pytest.mark.parametrize("mode,workers,chunks,want", [(WINDOW4, 65536, 65536, UNSUPPORTED), (WINDOW4, 65536, 70000, UNSUPPORTED),
                                                      (WINDOW4, 65535, 70000, WORKSPACE), (WINDOW4, 70000, 65535, WORKSPACE), (WINDOW, 65536, 65536, WORKSPACE)])
def test_row_blocks_of_more_parts_than_are_counted(mode, workers, chunks, want):
    """A row block's counter has sixteen bits for its parts; the workspace is too small for any of these, which is looked at next."""
    from georefine_b200 import _native

    lib = _native.lib()
    h = _native.BxrHeader(magic=MAGIC, mode=mode, rows=128, cols=128 * chunks, row_blocks=1, chunks=chunks, workers=workers, items=workers,
                          partial_slots=workers, layout_version=lib.bxr_layout_version())
    at = 1 << 20      # an address that nothing follows
    assert lib.grb_bxr_gemm(at, ctypes.byref(h), at, 128 * chunks, 1, at, 128, None, at, 256, at, None) == want
