"""grb_bctx_decode_packed checks what it is given before anything is launched: arguments that no launch may follow (no GPU needed)."""
import ctypes

import pytest

BAD_ARGUMENT, UNSUPPORTED = 1, 2


def arguments(rows=8, cols=256, mode=0):
    from georefine_b200 import _native

    t, p, at = _native.BctxTensor(), _native.BctxPacked(), 1 << 20      # addresses that nothing follows
    for name, kind in t._fields_:
        if kind is ctypes.c_void_p:
            setattr(t, name, at)
    t.rows, t.cols, t.n, t.nr, t.nc, t.mode, t.stride = rows, cols, rows * cols, 16, 4, mode, 128
    t.main_bytes, t.residual_bytes = 1000, -(-rows * cols * 6 // 8)
    p.tables = at
    p.shape[:] = (3, 16880, 8, 64 * 16880, 64 * 16880)
    return t, p


def status(t, p, count=16):
    from georefine_b200 import _native

    return _native.lib().grb_bctx_decode_packed(ctypes.byref(t), ctypes.byref(p), None, count, 1 << 20, 1 << 20, None, None)


@pytest.mark.parametrize("rows,cols", [(8, 256), (3, 257), (5, 17)])
def test_raw_residuals_that_end_early(rows, cols):
    t, p = arguments(rows, cols)
    t.residual_bytes -= 1
    assert status(t, p, -(-rows * cols // 128)) == BAD_ARGUMENT
    t.residual_bytes += 1
    assert status(t, p, 0) == 0                                  # nothing to do, nothing wrong


@pytest.mark.parametrize("wrong", [{"stride": 24}, {"cols": 15}, {"mode": 1}, {"residual_stream": (1 << 20) + 8}, {"main_states": None}])
def test_other_arguments(wrong):
    t, p = arguments()
    for name, value in wrong.items():
        setattr(t, name, value)
    t.n = t.rows * t.cols
    assert status(t, p) in (BAD_ARGUMENT, UNSUPPORTED)
