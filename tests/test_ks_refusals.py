"""dpl_shp_ks refuses a window that is too large whatever the cutoff, before any work."""

import ctypes as C

import pytest

from dolphin_gb300 import _lib

UNSUPPORTED = 5


@pytest.mark.parametrize("is_sorted", [0, 1])
@pytest.mark.parametrize("cutoff", [0.3, 0.0, -1.0, float("nan")])
def test_window_too_large(cutoff, is_sorted):
    lib = _lib.load()
    n, rows, cols, hy, hx = 20, 200, 200, 60, 60  # 121 x 121 pixels of 20 samples: 1.2 MB
    size = lib.dpl_shp_ks_workspace_size(n, rows, cols)
    buf = (C.c_char * 256)()  # refused before any of the arrays is touched
    p = C.addressof(buf)
    st = lib.dpl_shp_ks(p, n, rows, cols, hy, hx, 1, 1, cutoff, is_sorted, p, p, size, None)
    assert st == UNSUPPORTED
    assert b"window too large" in lib.dpl_last_error_message()


@pytest.mark.parametrize("n,rows,cols", [(1, 1, 1), (20, 37, 41), (64, 512, 512)])
def test_workspace_holds_the_sorted_samples_only(n, rows, cols):
    assert _lib.load().dpl_shp_ks_workspace_size(n, rows, cols) == -(-4 * n * rows * cols // 256) * 256
