"""Device scratch of the residual check, computed on the host (no GPU)."""
import ctypes
import os

import pytest

from rochpl_b200 import build


@pytest.mark.parametrize("n", [1, 300, 2049, 16384, 50000, 102400, 102401, 131072, 150000])
def test_scratch(n):
    """A regenerated matrix takes its row sums (2 per row and 2048 columns), and so
    does a stored one of 100 thousand rows and more, where the matrix may fill the
    GPU; below that a stored one takes at most 1 / 256 of itself on top."""
    lib = ctypes.CDLL(build.LIB) if os.path.exists(build.LIB) else ctypes.CDLL(build.build())
    f = lib["_ZN4hplb19residual_ws_doublesEib"]
    f.restype, f.argtypes = ctypes.c_size_t, [ctypes.c_int, ctypes.c_bool]
    rows = 2 * -(-n // 2048) * n
    small = n + 64  # per-block values
    assert f(n, True) <= rows + small
    if n > 102400:
        assert f(n, False) <= rows + small
    else:
        assert f(n, False) <= rows + 2 * 256 * 2048 + (-(-n // 256) + 1) * n + small
