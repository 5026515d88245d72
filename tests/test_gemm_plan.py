"""The trailing update's choice of tiles and grid, on the host (no GPU)."""
import ctypes
import os

import pytest

from rochpl_b200 import build


@pytest.fixture(scope="module")
def plan():
    lib = ctypes.CDLL(build.LIB) if os.path.exists(build.LIB) else ctypes.CDLL(build.build())
    f = lib["_ZN4hplb10plan_dgemmEiiiiPiPxS1_"]
    f.restype = None

    def call(m, n, sms, cap):
        small, tpc, grid = ctypes.c_int(), ctypes.c_longlong(), ctypes.c_longlong()
        f(m, n, sms, cap, ctypes.byref(small), ctypes.byref(tpc), ctypes.byref(grid))
        return bool(small.value), tpc.value, grid.value

    return call


def _tiles(m, n, t):
    return -(-m // t) * -(-n // t)


@pytest.mark.parametrize("cap", [0, 1, 48, 116, 132, 147])
def test_cap_holds_for_every_size(plan, cap):
    """HPLB_OPT_PANEL_SMS = k: at most SMs - k CTAs, small tiles included (products of
    up to two thirds of the SMs in 128 x 128 tiles launched four times as many
    CTAs as those whatever the cap)."""
    sms = 148
    for m in (1, 64, 65, 128, 129, 700, 1280, 1281, 1408, 2048, 4000, 16384, 130560):
        for n in (1, 63, 64, 128, 130, 1152, 1280, 1500, 4097, 130561):
            small, tpc, grid = plan(m, n, sms, cap)
            t = _tiles(m, n, 64 if small else 128)
            assert small == (3 * _tiles(m, n, 128) <= 2 * sms)
            assert grid == -(-t // tpc) and tpc >= 1, (m, n, tpc, grid)
            assert cap == 0 or grid <= cap, (m, n, cap, grid)
            if cap == 0 and small:
                assert tpc == 1


@pytest.mark.parametrize("sms", [132, 148, 160])
def test_small_tiles_leave_no_second_round(plan, sms):
    """Two small tiles fit an SM: products that take them need at most two rounds, the
    second at most a third full (from 100 to 111 tiles of 128 on 148 SMs the small ones
    were 5% slower than the large)."""
    for t in range(1, 2 * sms):
        small, tpc, grid = plan(128 * t, 128, sms, 0)
        if small:
            assert grid <= 2 * sms * 4 // 3, (t, grid)
        else:
            assert 3 * t > 2 * sms
