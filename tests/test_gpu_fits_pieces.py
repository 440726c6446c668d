"""The fits at points (ipg_thermal_coefficients) go through the device in
pieces of 2^18 points, in a workspace that the context keeps; a second
thread's call has one of its own, and a call whose result lies over its
points goes as one piece.  A point's coefficients depend on nothing but the
point, so every call must give, bit for bit, what small calls give."""
import threading

import numpy as np
import pytest

import ipole_b200 as ip
from tests import fits_points

pytestmark = pytest.mark.gpu

PIECE = 1 << 18


@pytest.fixture(scope="module")
def base():
    """points that no two pieces repeat in the same order, and theirs"""
    pts = fits_points.grid_points()
    with ip.Context() as c:
        return pts, c.thermal_coefficients(pts)


def tiled(base, n):
    at = np.arange(n) * 7919 % len(base[0])
    return base[0][at], base[1][at]


@pytest.mark.parametrize("n", [PIECE - 1, PIECE, PIECE + 1, 2 * PIECE + 3])
def test_pieces(base, n):
    pts, ref = tiled(base, n)
    with ip.Context() as c:
        for m in (5, n, 33):
            assert c.thermal_coefficients(pts[:m]).tobytes() == ref[:m].tobytes(), m


@pytest.mark.parametrize("n", [1000, PIECE + 1])
@pytest.mark.parametrize("shift", [0, 7, -7])
def test_result_over_the_points(base, n, shift):
    pts, ref = tiled(base, n)
    buf = np.empty(12 * n + 14)
    src, dst = buf[7:7 + 5 * n], buf[7 + shift:7 + shift + 12 * n]
    src[:] = pts.ravel()
    with ip.Context() as c:
        ip._check(ip.lib().ipg_thermal_coefficients(c._h, src.ctypes.data, n, 4, ip.IPG_FITS_FP64, dst.ctypes.data))
    assert dst.tobytes() == ref.tobytes()


def test_two_threads(base):
    got = {}
    with ip.Context() as c:
        def call(k, n):
            got[k] = [c.thermal_coefficients(tiled(base, n)[0]) for _ in range(4)]
        th = [threading.Thread(target=call, args=a) for a in ((0, PIECE + 5), (1, 40000))]
        for t in th:
            t.start()
        for t in th:
            t.join()
    for k, n in ((0, PIECE + 5), (1, 40000)):
        ref = tiled(base, n)[1].tobytes()
        assert all(g.tobytes() == ref for g in got[k])
