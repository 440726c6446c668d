"""The eight-lane geodesic's reciprocal of the finite-difference span
(gc_recip_2del) against CUDA's division, bit for bit, over the interval in
which its derivation holds: |x / (2 DEL) - 1| < 2^-18, its ends and middle
double by double, and the spans of the coordinates that rays have."""
import ctypes as C

import pytest

import ipole_b200 as ip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2])
def test_reciprocal_is_the_division(seed):
    bad = (C.c_ulonglong * 3)()
    rc = ip.lib().ipg__check_recip(0, 30_000_000, C.c_ulonglong(seed), C.c_double(2. ** -18), bad)
    assert rc == ip.IPG_OK
    assert list(bad) == [0, 0, 0]
