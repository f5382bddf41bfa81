"""The frequencies that the k^2-weighted twin leaves out: the weight of the
first one is below 1e-10 of the window's largest, two to three orders under
the single-precision rounding of the modes kept."""
import ctypes
import math
import os

import pytest

import peakpatch_b200 as pp

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(pp.__file__))), "libppb.so")


@pytest.mark.skipif(not os.path.exists(LIB), reason="library not built")
@pytest.mark.parametrize("n", [64, 192, 384, 512])
@pytest.mark.parametrize("cell", [0.3, 2.0, 6.4])
def test_dropped_weight(n, cell):
    flim = ctypes.CDLL(LIB)._ZN3ppb9twin_flimEidd
    flim.argtypes, flim.restype = [ctypes.c_int, ctypes.c_double, ctypes.c_double], ctypes.c_int
    box = n * cell
    for R in (0.1, 1.5, 3.0, 7.9, 13.0, 30.0, 200.0, 1e9):
        f = flim(n, box, R)
        assert 1 <= f <= n // 2
        if f < n // 2:
            x2 = (2 * math.pi * (f + 1) / box * R) ** 2
            assert x2 * math.exp(-x2 / 8) < 1e-10 * 8 / math.e, R
