"""What a small grid holds on the device (fields, both streams' buffers, plans
and their work areas, peak buffers) stays within the estimate that serving
charges for it."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import peakpatch_b200 as pp

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(pp.__file__))), "libppb.so")


def _estimate(n):
    f = ctypes.CDLL(LIB)._ZN3ppb19tile_bytes_estimateEi
    f.argtypes, f.restype = [ctypes.c_int], ctypes.c_uint64
    return f(n)


# own transforms (128, 160), cuFFT sizes without (150) and with work areas (111, 142)
@pytest.mark.parametrize("n", [111, 128, 142, 150, 160])
def test_held_bytes_within_the_estimate(n):
    import torch

    rng = np.random.default_rng(n)
    radii = [1.5 * 20 ** (i / 19) for i in range(20)]

    def search(c, m):
        d = rng.standard_normal((m, m, m)).astype(np.float32)
        c.peak_find_tile(d, radii, [3.0] * 20, np.zeros((m, m, m), np.int8), 0.0, 0.0, 0.0, 2.0, 4, 1, 1)

    with pp.Context(0) as c:   # loads every kernel
        search(c, n)
    with pp.Context(0) as c:
        search(c, 32)
        before = torch.cuda.mem_get_info()[0]
        search(c, n)
        held = before - torch.cuda.mem_get_info()[0]
    held += 32 * n ** 3   # the packed records, made by a run's gather only
    print(n, held >> 20, _estimate(n) >> 20)
    assert held <= _estimate(n)
