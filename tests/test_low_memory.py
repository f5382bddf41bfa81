"""A call that finds no device memory fails with a status and leaves nothing
half made: once the memory is there, the same call on the same context gives
the bytes of a context that never failed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import peakpatch_b200 as pp
from conftest import filter_bank
from test_gpu_parity import tile_config

RF = [f[2] for f in filter_bank()]
MIB = 1 << 20


def _cfg(n):
    cfg = tile_config()
    cfg.n, cfg.nbuff, cfg.boxsize = n, 16, 2.0 * n
    return cfg


def _context(eh_pk, T):
    c = pp.Context(0)
    c.set_pk_table(*eh_pk)
    c.set_collapse_table(pp.CollapseTable(T.data, T.x1, T.x2, T.y1, T.y2, T.z1, T.z2))
    return c


class Hog:
    """All of the device's free memory but `leave` bytes."""

    def __init__(self, leave):
        import torch
        torch.cuda.empty_cache()
        self.held = []
        for unit in (1 << 30, 64 * MIB, 4 * MIB):
            take = (torch.cuda.mem_get_info()[0] - leave) // unit * unit
            if take > 0:
                self.held.append(torch.empty(take, dtype=torch.uint8, device="cuda"))

    def give_back(self):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


# 128^3: own transforms; 142^3: full transforms, plans with work areas; 192^3: the fused search
@pytest.mark.parametrize("n", [128, 142, 192])
def test_a_run_without_memory_and_the_next_one(eh_pk, julia_table, n):
    with _context(eh_pk, julia_table) as c:   # also loads every kernel
        want, rmax, npk = c.run_tile_arrays(_cfg(n), 3, RF)
    assert len(want) > 20
    failed = 0
    for leave in (16, 48, 96, 144, 192, 256, 320, 400, 512, 700, 1000):
        with _context(eh_pk, julia_table) as c:
            hog = Hog(leave * MIB)
            try:
                c.run_tile_arrays(_cfg(n), 3, RF)
            except pp.PPBError as e:
                assert e.code in (-2, -3), (leave, str(e))   # a library without memory may answer with another status
                failed += 1
            finally:
                hog.give_back()
            got, r, k = c.run_tile_arrays(_cfg(n), 3, RF)
            assert got.tobytes() == want.tobytes() and r == rmax and k == npk, leave
    assert failed >= 4


def _keep_stub_buffers(c, n=256):
    """An analyse_peaks call whose staging (about 1 GiB) the context keeps."""
    rng = np.random.default_rng(1)
    f = {k: np.zeros((n, n, n), np.float32) for k in ("delta", "etax", "etay", "etaz", "eta2x", "eta2y", "eta2z")}
    f["delta"][:] = 2.5
    ipp = rng.integers(1, n ** 3, 50)
    c.analyse_peaks(f, ipp, np.full(50, 4.0), np.full(50, 3), 1.0, 1.686, 2.0, 2)


@pytest.mark.parametrize("call", ["tile", "served", "merge", "fields", "stub", "alloc"])
def test_kept_stub_buffers_are_given_back(eh_pk, julia_table, call):
    """A call that needs more than is free, and less than that with the kept
    staging of an earlier analyse_peaks, succeeds as it did before that call."""
    import ctypes

    rng = np.random.default_rng(2)
    rec = np.zeros((900000, 33), np.float32)
    rec[:, :3] = rng.uniform(-500, 500, (len(rec), 3))
    rec[:, 6] = 1.0

    def run(c):
        if call == "tile":
            return c.run_tile_arrays(_cfg(128), 3, RF)[0].tobytes()
        if call == "served":
            return c.wait(c.submit(_cfg(128), 3, RF))[0].tobytes()
        if call == "merge":
            return np.sort(c.merge_catalog(rec)[:, 0]).tobytes()
        if call == "fields":
            out = np.empty((128, 128, 128), np.float32)
            p = c._params(_cfg(128), 3, False)
            c._check(c.L.ppb_generate_fields(c.h, ctypes.byref(p), out.ctypes.data, None, None, None))
            return out.tobytes()
        if call == "stub":   # another stub call, whose buffers the kept ones do not hold
            d = rng.standard_normal((8, 8, 8)).astype(np.float32)
            big = np.zeros((320, 320, 320), np.float32)
            big[100:108, 100:108, 100:108] = np.abs(d) + 1
            return len(c.find_peaks(big, np.zeros(big.shape, np.int8), 0.0, 0.0, 0.0, 1.0, 4, 1.5)["i"]) > 0
        p = ctypes.c_void_p()
        c._check(c.L.ppb_alloc_device(c.h, ctypes.c_size_t(600 * MIB), ctypes.byref(p)))
        c._check(c.L.ppb_free_device(c.h, p))
        return True

    with _context(eh_pk, julia_table) as c:   # also loads every kernel
        _keep_stub_buffers(c)
        want = run(c)
    # less than the call needs: fields 260 MiB, a tile over 600, the merge over 250, the search over 500
    leave = {"tile": 250, "served": 250, "fields": 120, "merge": 100, "stub": 200, "alloc": 200}[call]
    with _context(eh_pk, julia_table) as c:
        _keep_stub_buffers(c)
        hog = Hog(leave * MIB)
        try:
            assert run(c) == want
        finally:
            hog.give_back()
