"""A call that finds no device memory fails with a status and leaves nothing
half made: once the memory is there, the same call on the same context gives
the bytes of a context that never failed."""
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
