"""The profile pool of a call in several batches: on the second identical call
no batch overflows the pool and runs again (each run of a batch is one graph
launch)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import peakpatch_b200 as pp
from conftest import filter_bank
from test_gpu_parity import tile_config
from test_low_memory import Hog


@pytest.mark.parametrize("order", ["large first", "mixed"])
def test_second_call_runs_each_batch_once(julia_table, order):
    T = julia_table
    n, npk, nhunt = 64, 60000, 24
    rng = np.random.default_rng(5)
    f = {k: rng.standard_normal((n, n, n)).astype(np.float32) for k in ("delta", "etax", "etay", "etaz")}
    f["delta"] += np.float32(4.0)   # above fcrit to the end of every list: all its shells are kept
    ipp = rng.integers(1, n ** 3 + 1, npk)
    big = np.arange(npk) < npk // 2   # lists of r^2 <= 576, about 480 shells, and of r^2 <= 9
    if order == "mixed":
        rng.shuffle(big)
    lim = np.where(big, nhunt ** 2, 9)
    rf = np.where(big, 24.0, 4.0)
    with pp.Context(0) as c:
        c.set_collapse_table(pp.CollapseTable(T.data, T.x1, T.x2, T.y1, T.y2, T.z1, T.z2))
        c.set_option(pp.OPT_AUTOTUNE, 0)
        hog = Hog(3 << 30)   # the pool may take half of what is left
        try:
            out, runs, batches = [], [], []
            for _ in range(3):
                before = c.graph_stats()["launches"]
                out.append(c.analyse_peaks(f, ipp, rf, 4, 1.0, 1.686, 2.0, nhunt, r2lim=lim))
                runs.append(c.graph_stats()["launches"] - before)
                batches.append(c.shell_stats()["batches"])
        finally:
            hog.give_back()
    assert batches[0] > 1
    assert runs[1:] == batches[1:], (runs, batches)
    assert out[0].tobytes() == out[1].tobytes() == out[2].tobytes()


def test_kinds_of_batch_in_turn_on_one_slot(julia_table, eh_pk):
    """A short-list batch, a plain tile, a lightcone tile and a tile, whose
    rows per peak differ by two orders, in turn on one context: the bytes of
    each alone, whatever the pool's size was before."""
    T = julia_table
    n, npk = 64, 20000
    rng = np.random.default_rng(6)
    f = {k: rng.standard_normal((n, n, n)).astype(np.float32) for k in ("delta", "etax", "etay", "etaz")}
    f["delta"] += np.float32(2.0)
    ipp = rng.integers(1, n ** 3 + 1, npk)
    rf = [r[2] for r in filter_bank()]
    calls = [lambda c: c.analyse_peaks(f, ipp, 4.0, 3, 1.0, 1.686, 2.0, 2),
             lambda c: c.run_tile_arrays(tile_config(), 3, rf, plain=True)[0],
             lambda c: c.run_tile_arrays(tile_config(ievol=1, z_max=1.0), 3, rf)[0],
             lambda c: c.run_tile_arrays(tile_config(n=80, box=160.0), 3, rf)[0]]

    def context():
        c = pp.Context(0)
        c.set_pk_table(*eh_pk)
        c.set_collapse_table(pp.CollapseTable(T.data, T.x1, T.x2, T.y1, T.y2, T.z1, T.z2))
        c.set_option(pp.OPT_TUNE_MIN_PEAKS, 1)
        return c

    alone = []
    for call in calls:
        with context() as c:
            alone.append(call(c).tobytes())
    assert all(len(a) > 0 for a in alone)
    with context() as c:
        for order in ([0, 1, 2, 3], [3, 0, 2, 1], [1, 0, 3, 2]):
            for i in order:
                assert calls[i](c).tobytes() == alone[i], (order, i)
