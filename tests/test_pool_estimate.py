"""The profile pool of a call in several batches: on the second identical call
no batch overflows the pool and runs again (each run of a batch is one graph
launch)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import peakpatch_b200 as pp
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
