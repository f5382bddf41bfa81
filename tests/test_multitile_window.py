"""run_multitile for one tile away from the grid's origin: its records are the
bytes that the same tile has in a run with other tiles, the k^2-weighted twin
at the peaks (d2Rf) among them."""
import pytest

pytestmark = pytest.mark.gpu

import peakpatch_b200 as pp
from conftest import filter_bank
from test_gpu_parity import tile_config

RF = [f[2] for f in filter_bank()]


@pytest.fixture(scope="module")
def gctx(julia_table, eh_pk):
    T = julia_table
    with pp.Context(0) as c:
        c.set_pk_table(*eh_pk)
        c.set_collapse_table(pp.CollapseTable(T.data, T.x1, T.x2, T.y1, T.y2, T.z1, T.z2))
        yield c


# full grids of 112^3 (own transforms) and 104^3 (full transforms)
@pytest.mark.parametrize("nbuff", [8, 12])
@pytest.mark.parametrize("tile", [(1, 1, 1), (2, 1, 1), (1, 2, 2)])
def test_one_tile_alone_and_among_others(gctx, nbuff, tile):
    cfg = tile_config()
    cfg.n, cfg.nbuff, cfg.boxsize = 64, nbuff, 128.0
    alone, _, _ = gctx.run_multitile_arrays(cfg, 5, RF, ntile=2, tiles=[tile])
    both, _, _ = gctx.run_multitile_arrays(cfg, 5, RF, ntile=2, tiles=[tile, (2, 2, 1)])
    assert alone.shape[1] == 33 and len(alone) > 20
    assert both[:len(alone)].tobytes() == alone.tobytes()
