"""analyse_peaks with shell lists short enough for a quarter of a warp per
peak (nhunt 2) against the oracle: batches that leave a warp's last quarters
without a peak, and peaks on the grid's faces and corners, whose shells are
cut by it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import peakpatch_b200 as pp

# the sums are exact to 2^-45 and single-redshift results are smooth in them;
# a factor of 1e4 is left for the interpolations and divisions between
RTOL = 1e-9


@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("npk", [1, 2, 3, 5, 64, 1003])
def test_short_lists_vs_oracle(ctx, ora, julia_table, npk, plain):
    n, alatt = 24, 2.0
    rng = np.random.default_rng(npk)
    f = {k: rng.standard_normal((n, n, n)).astype(np.float32) * s for k, s in
         (("delta", 1.0), ("etax", 1.0), ("etay", 1.0), ("etaz", 1.0), ("eta2x", 0.3), ("eta2y", 0.3), ("eta2z", 0.3),
          ("lapd", 1.0))}
    f["delta"] = (f["delta"] + np.float32(2.5)).astype(np.float32)
    f = {k: np.ascontiguousarray(v, np.float32) for k, v in f.items()}
    ijk = rng.integers(0, n, (npk, 3))
    edge = rng.random((npk, 3)) < 0.3
    ijk = np.where(edge, rng.choice([0, 1, n - 1], (npk, 3)), ijk)
    ipp = 1 + ijk[:, 0] + n * (ijk[:, 1] + n * ijk[:, 2])
    Rf = rng.choice([2.0, 3.0, 4.5], npk)
    ir2 = rng.integers(1, 4, npk)
    ctx.set_collapse_table(pp.CollapseTable(julia_table.data, julia_table.x1, julia_table.x2, julia_table.y1,
                                            julia_table.y2, julia_table.z1, julia_table.z2))
    o = ora.analyse_peaks(f, ipp, Rf, ir2, 1.0, 1.686, alatt, ora.precompute_shells(2), julia_table)
    g = ctx.analyse_peaks(f, ipp, Rf, ir2, 1.0, 1.686, alatt, 2, plain=plain)
    assert np.array_equal(g[:, 0] > 0, o[:, 0] > 0)
    if npk >= 64:
        assert (o[:, 0] > 0).sum() > 5
    fin = np.isfinite(o)
    assert np.array_equal(np.isfinite(g), fin)
    scale = np.maximum(np.abs(o), 1e-3 * np.nanmax(np.where(fin, np.abs(o), 0), axis=0, keepdims=True) + 1e-30)
    err = np.where(fin, np.abs(g - o) / scale, 0.0)
    assert err.max() <= RTOL, (err.max(), np.unravel_index(err.argmax(), err.shape))
