"""ppb_find_peaks on identical fields, bit for bit against the oracle: four-cell
groups marched along k (n1 and nbuff multiples of 4) at rows and columns that
leave a block or a warp partly empty, planes that leave a march short, NaN,
infinities and plateaus, and more peaks per warp than its list holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,n3,nbuff", [(12, 9, 9, 4), (16, 13, 10, 4), (36, 41, 23, 4), (64, 24, 19, 8),
                                            (136, 131, 149, 4), (160, 160, 160, 16)])
@pytest.mark.parametrize("kind", ["noise", "special", "flat"])
def test_march_bit_exact(ctx, ora, n1, n2, n3, nbuff, kind):
    rng = np.random.default_rng(n1 * n2 + n3)
    d = rng.standard_normal((n3, n2, n1)).astype(np.float32)
    fcrit = np.float32(0.25)
    if kind == "special":
        d = np.round(d * 2) / 2   # ties
        pick = rng.random(d.shape)
        d[pick < 0.01] = np.inf
        d[(pick >= 0.01) & (pick < 0.02)] = -np.inf
        d[(pick >= 0.02) & (pick < 0.05)] = np.nan
    if kind == "flat":
        d[:] = 1.0
    mo = (rng.random(d.shape) < 0.05).astype(np.int8)
    mg = mo.copy()
    o = ora.find_peaks(d, mo, 0.0, 0.0, 0.0, 1.0, nbuff, fcrit)
    g = ctx.find_peaks(d, mg, 0.0, 0.0, 0.0, 1.0, nbuff, fcrit)
    for key in ("i", "j", "k", "ipp"):
        assert np.array_equal(g[key], o[key]), key
    assert np.array_equal(g["delta"], o["delta"], equal_nan=True)
    assert np.array_equal(mg, mo)
