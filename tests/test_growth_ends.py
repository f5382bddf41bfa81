"""D(a) among the first entries of the growth table: the four interpolation
points never start before the first entry."""
import numpy as np
import pytest

import peakpatch_b200 as pp

STEP = np.exp(np.log(2.0 / 1e-7) / 2000)   # ratio of neighbouring entries
FIRST = 1e-7 * STEP ** np.ceil(np.log(1e7 / 1001.0) / np.log(STEP))   # the first one, at or above a = 1/1001


def test_growth_between_the_first_entries(ora):
    """Without baryons the growth's derivatives are continuous there and a
    four-point interpolation of D(a)/a is exact to (STEP - 1)^4 of its slow
    change, below 1e-10: a polynomial through the entries from the third on
    gives the values between the second and the third too."""
    cosmo = (0.315, 0.0, 0.685, 0.674)
    x = np.linspace(0.02, 9.98, 499)
    a = FIRST * STEP ** x
    g = np.asarray(ora.dlinear(*cosmo, a)) / a
    p = np.polynomial.Polynomial.fit(x[x > 2], g[x > 2], 6)
    assert np.abs(g / p(x) - 1).max() < 1e-10
    f = np.array([ora.fsc_of_z(*cosmo, 1 / v - 1) for v in a]) / (1.686 * a)
    assert np.allclose(f, g, rtol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("iforce", [1, 4, 6])
def test_table_started_among_the_first_entries(ora, iforce):
    """Nodes that start (a = 1 / (zinit_fac F)) before the first entry and
    between each of the following ones, bit for bit."""
    cosmo = (0.315, 0.049, 0.685, 0.674)
    kw = dict(Nx=25, Ny=3, Nz=3, X1=-5 * np.log10(STEP), X2=np.log10(STEP), iforce_strat=iforce,
              zinit_fac=1.0 / FIRST)
    with pp.Context(0) as c:
        g = c.make_table(*cosmo, pp.CollapseTableParams(**kw))
    o = ora.make_table(*cosmo, ora.TableParams(**kw))
    assert np.isfinite(o).all()
    assert g.tobytes() == o.tobytes(), np.abs(g - o).max()
