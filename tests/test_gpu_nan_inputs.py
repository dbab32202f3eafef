"""Point evaluations at coordinates that are no numbers, or whose geometry gives
none, read no table outside its bounds: they return, and the context goes on."""
import math

import numpy as np
import pytest

from conftest import COSMO1

pytestmark = pytest.mark.gpu
KMIN, KMAX = 1e-4, 1e3


@pytest.fixture(params=["fit", "table"])
def ctx(request, nz256):
    import threepoint_gb300 as tp

    c = tp.Context(0)
    kw = {}
    if request.param == "table":
        dk = math.log(KMAX / KMIN) / 256
        k = KMIN * np.exp(dk * np.arange(256))
        kw = dict(pk=2e4 * k / (1 + (k / 0.02) ** 2) ** 1.3, dk=dk, kmin=KMIN, kmax=KMAX)
    c.set_cosmology(tp.cosmology(**COSMO1), nz256, **kw)
    yield c
    c.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_not_a_number(ctx, prec):
    import threepoint_gb300 as tp

    arc, nan, inf = tp.ARCMIN, math.nan, math.inf
    ok = np.array([[1.0, 2.0, 0.5]])
    before = ctx.gamma_integrand_points(0, np.array([3, 4, 5]) * arc, ok, precision=prec)
    pts = np.array([[nan, 1, 1], [1, nan, 1], [1, 1, nan], [nan, nan, nan], [inf, 1, 1], [-inf, 1, 1], [1, inf, 1],
                    [1, 1, inf], [1, -1e300, 1], [-1, 1, 1]])
    for which in (0, 1):
        # an ordinary triangle and one whose angles are those of a line
        for x in ([3, 4, 5], [1, 0.5, 0.5], [1.0000000000000002, 0.5, 0.5]):
            got = ctx.gamma_integrand_points(which, np.array(x) * arc, pts, precision=prec)
            assert not np.any(np.abs(got[3:5]) > 0) or np.all(np.isfinite(got[3:5]))
    for bad in (nan, -1.0, 0.0):
        with pytest.raises(tp.ThreepointError):
            ctx.Pell([bad, 100.0], precision=prec)
    p = ctx.Pell([inf, 1e300, 100.0], precision=prec)
    assert np.isfinite(p[2]) and p[2] > 0
    b = ctx.bkappa([[nan, 1, 1], [inf, 10, 10], [-1, 2, 2], [100, 100, 100]], precision=prec)
    assert b[0] == 0 and b[2] == 0 and b[3] > 0
    for term, nd in ((5, 6), (7, 7)):
        x = np.full((4, nd), 3.0)
        for m in (nan, 1.0, -1.0, 1e40):
            x[:, -1] = m
            with pytest.raises(tp.ThreepointError):
                ctx.halo_integrand(term, np.full(6, 4 * arc), x, precision=prec)
    assert np.array_equal(ctx.gamma_integrand_points(0, np.array([3, 4, 5]) * arc, ok, precision=prec), before)
