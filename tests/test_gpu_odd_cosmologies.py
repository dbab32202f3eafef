"""The integer forms of the FP64 integrands against their reference forms for
cosmologies at the edges of their rows: tree-level nodes beyond z = 10, low and
high amplitudes, a steep spectrum, extreme densities, a shallow survey."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [dict(zmax=12.0), dict(sigma8=0.1, zmax=10.0), dict(sigma8=0.03), dict(sigma8=3.0), dict(ns=1.6), dict(ns=-0.5),
         dict(om=0.9, sigma8=1.6), dict(om=0.05, h=0.4, omb=0.01), dict(w=-0.3), dict(zmax=0.1), dict(omb=0.0)]


@pytest.mark.parametrize("change", CASES, ids=lambda c: ",".join(f"{k}={v}" for k, v in c.items()))
def test_forms_agree(nz256, change):
    import threepoint_gb300 as tp

    par = dict(om=0.3, sigma8=0.8, h=0.7, w=-1.0, ns=0.96)
    par.update(change)
    rng = np.random.default_rng(6)
    ell = []
    for lo, hi in ((1e-10, 1e-2), (1.0, 1e2), (1e2, 1e5), (1e5, 1e9)):  # and past both ends of the P(k) table
        l1, l2 = np.exp(rng.uniform(np.log(lo), np.log(hi), (2, 60)))
        c = np.cos(0.5 * rng.uniform(0, np.pi, 60))
        ell.append(np.stack([l1, l2, np.sqrt((l1 - l2) ** 2 + 4 * l1 * l2 * c * c)], 1))
    ell = np.concatenate(ell)
    x = np.array([10, 9, 3]) * tp.ARCMIN
    pts = rng.uniform((0.001, 0, 0.01), (min(par.get("zmax", 3.0), 3.0), 6.28, 1.56), (100, 3))
    t = 16 * tp.ARCMIN
    a, b = np.array([(t, t, t)]), np.array([(t, t, 2 * t)])
    got = []
    for on in (False, True):
        with tp.Context(0) as ctx:
            ctx.set_reference_forms(on)
            ctx.set_cosmology(tp.cosmology.flat(**par), nz256)
            ctx.set_shape_noise(0.3, 10 / tp.ARCMIN ** 2)
            kw = dict(thetaMax=600 * tp.ARCMIN, area=(600 * tp.ARCMIN) ** 2)
            got.append([ctx.bkappa(ell)] + [ctx.gamma_integrand_points(w, x, pts) for w in (0, 1)] +
                       [ctx.cov_total(1, a, b, geometry=tp.GEOM_INFINITE, **kw),
                        ctx.cov_total(2, a, b, geometry=tp.GEOM_CIRCLE, **kw)])
    v, r = got
    # F2's cancellation (l_max / l_min)^2 beside ~1e-12 of the rounding of a node
    ok = np.abs(r[0]) > 1e-290
    q = (ell.max(1) / ell.min(1))[ok]
    assert np.all(np.abs(v[0] / np.where(r[0] == 0, 1, r[0]) - 1)[ok] <= 1e-11 + 64 * 2.2e-16 * q ** 2)
    for k in (1, 2):
        assert np.max(np.abs(v[k] - r[k])) <= 1e-10 * np.max(np.abs(r[k]))
    for k in (3, 4):
        assert np.max(np.abs(v[k] - r[k]) / np.abs(r[k])) < 1e-11
