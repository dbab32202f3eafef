"""The fast forms of the integrands against their reference forms on the GPU:
the same regions are refined."""
import numpy as np
import pytest

from conftest import COSMO1

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair(nz256):
    """contexts of the default forms and of the reference forms alone"""
    import threepoint_gb300 as tp

    a, b = tp.Context(0), tp.Context(0)
    b.set_reference_forms(True)
    for c in (a, b):
        c.set_cosmology(tp.cosmology(**COSMO1), nz256)
        c.set_shape_noise(0.3, 10 / tp.ARCMIN ** 2)
    yield a, b
    a.close()
    b.close()


def test_map3_refines_the_regions_of_the_reference_form(pair):
    """Mirror-symmetric radii whose integrals, without the reference passes at
    the cut, take another sequence and are off by 1e-10 to 3e-7"""
    import threepoint_gb300 as tp

    th = np.array([(2.5, 2.5, 3), (3, 3, 4), (4, 4, 10), (5, 5, 20), (6, 6, 10), (6, 8, 8), (8, 8, 16), (10, 20, 20),
                   (12, 12, 16), (16, 16, 16), (4, 8, 16)]) * tp.ARCMIN
    (v, i), (r, j) = (c.map3_batch(th, return_info=True) for c in pair)
    assert np.array_equal(i["neval"], j["neval"])
    assert np.max(np.abs(v / r - 1)) < 1e-11


def test_gamma_fp64_takes_the_sequence_of_the_reference_form(pair):
    import threepoint_gb300 as tp

    x = np.array([(2, 2, 1), (3, 2.5, 2), (4, 4, 4)]) * tp.ARCMIN
    v, r = (c.gamma_batch(x) for c in pair)
    assert np.max(np.abs(v - r) / np.abs(r)) < 1e-10


@pytest.mark.parametrize("term,geometry", [(1, 2), (2, 1), (2, 0), (4, 2)])
def test_covariance_takes_the_sequence_of_the_reference_form(pair, term, geometry):
    import threepoint_gb300 as tp

    t = 14 * tp.ARCMIN
    a, b = np.array([(t, t, t), (t, t, 2 * t)]), np.array([(t, t, t), (t, 2 * t, 2 * t)])
    kw = dict(geometry=geometry, thetaMax=600 * tp.ARCMIN, area=(600 * tp.ARCMIN) ** 2)
    v, r = (c.cov_total(term, a, b, **kw) for c in pair)
    assert np.max(np.abs(v / r - 1)) < 1e-11
