"""The FP32 Gamma point record from the fast geometry has the floats of the
reference form's angles, next to degenerate triangles and cancelling sides too."""
import math

import numpy as np
import pytest

from conftest import COSMO1

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


@pytest.fixture(scope="module")
def pair(nz256):
    """contexts of the default forms and of the reference forms alone"""
    import threepoint_gb300 as tp

    a, b = tp.Context(0), tp.Context(0)
    b.set_reference_forms(True)
    for c in (a, b):
        c.set_cosmology(tp.cosmology(**COSMO1), nz256)
    yield a, b
    a.close()
    b.close()


TRIANGLES = [(10, 9, 3), (2, 2, 1), (1, 0.5, 0.5), (1, 0.50001, 0.5), (100, 99, 1.001), (5, 5, 1e-3), (3600, 3000, 2000)]


@pytest.mark.parametrize("tri", TRIANGLES)
@pytest.mark.parametrize("which", [0, 1])
def test_gamma_fp32_record_has_the_reference_forms_floats(pair, tri, which):
    """Random points, points near ell3 = 0 (phi = pi, psi = pi/4) and points
    where a side A_j or a phase cancels: equal records give equal sums"""
    import threepoint_gb300 as tp

    rng = np.random.default_rng(int(1e3 * tri[1]) + which)
    x = np.array(tri) * tp.ARCMIN
    n = 6000
    p = rng.uniform((0.01, 0, 0), (2.99, TWO_PI, math.pi / 2), (n, 3))
    e = 10.0 ** rng.uniform(-7, -1, (n, 2)) * rng.choice([-1, 1], (n, 2))
    near = np.stack([p[:, 0], math.pi + e[:, 0], math.pi / 4 + e[:, 1]], 1)
    # A_j = |x1 psi2 + x2 psi1 e^(i ...)| cancels for some j at these psi
    psi = np.arctan(np.array([tri[0] / tri[1], tri[1] / tri[2], tri[2] / tri[0]]))[rng.integers(0, 3, n)]
    cancel = np.stack([p[:, 0], p[:, 1], np.clip(psi + e[:, 1] * rng.integers(0, 2, n), 1e-6, 1.57)], 1)
    line = np.stack([p[:, 0], np.abs(math.pi * rng.integers(0, 3, n) + e[:, 0]) % TWO_PI, cancel[:, 2]], 1)
    for pts in (p, near, cancel, line):
        v, r = (c.gamma_integrand_points(which, x, pts, precision=1) for c in pair)
        assert np.array_equal(v, r, equal_nan=True), np.flatnonzero(v != r)[:5]


def test_gamma_fp32_integrals_are_the_reference_forms(pair):
    import threepoint_gb300 as tp

    x = np.array([(10, 9, 3), (2, 2, 1), (8, 8, 8), (5, 4, 2)]) * tp.ARCMIN
    v, r = (c.gamma_batch(x, precision=1) for c in pair)
    assert np.array_equal(v, r)
