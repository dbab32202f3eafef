"""The Gamma integrand at angles outside [0, 2 pi) and [0, pi / 2]."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TWO_PI = 2 * math.pi


@pytest.mark.parametrize("which", [0, 1])
def test_gamma_fp32_points_at_any_angle(gpu_ctx, which):
    """angles outside [0, 2 pi): the integrand is periodic in phi, and FP32
    agrees with FP64 as inside"""
    import threepoint_gb300 as tp

    rng = np.random.default_rng(which)
    x = np.array((4, 6, 8)) * tp.ARCMIN
    p = rng.uniform((0.05, 0, 0.05), (2.9, TWO_PI, 1.5), (200, 3))
    ref = gpu_ctx.gamma_integrand_points(which, x, p)
    for turns in (-7, -3, -1, 1, 2, 5, 11):
        q = p + [0, turns * TWO_PI, 0]
        for prec, tol in ((0, 1e-10), (1, 1e-3)):
            got = gpu_ctx.gamma_integrand_points(which, x, q, precision=prec)
            assert np.max(np.abs(got - ref)) < tol * np.max(np.abs(ref)), (turns, prec)
    q = p + [0, 0, TWO_PI]
    got = gpu_ctx.gamma_integrand_points(which, x, q, precision=1)
    assert np.max(np.abs(got - ref)) < 1e-3 * np.max(np.abs(ref))
