"""FP64 b_kappa of a triangle does not depend on the batch it is in: the forms
for few and for many points, both forms of a node, block remainders."""
import math

import numpy as np
import pytest

from conftest import COSMO1

pytestmark = pytest.mark.gpu
KMIN, KMAX = 1e-4, 1e3


@pytest.mark.parametrize("table", [False, True])
def test_same_bits_in_any_batch(nz256, table):
    import threepoint_gb300 as tp

    rng = np.random.default_rng(5)
    l1, l2 = np.exp(rng.uniform(np.log(1.0), np.log(4e4), (2, 4000)))
    c = np.cos(0.5 * rng.uniform(0, np.pi, 4000))
    ell = np.stack([l1, l2, np.sqrt((l1 - l2) ** 2 + 4 * l1 * l2 * c * c)], 1)
    ell[::97] = [1e-11, 5, 5]
    ell[1::97] = [3e7, 3e7, 3e7]  # beyond the integer form's P(k) table
    kw = {}
    if table:
        dk = math.log(KMAX / KMIN) / 256
        k = KMIN * np.exp(dk * np.arange(256))
        kw = dict(pk=2e4 * k / (1 + (k / 0.02) ** 2) ** 1.3, dk=dk, kmin=KMIN, kmax=KMAX)
    with tp.Context(0) as ctx:
        ctx.set_cosmology(tp.cosmology(**COSMO1), nz256, **kw)
        many = ctx.bkappa(ell)
        for n in (1, 7, 8, 9, 31, 257, 2432, 2433):
            for at in (0, 13):
                assert np.array_equal(ctx.bkappa(ell[at:at + n]), many[at:at + n]), (n, at)
        assert np.all(np.isfinite(many)) and np.all(many[::97] == 0)
