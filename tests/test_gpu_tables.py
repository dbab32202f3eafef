"""The table build's forms for few and for many cosmologies give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cosmologies(n):
    import threepoint_gb300 as tp

    rng = np.random.default_rng(12)
    odd = [tp.cosmology.flat(0.3, 0.0, 0.7, -1.0, 0.96), tp.cosmology.flat(1.0, 0.8, 0.7, -1.0, 0.96),
           tp.cosmology.flat(0.2, 0.7, 0.6, -0.4, 1.1, zmax=0.4), tp.cosmology.flat(0.4, 0.9, 0.8, -1.3, 0.9, zmax=40.0)]
    box = [tp.cosmology.flat(om, s8, h, w, ns) for om, s8, h, w, ns in
           rng.uniform((0.2, 0.7, 0.6, -1.2, 0.92), (0.4, 0.9, 0.8, -0.8, 1.0), (n - len(odd), 5))]
    return odd + box


# set sizes at which the bins a warp or the form change: 6 -> 1 bin, 7 and 12 -> 2, 13 and 24 -> 4, 25 the narrow form
@pytest.mark.parametrize("size", [1, 6, 7, 12, 13, 24])
def test_few_cosmologies_have_the_tables_of_many(nz256, size):
    import threepoint_gb300 as tp

    cs = cosmologies(25)
    many, few = tp.Context(0), tp.Context(0)
    try:
        many.set_cosmologies(cs, nz256)
        for i0 in range(0, 25 if size > 1 else 6, size):
            part = cs[i0:i0 + size]
            few.set_cosmologies(part, nz256)
            for i in range(len(part)):
                a, b = few.tables(i), many.tables(i0 + i)
                for k in b:
                    assert np.array_equal(a[k], b[k], equal_nan=True), (k, i0 + i)
    finally:
        many.close()
        few.close()
