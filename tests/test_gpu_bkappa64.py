"""FP64 b_kappa in integer arithmetic against the CPU oracle: block remainders,
the edges of its ell domain and the inputs that keep the FP64 instructions."""
import numpy as np
import pytest

from conftest import COSMO1

pytestmark = pytest.mark.gpu


def _tri(rng, n, lo, hi):
    l1, l2 = np.exp(rng.uniform(np.log(lo), np.log(hi), (2, n)))
    c = np.cos(0.5 * rng.uniform(0, np.pi, n))
    return np.stack([l1, l2, np.sqrt((l1 - l2) ** 2 + 4 * l1 * l2 * c * c)], 1)


def _bound(ell):
    """The cosines of the tree-level kernel F2 come from differences of squares
    of the given ell, an error of a few eps (l_max / l_min) that F2 multiplies
    by l_max / l_min: 64 eps (l_max / l_min)^2, beside ~1e-12 of the ~100
    roundings of a node and of the tables' r_sigma."""
    return 1e-12 + 64 * 2.2e-16 * (ell.max(1) / ell.min(1)) ** 2


@pytest.mark.parametrize("n", [1, 31, 32, 33, 257])
@pytest.mark.parametrize("lo,hi", [(1.0, 100.0), (400.0, 4e4), (1e-9, 1e-7), (1e6, 1e8)])
def test_points(gpu_ctx, oracle_tables, n, lo, hi):
    ell = _tri(np.random.default_rng(n), n, lo, hi)
    ref = oracle_tables.bkappa_batch(ell)
    got = gpu_ctx.bkappa(ell)
    assert np.all(np.isfinite(got))
    ok = np.abs(ref) > 1e-290
    assert np.all((np.abs(got - ref) <= _bound(ell) * np.abs(ref))[ok])
    term, _ = gpu_ctx.bkappa_nodes(ell)
    assert np.max(np.abs(term.sum(1) - got) / np.maximum(np.abs(term).sum(1), 1e-300)) < 1e-13


def test_cosmologies_outside_the_integer_domain(nz256):
    """zmax > 10 (tree-level nodes), a spectrum with alpha_n's limit below 0 and
    an extreme density in one batch with an ordinary cosmology"""
    import oracle as O
    import threepoint_gb300 as tp

    cs = [dict(COSMO1), dict(COSMO1, zmax=12.0), dict(COSMO1, ns=1.6), dict(COSMO1, om=0.9, ow=0.1, omc=0.852, sigma8=1.6)]
    ell = _tri(np.random.default_rng(3), 40, 100.0, 1e4)
    with tp.Context(0) as ctx:
        ctx.set_cosmologies([tp.cosmology(**c) for c in cs], nz256)
        for i, c in enumerate(cs):
            ref = O.Tables(c, nz256).bkappa_batch(ell)
            got = ctx.bkappa(ell, cosmo_index=i)
            # 1e-10: the agreement of the z tables (test_gpu_core), to the powers of BiHalofit
            assert np.all(np.abs(got - ref) <= (_bound(ell) + 1e-8) * np.abs(ref)), i


@pytest.mark.parametrize("th", [(8.0, 8.0, 8.0), (8.0, 8.0, 16.0), (8.0, 16.0, 16.0)])
def test_symmetric_integrals_keep_the_reference_sequence(gpu_ctx, oracle_tables, th):
    """Radii with mirror-image regions: the ties at the cut and the split axes
    are decided by the FP64 form, so one CTA, an 8- and a 16-CTA cluster agree
    to rounding and the result is the oracle's within the tolerance"""
    import threepoint_gb300 as tp

    t = [np.array(th) * tp.ARCMIN]
    v16, i16 = gpu_ctx.map3_batch(t, return_info=True)
    try:
        gpu_ctx.set_map3_cluster(2)
        v8, i8 = gpu_ctx.map3_batch(t, return_info=True)
        gpu_ctx.set_map3_cluster(False)
        v1, i1 = gpu_ctx.map3_batch(t, return_info=True)
    finally:
        gpu_ctx.set_map3_cluster(True)
    assert i16["neval"][0, 0] == i8["neval"][0, 0] == i1["neval"][0, 0]
    assert abs(v16[0, 0] / v1[0, 0] - 1) < 1e-13 and abs(v8[0, 0] / v1[0, 0] - 1) < 1e-13
    assert abs(v1[0, 0] / oracle_tables.map3(list(t[0]))[0] - 1) < 1e-6
