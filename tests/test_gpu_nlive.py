"""nlive of tp_map3_jobs_device: the points whose line-of-sight sum was
evaluated, in FP64 for every kind of cosmology."""
import math

import numpy as np
import pytest

from conftest import COSMO1

pytestmark = pytest.mark.gpu
KMIN, KMAX = 1e-4, 1e3


def _run(ctx, tp, torch, prec=0):
    th = torch.tensor(np.array([(8, 8, 16), (16, 16, 16)]) * tp.ARCMIN, dtype=torch.float64, device="cuda")
    jc = torch.zeros(2, dtype=torch.int32, device="cuda")
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    nev, nl = (torch.full((2,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ctx.map3_jobs_device(jc, th, out, neval=nev, nlive=nl, precision=prec)
    torch.cuda.synchronize()
    return out.cpu().numpy(), nev.cpu().numpy(), nl.cpu().numpy()


@pytest.mark.parametrize("kind", ["table", "fit", "spectrum"])
def test_nlive_counts_every_form(nz256, kind):
    """a tabulated P(k), the fit, and a spectral index outside the integer form"""
    import threepoint_gb300 as tp
    import torch

    kw = {}
    c = dict(COSMO1, ns=1.6) if kind == "spectrum" else dict(COSMO1)
    if kind == "table":
        dk = math.log(KMAX / KMIN) / 256
        k = KMIN * np.exp(dk * np.arange(256))
        kw = dict(pk=2e4 * k / (1 + (k / 0.02) ** 2) ** 1.3, dk=dk, kmin=KMIN, kmax=KMAX)
    with tp.Context(0) as a, tp.Context(0) as b:
        b.set_reference_forms(True)
        for ctx in (a, b):
            ctx.set_cosmology(tp.cosmology(**c), nz256, **kw)
        va, na, la = _run(a, tp, torch)
        vb, nb, lb = _run(b, tp, torch)
    assert np.all(la > 0) and np.all(la <= na)
    assert np.array_equal(na, nb) and np.array_equal(la, lb)
    if kind == "fit":
        assert np.max(np.abs(va / vb - 1)) < 1e-11
    else:  # one form alone: the same bits
        assert np.array_equal(va, vb)
