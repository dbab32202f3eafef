"""The integer-arithmetic tables of the FP64 integrands are there for the calls
that read them, and a large FP32 set of cosmologies does not hold them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set(n):
    import threepoint_gb300 as tp

    rng = np.random.default_rng(8)
    return [tp.cosmology.flat(*v) for v in rng.uniform((0.2, 0.7, 0.6, -1.2, 0.92), (0.4, 0.9, 0.8, -0.8, 1.0), (n, 5))]


def test_large_sets_build_them_on_the_first_fp64_call(nz256):
    import threepoint_gb300 as tp
    import torch

    cs, i = _set(256), 200
    th = np.array([(16, 16, 16), (8, 16, 16)]) * tp.ARCMIN
    x = np.array([(2, 2, 1)]) * tp.ARCMIN
    pts = np.array([[1.0, 2.0, 0.5], [0.4, 5.0, 1.1]])
    ell = np.exp(np.random.default_rng(1).uniform(3, 9, (20, 1))) * np.array([[1.0, 1.1, 1.3]])
    kw = dict(geometry=tp.GEOM_INFINITE, area=(600 * tp.ARCMIN) ** 2)
    calls = [lambda c, k: c.bkappa(ell, cosmo_index=k), lambda c, k: np.stack(c.bkappa_nodes(ell, cosmo_index=k)),
             lambda c, k: c.map3_batch(th, cosmo_index=[k])[0], lambda c, k: c.gamma_batch(x, rel_tol=1e-2, cosmo_index=k),
             lambda c, k: c.gamma_integrand_points(0, x[0], pts, cosmo_index=k),
             lambda c, k: c.cov_total(1, th[:1], th[1:], cosmo_index=k, **kw),
             lambda c, k: c.cov_total(4, th[:1], th[:1], cosmo_index=k, **kw)]
    with tp.Context(0) as one:
        one.set_cosmology(cs[i], nz256)
        ref = [f(one, 0) for f in calls]
    for f, r in zip(calls, ref):
        with tp.Context(0) as ctx:
            free = torch.cuda.mem_get_info()[0]
            ctx.set_cosmologies(cs, nz256)
            held = free - torch.cuda.mem_get_info()[0]
            assert held < 256 * 400e3, held  # 327 KB a cosmology, 709 with the tables
            v = f(ctx, i)  # the first FP64 call
            assert np.array_equal(v, r)
            # a later set, and a larger one, are built with them
            ctx.set_cosmologies(cs[::-1] + cs[:3], nz256)
            assert np.array_equal(f(ctx, 255 - i), r)


def test_under_capture_without_tables(nz256):
    """A captured FP64 <Map^3> launch before any other FP64 call of a large set:
    nothing is allocated, and the FP64 instructions give the same integrals"""
    import math

    import threepoint_gb300 as tp
    import torch

    th = torch.tensor(np.array([(16, 16, 16), (8, 16, 16)]) * tp.ARCMIN, dtype=torch.float64, device="cuda")
    jc = torch.full((2,), 30, dtype=torch.int32, device="cuda")
    out, ref = (torch.zeros(2, dtype=torch.float64, device="cuda") for _ in range(2))
    L = tp.lib()
    with tp.Context(0) as ctx:
        ctx.set_cosmologies(_set(40), nz256)
        torch.cuda.synchronize()
        rt = torch.cuda.ExternalStream(ctx.stream_handle)
        g = torch.cuda.CUDAGraph()
        p = lambda t: t.data_ptr()  # noqa: E731
        L.tp_map3_jobs_noalloc(ctx._h, p(jc), p(th), 2, 0.0, 2 * math.pi, 1.0, 0.0, 1e-4, 0, p(out), None, None)
        torch.cuda.synchronize()
        out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=rt):
            rc = L.tp_map3_jobs_noalloc(ctx._h, p(jc), p(th), 2, 0.0, 2 * math.pi, 1.0, 0.0, 1e-4, 0, p(out), None, None)
        assert rc == 0
        g.replay()
        torch.cuda.synchronize()
        ctx.map3_jobs_device(jc, th, ref, precision=0)
        torch.cuda.synchronize()
        a, b = out.cpu().numpy(), ref.cpu().numpy()
    assert np.all(a > 0) and np.max(np.abs(a / b - 1)) < 1e-11
