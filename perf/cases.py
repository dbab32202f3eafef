"""Workloads of the framework at the sizes its users run, for timing.

listed() gives the fixed cases and draw(rng) more of the same kinds and ranges;
prepare(case, seed) makes what a program holds before the call (contexts,
networks, likelihoods, catalogues), run(state) is one pass through the public
entry points, work(case) the bytes and operations the path cannot do without,
and exact(case, seed) what run() returns in 64 bits from plain torch and numpy.

Kinds:
  map3   a sampler's step: set_cosmologies, then <Map^3> of every triplet
  bkappa the convergence bispectrum at given triangles (surrogate targets)
  gamma  the four natural components of the shear 3PCF at given triangles
  cov    a block of <Map^3> covariance entries, one term
  apm    the <Map^3> measurement of a shear catalogue
  train  optimiser steps of the b_kappa network
  chi2   the likelihood of a batch of model vectors
"""
import math

import numpy as np
import torch

import threepoint_gb300 as tp
from threepoint_gb300 import aperture_mass
from threepoint_gb300.surrogate import sample_triangles

ARCMIN = tp.ARCMIN
FP = {"fp64": tp.FP64, "fp32": tp.FP32}
BOX = (("om", 0.2, 0.4), ("sigma8", 0.7, 0.9), ("h", 0.6, 0.8), ("w", -1.2, -0.8), ("ns", 0.92, 1.0))
SURVEY = 600 * ARCMIN  # side of the 10 x 10 deg^2 survey
SIGMA_EPS, N_GAL = 0.3, 10.0 / ARCMIN ** 2
FIELD = 240.0  # arcmin


def listed():
    return [
        # one step of a parameter sampler through the cosmosis module: a new
        # cosmology, then the 20 triplets of {2, 4, 8, 16}', FP32 integrand
        dict(name="step_fp32", kind="map3", cosmologies=1, radii="2,4,8,16", precision="fp32"),
        # the same step at the default precision, three radii
        dict(name="step_fp64", kind="map3", cosmologies=1, radii="4,8,16", precision="fp64"),
        # the throughput batch: 64 cosmologies of the parameter box x the 220
        # triplets of ten log-spaced radii on 1-32'
        dict(name="batch_fp32", kind="map3", cosmologies=64, radii="log10", precision="fp32"),
        # FP64 training targets of one cosmology of the surrogate's data set
        dict(name="bkappa_fp64", kind="bkappa", points=1 << 18, precision="fp64"),
        # one shear-3PCF triangle at the default precision
        dict(name="gamma_fp64", kind="gamma", triangles=1, r=2.0, precision="fp64"),
        # a block of the shear-3PCF grid
        dict(name="gamma_fp32", kind="gamma", triangles=64, r=10.0, precision="fp32"),
        # covariance blocks: the trispectrum-like product term in FP32, the
        # finite-survey term at the default precision, and the one-halo
        # pentaspectrum term in FP32
        dict(name="cov_t4_fp32", kind="cov", term=4, pairs=8, theta=8.0, precision="fp32"),
        dict(name="cov_t2_fp64", kind="cov", term=2, pairs=2, theta=16.0, precision="fp64"),
        dict(name="cov_t7_fp32", kind="cov", term=7, pairs=8, theta=8.0, precision="fp32"),
        # the measurement of one field: 10 galaxies per arcmin^2 on a 240' side
        dict(name="apm_field", kind="apm", npix=4096, apertures=4, density=10.0),
        # optimiser steps of the network at the batch its training runs with
        dict(name="train", kind="train", batch=65536, steps=8),
        # the smallest call: a handful of walkers' model vectors
        dict(name="chi2", kind="chi2", n=220, models=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["map3", "map3", "bkappa", "gamma", "cov", "apm", "train", "chi2"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "map3":
        if prec == "fp32":
            radii = sorted(math.exp(rng.uniform(math.log(1.5), math.log(25.0))) for _ in range(rng.randint(1, 6)))
            n = _log_int(rng, 1, 24)
        else:
            radii = sorted(math.exp(rng.uniform(math.log(5.0), math.log(25.0))) for _ in range(rng.randint(1, 3)))
            n = rng.randint(1, 2)
        return dict(kind=kind, cosmologies=n, radii=",".join("%.3f" % r for r in radii), precision=prec)
    if kind == "bkappa":
        return dict(kind=kind, points=_log_int(rng, 1, 1 << 18), precision=prec)
    if kind == "gamma":
        if prec == "fp32":
            return dict(kind=kind, triangles=_log_int(rng, 1, 48), r=round(math.exp(rng.uniform(0.0, math.log(15.0))), 3),
                        precision=prec)
        return dict(kind=kind, triangles=1, r=round(rng.uniform(1.0, 3.0), 3), precision=prec)
    if kind == "cov":
        term = rng.choice([1, 2, 4, 5, 7])
        if term in (1, 2) and prec == "fp64":
            return dict(kind=kind, term=term, pairs=rng.randint(1, 2), theta=round(rng.uniform(14.0, 20.0), 3),
                        precision=prec)
        return dict(kind=kind, term=term, pairs=rng.randint(1, 7), theta=round(rng.uniform(6.0, 18.0), 3),
                    precision="fp32")
    if kind == "apm":
        return dict(kind=kind, npix=_log_int(rng, 200, 3000), apertures=rng.randint(1, 6),
                    density=round(rng.uniform(1.0, 10.0), 2))
    if kind == "train":
        return dict(kind=kind, batch=_log_int(rng, 500, 65536), steps=rng.randint(1, 8))
    return dict(kind=kind, n=_log_int(rng, 4, 700), models=_log_int(rng, 1, 4096))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _nz():
    zs = np.arange(3001) * 1e-3
    return tp.rebin_n_of_z(zs, zs ** 2 * np.exp(-(zs / 0.5) ** 1.5))


def _cosmologies(n, seed):
    """n cosmologies, one in each of n strata of every box parameter"""
    rng = np.random.default_rng(seed)
    col = {k: lo + (rng.permutation(n) + rng.uniform(size=n)) / n * (hi - lo) for k, lo, hi in BOX}
    return [dict({k: float(col[k][i]) for k in col}, omb=0.048, omc=float(col["om"][i]) - 0.048,
                 ow=1 - float(col["om"][i]), zmax=3.0) for i in range(n)]


def _radii(case):
    r = np.exp(np.linspace(0.0, math.log(32.0), 10)) if case["radii"] == "log10" else \
        np.array([float(v) for v in case["radii"].split(",")])
    return np.array(tp.theta_triplets(list(r))) * ARCMIN


def _triangles(case, seed):
    """triangles of bin centres (r, u, v) around the case's scale: r the middle
    side, u = smallest / middle, v = (largest - middle) / smallest"""
    n = case["triangles"]
    rng = np.random.default_rng(seed)
    r = case["r"] * np.exp(rng.uniform(-0.3, 0.3, n)) * ARCMIN
    u, v = rng.uniform(0.6, 0.95, n), rng.uniform(0.1, 0.5, n)
    return np.stack([r + v * u * r, r, u * r], axis=1)


def _pairs(case):
    """pairs of triplets with radii t and 2 t (all patterns of equal and
    unequal radii that the totals distinguish)"""
    t = case["theta"]
    trip = [(t, t, t), (t, t, 2 * t), (t, 2 * t, 2 * t), (2 * t, 2 * t, 2 * t)]
    order = [(1, 2), (0, 0), (0, 1), (2, 2), (1, 1), (0, 2), (2, 3), (3, 3)]
    a = [trip[order[i % 8][0]] for i in range(case["pairs"])]
    b = [trip[order[i % 8][1]] for i in range(case["pairs"])]
    return np.array(a) * ARCMIN, np.array(b) * ARCMIN


def _catalogue(case, seed):
    """uniform positions, a smooth shear pattern and shape noise"""
    rng = np.random.default_rng(seed)
    n = int(case["density"] * FIELD * FIELD)
    x, y = rng.uniform(0.0, FIELD, n), rng.uniform(0.0, FIELD, n)
    g = 0.02 * np.exp(2j * np.pi * (x / 37.0 + y / 53.0)) + \
        SIGMA_EPS * (rng.standard_normal(n) + 1j * rng.standard_normal(n)) / math.sqrt(2)
    return x, y, g


def _apertures(case):
    return [2.0, 4.0, 8.0, 16.0, 3.0, 6.0][:case["apertures"]]


def _network(case, seed):
    """He-style initial weights and the minibatches of the steps"""
    rng = np.random.default_rng(seed)
    w = tp.MLP.WIDTHS
    params = [(rng.normal(0.0, math.sqrt(2.0 / w[i]), (w[i + 1], w[i])), np.zeros(w[i + 1])) for i in range(len(w) - 1)]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.rand((case["steps"], case["batch"], 8), generator=gen, device="cuda", dtype=torch.float32) * 2 - 1
    t = torch.sin(2 * x[..., 0] + x[..., 1]) * x[..., 3] + 0.5 * x[..., 2] * x[..., 4]
    return params, x.contiguous(), t.contiguous()


def _vectors(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    a = rng.standard_normal((n, n)) / math.sqrt(n)
    cov = a @ a.T + np.diag(rng.uniform(0.5, 1.5, n))
    data = rng.standard_normal(n)
    return data, cov, data + 0.5 * rng.standard_normal((case["models"], n))


LR = 1e-3


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "chi2":
        data, cov, s["models"] = _vectors(case, seed)
        s["like"] = tp.Likelihood(data, cov)
        return s
    if kind == "train":
        params, s["x"], s["t"] = _network(case, seed)
        s["net"] = tp.MLP(max_batch=case["batch"])
        s["net"].set_params(params)
        s["loss"] = torch.zeros(case["steps"], device="cuda", dtype=torch.float32)
        torch.cuda.synchronize()
        return s
    s["ctx"] = tp.Context(0)
    if kind == "apm":
        s["catalogue"] = _catalogue(case, seed)
        return s
    s["nz"] = _nz()
    s["cosmologies"] = [tp.cosmology(**c) for c in _cosmologies(case.get("cosmologies", 1), seed)]
    if kind == "map3":
        s["thetas"] = _radii(case)
        return s
    # the other kinds call a context that holds its cosmology
    s["ctx"].set_cosmologies(s["cosmologies"], s["nz"])
    if kind == "bkappa":
        s["ell"] = sample_triangles(np.random.default_rng(seed), case["points"])
    elif kind == "gamma":
        s["x"] = _triangles(case, seed)
    else:
        s["ctx"].set_shape_noise(SIGMA_EPS, N_GAL)
        s["a"], s["b"] = _pairs(case)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "map3":
        s["ctx"].set_cosmologies(s["cosmologies"], s["nz"])
        return s["ctx"].map3_batch(s["thetas"], precision=FP[case["precision"]])
    if kind == "bkappa":
        return s["ctx"].bkappa(s["ell"], precision=FP[case["precision"]])
    if kind == "gamma":
        return s["ctx"].gamma_batch(s["x"], precision=FP[case["precision"]])
    if kind == "cov":
        geometry = tp.GEOM_SQUARE if case["term"] == 2 else tp.GEOM_INFINITE
        return s["ctx"].cov_total(case["term"], s["a"], s["b"], geometry=geometry, thetaMax=SURVEY, area=SURVEY ** 2,
                                  precision=FP[case["precision"]])
    if kind == "apm":
        x, y, g = s["catalogue"]
        return aperture_mass.extract_Map3(x, y, g, case["npix"], _apertures(case), FIELD, ctx=s["ctx"])
    if kind == "train":
        for i in range(case["steps"]):
            s["net"].train_step_device(s["x"][i], s["t"][i], LR, s["loss"][i:i + 1])
        return s["net"].get_params(flat=True), s["loss"]
    return s["like"].chi2(s["models"])


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
NODE_FLOPS = 300.0  # arithmetic of one line-of-sight node of the bispectrum, a special function counted as ten


def work(case):
    kind = case["kind"]
    if kind == "map3":
        n = case["cosmologies"] * len(_radii(case))
        # about 1.5e5 integrand points per integral at the relative tolerance 1e-4
        return dict(bytes=n * 32.0 + case["cosmologies"] * 2120.0, flops=n * 1.5e5 * 96 * NODE_FLOPS)
    if kind == "bkappa":
        return dict(bytes=case["points"] * 32.0, flops=case["points"] * 96 * NODE_FLOPS)
    if kind == "gamma":
        # four components, about 4e4 points each, 96 bispectra a point
        return dict(bytes=case["triangles"] * 88.0, flops=case["triangles"] * 4 * 4e4 * 96 * NODE_FLOPS)
    if kind == "cov":
        points, nodes, ops = {1: (2e5, 3 * 96, 150), 2: (1e5, 96, 150), 4: (4e5, 2 * 96, NODE_FLOPS),
                              5: (1.5e6, 5 * 96, 200), 7: (5e5, 6 * 96, 200)}[case["term"]]
        return dict(bytes=case["pairs"] * 56.0, flops=case["pairs"] * points * nodes * float(ops))
    if kind == "apm":
        n, t = case["npix"], case["apertures"]
        gal = int(case["density"] * FIELD * FIELD)
        # three input grids, and per aperture three filters and two maps: real transforms of the 'same' convolution
        f = 1.5 * n
        transforms = 3 + 5 * t
        return dict(bytes=gal * 32.0 + 2.0 * 8 * n * n * (3 + 5 * t), flops=transforms * 2.5 * f * f * math.log2(f * f))
    if kind == "train":
        per_row = 2.0 * (8 * 256 + 3 * 256 * 256 + 256)
        return dict(bytes=case["steps"] * (case["batch"] * 36.0 + 201217 * 32.0),
                    flops=case["steps"] * case["batch"] * 3 * per_row)
    n, m = case["n"], case["models"]
    return dict(bytes=8.0 * (n * (n + 1) / 2 + n + m * n + m), flops=float(m) * n * (n + 1))


# ---------------------------------------------------------------------------
# run()'s values in 64 bits from plain torch and numpy
# ---------------------------------------------------------------------------
C_H0 = 2997.92  # c / H0 in Mpc/h
H0_C = 100.0 / 299792.0


def _dev(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")


class _Model:
    """BiHalofit b_kappa of one cosmology: the redshift tables on 256 bin
    centres and the 96-node line-of-sight sum."""

    NB = 256

    def __init__(self, c, nz):
        self.c = c
        zmax, om, ow, w = c["zmax"], c["om"], c["ow"], c["w"]
        a, wt = np.polynomial.legendre.leggauss(96)
        dz = zmax / self.NB
        zb = (np.arange(self.NB) + 0.5) * dz
        E = lambda z: np.sqrt(om * (1 + z) ** 3 + ow * (1 + z) ** (3 * (1 + w)))  # noqa: E731
        zz = 0.5 * zb[:, None] * (1 + a)
        self.fK = C_H0 * 0.5 * zb * (wt / E(zz)).sum(1)
        g = np.zeros(self.NB)
        for i in range(self.NB):
            term = nz[i:] * (self.fK[i:] - self.fK[i]) / self.fK[i:]
            g[i] = (term.sum() - 0.5 * term[0] - (0.5 * term[-1] if len(term) > 1 else 0.0)) * dz
        g[0] = 1.0
        self.g = g
        self.D1 = self._growth(zb) / self._growth(np.array([0.0]))
        self._norm()
        self._scales()
        # nodes of the line of sight
        self.z = 0.5 * zmax * (1 + a)
        self.wq = 0.5 * zmax * wt
        self.E = E(self.z)

    def _growth(self, z):
        c = self.c
        n = 4000
        x = np.full(len(z), math.log(1.0 / 1100.0))
        h = (-np.log1p(z) - x) / n
        y = np.stack([np.ones(len(z)), np.zeros(len(z))])

        def rhs(x, y):
            ap = np.exp(-3.0 * c["w"] * x)
            d = -0.5 * (5 * c["om"] + (5 - 3 * c["w"]) * c["ow"] * ap) * y[1] - 1.5 * (1 - c["w"]) * c["ow"] * ap * y[0]
            return np.stack([y[1], d / (c["om"] + c["ow"] * ap)])

        for _ in range(n):
            k1 = rhs(x, y)
            k2 = rhs(x + 0.5 * h, y + 0.5 * h * k1)
            k3 = rhs(x + 0.5 * h, y + 0.5 * h * k2)
            k4 = rhs(x + h, y + h * k3)
            y = y + h * (k1 + 2 * k2 + 2 * k3 + k4) / 6
            x = x + h
        return y[0] / (1 + z)

    def _pk(self, k):
        """linear P(k) [h^-3 Mpc^3] by the Eisenstein & Hu no-wiggle fit, k in h/Mpc"""
        c = self.c
        fc, fb, th = c["omc"] / c["om"], c["omb"] / c["om"], 2.728 / 2.7
        pc = 0.25 * (5 - math.sqrt(1 + 24 * fc))
        om2, ob2 = c["om"] * c["h"] ** 2, c["omb"] * c["h"] ** 2
        zeq = 2.5e4 * om2 / th ** 4
        b1 = 0.313 * om2 ** -0.419 * (1 + 0.607 * om2 ** 0.674)
        zd = 1291 * om2 ** 0.251 / (1 + 0.659 * om2 ** 0.828) * (1 + b1 * ob2 ** (0.238 * om2 ** 0.223))
        yd = (1 + zeq) / (1 + zd)
        sh = 44.5 * math.log(9.83 / om2) / math.sqrt(1 + 10 * ob2 ** 0.75)
        al = fc * (5 - 2 * pc) / 5 * (1 - 0.553 * fb + 0.126 * fb ** 3) * (1 + yd) ** -pc * \
            (1 + 0.5 * pc * (1 + 1 / (7 * (3 - 4 * pc))) / (1 + yd))
        sa = math.sqrt(al)
        kk = k * c["h"]
        geff = om2 * (sa + (1 - sa) / (1 + (0.43 * kk * sh) ** 4))
        q = kk / geff * th * th
        L = torch.log(2.718281828 + 1.84 * sa / (1 - 0.949 * fb) * q)
        C = 14.4 + 325.0 / (1 + 60.5 * q ** 1.11)
        return c["h"] ** 3 * 2 * math.pi ** 2 * self.norm ** 2 * (2997.9 / c["h"]) ** (3 + c["ns"]) * kk ** c["ns"] * \
            (L / (L + C * q * q)) ** 2

    def _moments(self, r, kinds):
        """sigma-like integrals over ln k of k^3 P(k) / (2 pi^2) times the windows at radii r"""
        t = torch.linspace(-18.0, 14.0, 20001, dtype=torch.float64, device="cuda")
        k = torch.exp(t)
        base = k ** 3 * self._pk(k) / (2 * math.pi ** 2) * (t[1] - t[0])
        x = k[None] * r[:, None]
        x2 = x * x
        out = []
        for j in kinds:
            if j == 0:
                wdw = torch.where(x < 1e-2, 1 - x2 / 10, 3 / x ** 3 * (torch.sin(x) - x * torch.cos(x))) ** 2
            else:
                wdw = torch.exp(-x2) * (1.0 if j == 1 else x2)
            out.append((base[None] * wdw).sum(1))
        return out

    def _norm(self):
        self.norm = 1.0
        s8 = self._moments(_dev([8.0]), [0])[0].sqrt().item()
        self.norm = self.c["sigma8"] / s8

    def _scales(self):
        D1 = _dev(self.D1)
        lo, hi = torch.full_like(D1, -25.0), torch.full_like(D1, 12.0)  # ln R
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            s = D1 * self._moments(torch.exp(mid), [1])[0].sqrt()
            lo, hi = torch.where(s > 1, mid, lo), torch.where(s > 1, hi, mid)
        r = torch.exp(0.5 * (lo + hi))
        self.rs = r.cpu().numpy()
        self.ne = (-3 + 2 * D1 * D1 * self._moments(r, [2])[0]).cpu().numpy()

    def _mid(self, arr, f):
        """two-point interpolation between bin centres at fractional bin f"""
        i = np.minimum(f.astype(int), self.NB - 1)
        d = np.where(f.astype(int) > self.NB - 1, 1.0, f - i)
        w = 1 - np.abs(d - 0.5)
        n = np.where(d > 0.5, np.minimum(i + 1, self.NB - 1), np.where(d < 0.5, np.maximum(i - 1, 0), i))
        iw = np.where((d > 0.5) & (i == self.NB - 1), 0.0, 1 - w)
        return arr[i] * w + arr[n] * iw

    def bkappa(self, l):
        """b_kappa of triangles l [n, 3] (CUDA float64)"""
        c = self.c
        f = self.z / c["zmax"] * self.NB
        g, fK, D1, rs, ne = (self._mid(v, f) for v in (self.g, self.fK, self.D1, self.rs, self.ne))
        W = self.wq * 27 / 8 * c["om"] ** 3 * H0_C ** 5 * (g * (1 + self.z)) ** 3 / fK / self.E
        ls = np.log10(D1 * c["sigma8"])
        omz = c["om"] / (c["om"] + c["ow"] * (1 + self.z) ** (3 * c["w"]))
        a, _ = torch.sort(l, dim=1, descending=True)
        r1, r2 = a[:, 2] / a[:, 0], (a[:, 1] + a[:, 2] - a[:, 0]) / a[:, 0]

        def tree(x, y, z):
            m = 0.5 * (z * z - x * x - y * y) / (x * y)
            return 5 / 7 + 0.5 * m * (x / y + y / x) + 2 / 7 * m * m

        F = [tree(l[:, i], l[:, (i + 1) % 3], l[:, (i + 2) % 3]) for i in range(3)]
        out = torch.zeros(len(l), dtype=torch.float64, device=l.device)
        for j in range(len(self.z)):
            n, s = float(ne[j]), float(ls[j])
            an = 10 ** (-2.167 - 2.944 * s - 1.106 * s * s - 2.865 * s ** 3 - 0.310 * r1 ** (10 ** (0.182 + 0.57 * n)))
            bn, cn = 10 ** (-3.428 - 2.681 * s + 1.624 * s * s - 0.095 * s ** 3), 10 ** (0.159 - 1.107 * n)
            al = torch.clamp(10 ** (-4.348 - 3.006 * n - 0.5745 * n * n + 10 ** (-0.9 + 0.2 * n) * r2 ** 2),
                             max=1 - 2 / 3 * c["ns"])
            be = 10 ** (-1.731 - 2.845 * n - 1.4995 * n * n - 0.2811 * n ** 3 + 0.007 * r2)
            fn = 10 ** (-10.533 - 16.838 * n - 9.3048 * n * n - 1.8263 * n ** 3)
            gn, hn = 10 ** (2.787 + 2.405 * n + 0.4577 * n * n), 10 ** (-1.118 - 0.394 * n)
            mn, nn = 10 ** (-2.605 - 2.434 * s + 5.71 * s * s), 10 ** (-4.468 - 3.08 * s + 1.035 * s * s)
            mu, nu = 10 ** (15.312 + 22.977 * n + 10.9579 * n * n + 1.6586 * n ** 3), 10 ** (1.347 + 1.246 * n + 0.4525 * n * n)
            pn, en = 10 ** (0.071 - 0.433 * n), 10 ** (-0.632 + 0.646 * n)
            dn = 10 ** (-0.483 + 0.892 * s - 0.086 * float(omz[j]))
            b1, P, q = 1.0, [], []
            for i in range(3):
                qi = l[:, i] * float(rs[j] / fK[j])
                b1 = b1 / ((an * qi ** al + bn * qi ** be) * (1 + 1 / (cn * qi)))
                pl = float(D1[j]) ** 2 * self._pk(l[:, i] / float(fK[j]))
                x = pn * qi
                P.append((1 + fn * qi * qi) / (1 + gn * qi + hn * qi * qi) * pl +
                         1 / ((mn * qi ** mu + nn * qi ** nu) * (1 + x ** -3)))
                q.append(qi)
            b3 = 2 * ((F[0] + dn * q[2]) * P[0] * P[1] + (F[1] + dn * q[0]) * P[1] * P[2] + (F[2] + dn * q[1]) * P[2] * P[0])
            out += float(W[j]) * (b1 + b3 / ((1 + en * q[0]) * (1 + en * q[1]) * (1 + en * q[2])))
        return out

    def map3(self, thetas):
        """<Map^3> of radii triplets [rad] by Gauss-Legendre products over (ln l1, ln l2, phi);
        l1 and l2 belong to the two larger radii, so that l3 is not confined to a corner"""
        out = []
        xl, wl = (_dev(v) for v in np.polynomial.legendre.leggauss(64))
        xp, wp = (_dev(v) for v in np.polynomial.legendre.leggauss(40))
        u = lambda e: 0.5 * e * e * torch.exp(-0.5 * e * e)  # noqa: E731
        for th in np.sort(thetas, axis=1)[:, ::-1]:
            hi = math.log(10.0 / min(th))
            t, w = 0.5 * hi * (1 + xl), 0.5 * hi * wl
            p, v = 0.5 * math.pi * (1 + xp), math.pi * wp  # phi on (0, pi), twice
            l1, l2, ph = torch.meshgrid(torch.exp(t), torch.exp(t), p, indexing="ij")
            l3 = torch.sqrt((l1 - l2) ** 2 + 4 * l1 * l2 * torch.cos(0.5 * ph) ** 2)
            wt = (l1 * l2) ** 2 * w[:, None, None] * w[None, :, None] * v[None, None, :]
            wt = (wt * u(l1 * th[0]) * u(l2 * th[1]) * u(l3 * th[2])).reshape(-1)
            keep = wt > 1e-14 * wt.max()
            l = torch.stack([l1.reshape(-1), l2.reshape(-1), l3.reshape(-1)], 1)[keep]
            out.append(float((wt[keep] * self.bkappa(l)).sum() / (2 * math.pi) ** 3))
        return out


def _exact_apm(case, seed):
    x, y, g = _catalogue(case, seed)
    n, thetas = case["npix"], _apertures(case)
    cell = FIELD / (n - 1)
    edges = _dev(np.arange(n + 1) / (n - 1) * FIELD)
    x, y, g1, g2 = _dev(x), _dev(y), _dev(g.real), _dev(g.imag)

    def bins(v):
        b = torch.searchsorted(edges, v, right=True) - 1
        b = torch.where(v == edges[-1], torch.full_like(b, n - 1), b)
        return b, (v >= edges[0]) & (v <= edges[-1])

    dx, dy = torch.frac(x / cell), torch.frac(y / cell)
    grids = torch.zeros((3, n * n), dtype=torch.float64, device="cuda")
    for ox, wx in ((0.0, 1 - dx), (cell, dx)):
        bx, okx = bins(x + ox)
        for oy, wy in ((0.0, 1 - dy), (cell, dy)):
            by, oky = bins(y + oy)
            ok = okx & oky
            w, at = (wx * wy)[ok], (bx * n + by)[ok]
            for q, v in enumerate((g1[ok] * w, g2[ok] * w, w)):
                grids[q].scatter_add_(0, at, v)
    F = 2 * n
    spec = [torch.fft.rfft2(q.reshape(n, n), s=(F, F)) for q in grids]
    i = torch.arange(n, dtype=torch.float64, device="cuda") - n / 2
    zr, zi = torch.meshgrid(i, i, indexing="ij")
    z2 = zr * zr + zi * zi
    off = (n - 1) // 2
    maps = []
    for th in thetas:
        t2 = z2 * (FIELD / n / th) ** 2
        Q = t2 / (4 * math.pi * th * th) * torch.exp(-t2 / 2)
        inv = torch.where(z2 > 0, 1 / torch.clamp(z2, min=1e-300), torch.zeros_like(z2))
        re, im = Q * (zr * zr - zi * zi) * inv, Q * (-2 * zr * zi) * inv
        conv = lambda s, q: s * torch.fft.rfft2(q, s=(F, F))  # noqa: E731
        num = torch.fft.irfft2(conv(spec[1], im) - conv(spec[0], re), s=(F, F))
        den = torch.fft.irfft2(conv(spec[2], torch.sqrt(re * re + im * im)), s=(F, F))
        maps.append((num / den)[off:off + n, off:off + n].clone())
        del num, den
    cut = int(np.round(max(thetas) / FIELD * n * 4.0))
    m = [v[cut:n - cut, cut:n - cut] for v in maps]
    T = len(thetas)
    return np.array([float((m[a] * m[b] * m[c]).mean()) for a in range(T) for b in range(a, T) for c in range(b, T)])


def _exact_train(case, seed):
    params, xs, ts = _network(case, seed)
    # the masters are FP32 numbers; the network in 64 bits, without the BF16 rounding of the operands
    ps = [torch.tensor(np.asarray(p, dtype=np.float32).astype(np.float64), device="cuda", requires_grad=True)
          for W, b in params for p in (W, b)]
    mom = [(torch.zeros_like(p), torch.zeros_like(p)) for p in ps]
    losses = []
    for i in range(case["steps"]):
        h = xs[i].double()
        for l in range(5):
            h = h @ ps[2 * l].T + ps[2 * l + 1]
            if l < 4:
                h = torch.nn.functional.silu(h)
        loss = ((h[:, 0] - ts[i].double()) ** 2).mean()
        grads = torch.autograd.grad(loss, ps)
        losses.append(float(loss.detach()))
        with torch.no_grad():
            for p, g, (m, v) in zip(ps, grads, mom):
                m.mul_(0.9).add_(g, alpha=0.1)
                v.mul_(0.999).addcmul_(g, g, value=0.001)
                p -= LR * (m / (1 - 0.9 ** (i + 1))) / (torch.sqrt(v / (1 - 0.999 ** (i + 1))) + 1e-8)
    flat = torch.cat([p.detach().reshape(-1) for p in ps]).cpu().numpy()
    return flat, np.array(losses)


def exact(case, seed):
    kind = case["kind"]
    if kind == "chi2":
        data, cov, models = _vectors(case, seed)
        d = models - data
        return np.einsum("ij,ij->i", d, np.linalg.solve(cov, d.T).T)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "apm":
        return _exact_apm(case, seed)
    if kind == "bkappa":
        m = _Model(_cosmologies(1, seed)[0], _nz())
        return m.bkappa(_dev(sample_triangles(np.random.default_rng(seed), case["points"]))).cpu().numpy()
    if kind == "map3" and case["cosmologies"] * len(_radii(case)) <= 60:
        nz = _nz()
        return np.array([_Model(c, nz).map3(_radii(case)) for c in _cosmologies(case["cosmologies"], seed)])
    # the larger batches, the 3-D Hankel sums of gamma and the products of 2-D
    # to 7-D covariance integrals take longer than about 20 s this way
    return None
