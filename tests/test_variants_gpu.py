"""Forms of the kernels that only large or rare arguments reach: radstep's narrower blocks, the FP32 output transforms,
Legendre sums whose modes are staged in parts.

Tolerances, fixed beforehand.  Radiation FP64 1e-9 (the longwave effective emission divides by the logarithm of a
transmissivity clamped at 1 - 1e-6, which amplifies a few roundings of 1.1e-16 a million times).  FP32: shortwave 2e-3;
in the longwave that quotient is known to a few per cent only, so the median column is held, to 1e-4 (1e-5 at 20 levels,
and up to three times as many terms a sum).  FP32 output transforms 2e-5 against FP64, the bar of the FP32 sets.  The
Legendre functions by a recurrence of 534 steps in each direction, whose factors are rounded differently from the
library's: 1e-10; sets against their parts, the same sums, 1e-12."""
import ctypes as C

import numpy as np
import pytest
import torch

from exoplasim_b200 import radiation as R
from exoplasim_b200 import synthetic as S
from exoplasim_b200._lib import FP32, FP64, call
from exoplasim_b200.transforms import EZ, Plan, _ptr, _stream, fc2gp
from tests._util import relerr

pytestmark = pytest.mark.gpu


def _one_latitude(nlev, ncol, seed):
    cols, _ = S.radiation_columns(8, nlev, seed=seed)
    pick = np.random.default_rng(seed).permutation(cols["dp"].shape[0])[:ncol]
    return {k: v if k in ("sid", "cola") else np.ascontiguousarray(v[pick] if k == "dsalb" else v[..., pick])
            for k, v in cols.items()}


# FP64 blocks have 16 columns to 33 levels, 8 to 55, then 4; FP32 ones 16 to 34, 8 to 56
@pytest.mark.parametrize("nlev,prec", [(33, "fp64"), (34, "fp64"), (55, "fp64"), (56, "fp64"), (64, "fp64"), (34, "fp32"),
                                       (35, "fp32"), (56, "fp32"), (57, "fp32"), (64, "fp32")])
@pytest.mark.parametrize("ncol", [13, 17])
def test_radstep_many_levels(oracle, nlev, prec, ncol):
    cols = _one_latitude(nlev, ncol, nlev)
    params = R.default_params(nlev, ncol, ncol, nsol=0)
    sig = [np.array(getattr(params, k)[:nlev]) for k in ("sigma", "sigmah", "dsigma")]
    ref = oracle.radstep(oracle.radpar(nlev, ncol, ncol, *sig, nsol=0), cols["sid"], cols["cola"],
                         {k: v.copy() for k, v in cols.items()})
    dt = torch.float64 if prec == "fp64" else torch.float32

    def run(order):
        dev = {k: torch.as_tensor(np.ascontiguousarray(v if k in ("sid", "cola") else v[order] if k == "dsalb" else v[..., order]),
                                  dtype=dt, device="cuda") for k, v in cols.items()}
        return R.radstep(params, dev, precision=prec)

    out = run(np.arange(ncol))
    turned = run(np.arange(ncol)[::-1])
    for k in ("dfu", "dfd", "dftu", "dftd", "dswfl", "dlwfl", "dflux", "dtdtswr", "dtdtlwr"):
        assert torch.equal(out[k], turned[k].flip(-1)), k      # a column's place in its block changes nothing
        got = out[k].double().cpu().numpy()
        if prec == "fp64":
            assert relerr(got, ref[k]) < 1e-9, k
        elif k in ("dfu", "dfd", "dswfl", "dtdtswr"):
            assert relerr(got, ref[k]) < 2e-3, k
        else:
            assert np.median(np.max(np.abs(got - ref[k]), axis=0)) < 1e-4 * np.max(np.abs(ref[k])), k


@pytest.mark.parametrize("nlat,nlev", [(32, 1), (48, 3), (96, 7), (160, 2)])
@pytest.mark.parametrize("roll", [0, 1])
def test_output_transforms_in_fp32(nlat, nlev, roll):
    p = Plan(nlat, pyfft_nfs=0, plavor=0.0)
    g = torch.Generator(device="cuda").manual_seed(nlat)
    a, b = (torch.randn((nlev, p.nrsp), generator=g, device="cuda", dtype=torch.float64).float() for _ in range(2))
    rows = torch.rand(nlat, generator=g, device="cuda", dtype=torch.float64) + 0.5
    got = {}
    for prec, dt in ((FP64, torch.float64), (FP32, torch.float32)):
        x, y = a.to(dt), b.to(dt)
        work = torch.empty(2 * nlev * nlat * (p.ntru + 1) * 2, dtype=dt, device="cuda")
        t, u, v = (torch.zeros((nlev, nlat, 2 * nlat), dtype=dt, device="cuda") for _ in range(3))
        call("exotx_sp2gp_scaled", p._h, prec, _ptr(x), _ptr(t), nlev, C.c_double(1.5), roll, _ptr(work), _stream())
        call("exotx_dv2gp_scaled", p._h, prec, _ptr(x), _ptr(y), _ptr(u), _ptr(v), nlev, _ptr(rows), C.c_double(1.5), roll,
             _ptr(work), _stream())
        back, keep = torch.zeros_like(x), t.clone()
        call("exotx_gp2sp_scaled", p._h, prec, _ptr(t), _ptr(back), nlev, C.c_double(0.7), _ptr(work), _stream())
        assert torch.equal(t, keep)
        got[prec] = [z.double().cpu().numpy() for z in (t, u, v, back)]
    for x, y in zip(got[FP32], got[FP64]):
        for f in range(nlev):
            assert relerr(x[f], y[f]) < 2e-5


@pytest.fixture(scope="module")
def t533():
    return Plan(800)


def _functions(p, m):
    """P and (1 - mu^2) dP/dmu of wavenumber m, (modes, lat), by the recurrence in n."""
    mu, _ = p.gauss()
    c = np.sqrt(1.0 - mu * mu)
    cur = np.full(p.nlat, np.sqrt(0.5))
    for k in range(1, m + 1):
        cur = -cur * c * np.sqrt((2 * k + 1) / (2.0 * k))
    eps = lambda n: np.sqrt((n * n - m * m) / (4.0 * n * n - 1.0))  # noqa: E731
    prev, P, Q = np.zeros(p.nlat), [], []
    for n in range(m, p.ntru + 1):
        e = eps(n) if n else 0.0
        P.append(cur)
        Q.append((2 * n + 1) * e * prev - n * mu * cur)
        prev, cur = cur, (mu * cur - e * prev) / eps(n + 1)
    return np.array(P), np.array(Q)


# 534 wavenumbers: the modes of the wind transforms are staged 256 at a time
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 2e-5)])
def test_modes_staged_in_parts(t533, prec, tol):
    p, dt = t533, torch.float64 if prec == "fp64" else torch.float32
    rng = np.random.default_rng(1)
    n = np.arange(p.ntru + 1)
    d, z = (torch.zeros((1, p.nrsp), dtype=dt, device="cuda") for _ in range(2))
    first = lambda m: m * (p.ntru + 1) - m * (m - 1) // 2  # noqa: E731
    want = {}
    for m in (0, 3, 277):
        k = p.ntru + 1 - m
        x = rng.standard_normal((2, k, 2)).astype(np.float32).astype(np.float64) / (1.0 + n[m:, None] * (n[m:, None] + 1))
        if m == 0:
            x[..., 1] = 0.0
        x = torch.as_tensor(x, dtype=dt)
        for t, v in ((d, x[0]), (z, x[1])):
            t[0, 2 * first(m):2 * (first(m) + k)] = v.reshape(-1).cuda()
        D, Z = (x.double().numpy()[..., 0] + 1j * x.double().numpy()[..., 1])
        if m == 0:
            Z = Z.copy()
            Z[1] -= EZ
        P, Q = _functions(p, m)
        nn1 = np.where(n[m:] > 0, 1.0 / np.maximum(n[m:] * (n[m:] + 1), 1), 0.0)[:, None]
        qu, qv = P * nn1 * m, Q * nn1
        want[m] = (Z @ qv - 1j * (D @ qu), -1j * (Z @ qu) - D @ qv, D @ P)
    u, v = p.dv2uv(d, z, prec)
    t = p.sp2fc(d, prec)
    for m, ref in want.items():
        for got, r in zip((u, v, t), ref):
            g = got[0].double().cpu().numpy()[:, 2 * m] + 1j * got[0].double().cpu().numpy()[:, 2 * m + 1]
            assert np.max(np.abs(g - r)) < tol * np.max(np.abs(r)), m
    sp = torch.cat([d, d, z, d, d]).contiguous()        # sd st sz sq sp of one level
    g = p.inverse_set(sp, 1, prec)
    for f, part in ((0, u), (1, v), (2, t)):
        fc2gp(part)
        assert relerr(g[f].double().cpu().numpy(), part[0].double().cpu().numpy()) < (1e-12 if prec == "fp64" else tol)
