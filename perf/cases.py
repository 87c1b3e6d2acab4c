"""The work that this library is timed on, through its public entry points.

Seven kinds of case:

  sets       the spectral transforms of one model time step for `ninst` states
             (Plan.inverse_set_batch, forward_set_batch and their gridpointd
             forms): the transform core that runs on every dynamics step
  ensemble   the round trip of an uneven ensemble (ensemble.Ensemble)
  output     an output file's variables brought to the grid and back
             (postprocess.transformvar / transformvectorvar, float64)
  gridpoint  the grid-point step between the two transform sets
  radiation  the longwave and shortwave column pass (radiation.radstep)
  surrogate  the packaged network in radstep's place (surrogate.surrogate_step)
  training   one optimiser step of such a network (Mlp.backward, Mlp.adam)

Spectral coefficients fall off as 1/(n(n+1)) and grid tendencies are
N(0, 1e-5^2), as in exoplasim_b200.synthetic; radiation columns are drawn by
synthetic.radiation_columns.  exact() restates each kind in float64 torch.
"""
import functools
import math

import numpy as np
import torch

from exoplasim_b200 import ensemble, gridpoint, postprocess, radiation, surrogate, synthetic
from exoplasim_b200.transforms import EZ, Plan

NLATS = (32, 64, 96, 128, 160, 192, 256)  # T21, T42, T63, T85, T106, T127, T170
ESIZE = {"fp64": 8, "fp32": 4, "mixed": 4}
RADIUS = 6371220.0


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the model's default resolution and 8-byte reals, one state: the smallest call, bound by latency
        dict(name="sets_t21_l10_fp64", kind="sets", nlat=32, nlev=10, ninst=1, precision="fp64"),
        # T42 L20 with 8-byte reals: the usual higher resolution of an 8-byte model
        dict(name="sets_t42_l20_fp64", kind="sets", nlat=64, nlev=20, ninst=1, precision="fp64"),
        # a 4-byte model at T85 with an odd level count, three states
        dict(name="sets_t85_l13_x3_fp32", kind="sets", nlat=128, nlev=13, ninst=3, precision="fp32"),
        # one T42 L20 state on the tensor-core path: launch-bound
        dict(name="sets_t42_l20_mixed", kind="sets", nlat=64, nlev=20, ninst=1, precision="mixed"),
        # eight T127 L20 states on the tensor-core path: the throughput configuration
        dict(name="sets_t127_l20_x8_mixed", kind="sets", nlat=192, nlev=20, ninst=8, precision="mixed"),
        # the largest resolution, where the tensor-core kernels change variant
        dict(name="sets_t170_l25_mixed", kind="sets", nlat=256, nlev=25, ninst=1, precision="mixed"),
        # 96 states of T21, T42 and T63 with 10, 15 and 20 levels: a parameter sweep in one program
        dict(name="ensemble_96", kind="ensemble", ninst=96, pick=0),
        # a year of monthly T42 L10 output: temperature to the grid, winds from divergence and vorticity,
        # and a grid variable to spectral modes
        dict(name="output_t42_l10", kind="output", nlat=64, nlev=10, ntimes=12),
        # the grid-point step of eight T127 L20 states
        dict(name="gridpoint_t127_l20_x8_fp32", kind="gridpoint", nlat=192, nlev=20, ninst=8, precision="fp32"),
        # the radiation pass of a T42 L20 model with 8-byte reals (8192 columns)
        dict(name="radiation_t42_l20_fp64", kind="radiation", nlat=64, nlev=20, precision="fp64"),
        # the network in place of that pass
        dict(name="surrogate_t42_l20", kind="surrogate", nlat=64, precision="fp64"),
        # one step of training it, at the default batch
        dict(name="training_l20_b4096", kind="training", nlev=20, batch=4096),
    ]


def draw(rng):
    """One more case of the listed kinds: resolutions, level counts (odd ones among them), batches and precisions."""
    kind = rng.choice(("sets",) * 6 + ("ensemble", "output", "gridpoint", "radiation", "surrogate", "training"))
    top = _cost(listed()[4])
    while True:
        c = dict(kind=kind)
        if kind == "sets":
            c.update(nlat=rng.choice(NLATS), nlev=rng.randint(5, 25), ninst=_log(rng, 1, 9),
                     precision=rng.choice(("fp64", "fp32", "mixed", "mixed")))
        elif kind == "ensemble":
            c.update(ninst=_log(rng, 12, 110), pick=rng.randint(1, 999))
        elif kind == "output":
            c.update(nlat=rng.choice(NLATS[:6]), nlev=rng.randint(5, 20), ntimes=_log(rng, 1, 24))
        elif kind == "gridpoint":
            c.update(nlat=rng.choice(NLATS), nlev=rng.randint(5, 25), ninst=_log(rng, 1, 9),
                     precision=rng.choice(("fp32", "fp32", "fp64")))
        elif kind == "radiation":
            c.update(nlat=rng.choice((32, 48, 64, 96)), nlev=rng.randint(5, 25), precision=rng.choice(("fp64", "fp32")))
        elif kind == "surrogate":
            c.update(nlat=rng.choice((32, 40, 48, 64, 80, 96, 128)), precision=rng.choice(("fp64", "fp32")))
        else:
            c.update(nlev=rng.randint(5, 23), batch=_log(rng, 300, 6000))
        if _cost(c) <= top:
            return c


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _cost(c):
    w = work(c)
    # float64 and float32 contractions run at a few per cent of the tensor cores' rate
    slow = 12.0 if c.get("precision") in ("fp64", "fp32") or c["kind"] == "output" else 1.0
    return max(w["bytes"], w["flops"] * slow / 50.0)


# --------------------------------------------------------------- preparations
def _dims(nlat):
    ntru = (2 * nlat - 1) // 3
    return 2 * nlat, ntru, (ntru + 1) * (ntru + 2)  # NLON, NTRU, NRSP


@functools.lru_cache(maxsize=8)
def _plan(nlat):
    """A program keeps one plan per resolution."""
    return Plan(nlat)


@functools.lru_cache(maxsize=2)
def _ensemble(ninst, pick):
    return ensemble.Ensemble(*ensemble.draw(ninst, seed=pick))


@functools.lru_cache(maxsize=1)
def _network():
    return surrogate.Mlp.load(surrogate.DEFAULT_NET)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _spectra(gen, nlat, nlev, ninst, dtype):
    """(ninst, 4L+1, NRSP) states: sd, st, sz, sq, sp."""
    _, ntru, nrsp = _dims(nlat)
    m, n = synthetic.mode_mn(ntru)
    amp = torch.as_tensor(np.repeat(synthetic.amplitude(n), 2), device="cuda")
    amp[1::2][torch.as_tensor(m == 0, device="cuda")] = 0.0
    x = torch.randn((ninst, 4 * nlev + 1, nrsp), generator=gen, device="cuda", dtype=torch.float64) * amp
    x[:, 3 * nlev:4 * nlev] *= amp.sqrt()
    x[:, 2 * nlev:3 * nlev, 2] += EZ
    x[:, 4 * nlev, 0] = math.log(1.0e5)
    return x.to(dtype)


def _columns(nlat, nlev, seed, dtype, teff=True):
    cols, g = synthetic.radiation_columns(nlat, nlev, seed=int(seed), teff=teff)
    zsol = surrogate.zsol_for(cols.pop("teff"))
    dev = {k: torch.as_tensor(np.ascontiguousarray(v), dtype=dtype, device="cuda") for k, v in cols.items()}
    dev["zsol"] = torch.as_tensor(np.ascontiguousarray(zsol), dtype=dtype, device="cuda")
    return dev, g


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    dtype = torch.float64 if case.get("precision") == "fp64" else torch.float32
    s = dict(kind=kind)
    if kind == "sets":
        nlat, L, ninst, prec = case["nlat"], case["nlev"], case["ninst"], case["precision"]
        p = _plan(nlat)
        grid = lambda n, f: f((ninst, n, nlat, 2 * nlat), device="cuda", dtype=dtype)  # noqa: E731
        noise = lambda *a, **k: torch.randn(*a, generator=gen, **k) * 1e-5  # noqa: E731
        s.update(plan=p, nlev=L, precision=prec, sp=_spectra(gen, nlat, L, ninst, dtype),
                 ta=grid(9 * L + 1, noise), td=grid(4 * L, noise),
                 ga=grid(6 * L + 3, torch.zeros), gd=grid(4 * L + 1, torch.zeros),
                 sa=torch.zeros((ninst, 4 * L + 1, p.nrsp), device="cuda", dtype=dtype),
                 sd=torch.zeros((ninst, 4 * L, p.nrsp), device="cuda", dtype=dtype))
    elif kind == "ensemble":
        e = _ensemble(case["ninst"], case["pick"])
        spin, gout, gin, spout = e.buffers()
        for i in range(len(e.nlat)):
            n = (4 * e.nlev[i] + 1) * e.dims(i)[2]
            spin[int(e.spec_off[i]):][:n] = _spectra(gen, e.nlat[i], e.nlev[i], 1, torch.float32).reshape(-1)
        gin.copy_(torch.randn(gin.shape, generator=gen, device="cuda") * 1e-5)
        s.update(ens=e, spin=spin, gout=gout, gin=gin, spout=spout)
    elif kind == "output":
        nlat, L, nt = case["nlat"], case["nlev"], case["ntimes"]
        x = _spectra(gen, nlat, L, nt, torch.float64)
        lats = np.degrees(np.arcsin(_gauss(nlat)[0]))
        # relative vorticity, as an output file holds it
        zeta = x[:, 2 * L:3 * L].contiguous()
        zeta[..., 2] -= EZ
        s.update(nlat=nlat, nlev=L, lats=lats, temp=x[:, L:2 * L].contiguous(), div=x[:, :L].contiguous(), zeta=zeta,
                 cloud=torch.rand((nt, L, nlat, 2 * nlat), generator=gen, device="cuda", dtype=torch.float64))
    elif kind == "gridpoint":
        nlat, L, ninst = case["nlat"], case["nlev"], case["ninst"]
        const = gridpoint.GpConst(gridpoint.default_params(L))
        g = torch.randn((ninst, 6 * L + 3, nlat, 2 * nlat), generator=gen, device="cuda", dtype=dtype)
        sid = torch.as_tensor(_gauss(nlat)[0], device="cuda", dtype=dtype)[:, None]
        g[:, :2 * L] *= 0.03 * torch.sqrt(1 - sid ** 2)         # u, v times cos(lat), in units of the planet's rotation
        g[:, 2 * L:3 * L] *= 0.02                               # temperature about its reference profile
        g[:, 3 * L:4 * L] *= 0.01                               # divergence
        g[:, 4 * L:5 * L] = 0.1 * g[:, 4 * L:5 * L] + 2 * sid   # absolute vorticity
        g[:, 5 * L:6 * L] = g[:, 5 * L:6 * L].abs() * 0.005     # humidity times surface pressure
        g[:, 6 * L:6 * L + 2] *= 0.01                           # gradient of ln(ps)
        g[:, 6 * L + 2] *= 0.02                                 # ln(ps)
        out = torch.zeros((ninst, 9 * L + 1, nlat, 2 * nlat), device="cuda", dtype=dtype)
        s.update(plan=_plan(nlat), const=const, gin=g, gout=out)
    elif kind == "radiation":
        nlat, L = case["nlat"], case["nlev"]
        cols, g = _columns(nlat, L, seed, dtype)
        r = np.random.default_rng(seed)
        land = r.random(g["nhor"]) < 0.3
        cols["dls"] = torch.as_tensor(land.astype(np.float64), dtype=dtype, device="cuda")
        cols["dicec"] = torch.as_tensor(np.where(land, 0.0, np.maximum(0.0, r.uniform(-2.0, 1.0, g["nhor"]))),
                                        dtype=dtype, device="cuda")
        par = radiation.default_params(L, g["nhor"], g["nlon"], nsol=0)
        s.update(params=par, cols=cols, out=radiation.alloc_outputs(par, dtype), precision=case["precision"])
    elif kind == "surrogate":
        cols, g = _columns(case["nlat"], 20, seed, dtype)
        par = radiation.default_params(20, g["nhor"], g["nlon"], nsol=0)
        s.update(params=par, cols=cols, out=radiation.alloc_outputs(par, dtype), precision=case["precision"],
                 net=_network())
    else:
        L, n = case["nlev"], case["batch"]
        net = surrogate.Mlp(surrogate.nin_for(L), surrogate.nout_for(L), max_batch=n)
        net.init(seed)
        net.grads.owner = net.params.owner = net  # views of the network's own memory: whoever holds one keeps the network
        s.update(net=net, step=0, loss=torch.zeros(1, device="cuda"),
                 x=torch.randn((n, net.nin), generator=gen, device="cuda"),
                 t=torch.randn((n, net.nout), generator=gen, device="cuda"))
    return s


def run(s):
    kind = s["kind"]
    if kind == "sets":
        p, L, prec = s["plan"], s["nlev"], s["precision"]
        p.inverse_set_batch(s["sp"], L, prec, s["ga"])
        p.forward_set_batch(s["ta"], L, prec, s["sa"])
        p.inverse_set_d_batch(s["sp"], L, prec, s["gd"])
        p.forward_set_d_batch(s["td"], L, prec, s["sd"])
        return s["ga"], s["sa"], s["gd"], s["sd"]
    if kind == "ensemble":
        return s["ens"].inverse(s["spin"], s["gout"]), s["ens"].forward(s["gin"], s["spout"])
    if kind == "output":
        nlat, L = s["nlat"], s["nlev"]
        nlon, ntru, _ = _dims(nlat)
        temp = postprocess.transformvar(s["temp"], nlat, nlon, L, ntru, mode="grid")
        u, v = postprocess.transformvectorvar(s["div"], s["zeta"], s["lats"], nlon, L, ntru, radius=RADIUS)
        cloud = postprocess.transformvar(s["cloud"], nlat, nlon, L, ntru, mode="spectral")
        return temp, u, v, cloud
    if kind == "gridpoint":
        return gridpoint.gridpoint(s["plan"], s["const"], s["gin"], s["gout"])
    if kind == "radiation":
        out = radiation.radstep(s["params"], s["cols"], s["out"], s["precision"])
        return dict(out, **{k: s["cols"][k] for k in ("dqo3", "dalb", "dsalb", "dtdt")})
    if kind == "surrogate":
        surrogate.surrogate_step(s["net"], s["params"], s["cols"], s["out"], s["precision"])
        return dict(s["out"], dtdt=s["cols"]["dtdt"])
    s["step"] += 1
    s["loss"].zero_()
    s["net"].backward(s["x"], s["t"], s["loss"])
    s["net"].adam(1e-4, s["step"])
    return s["loss"], s["net"].grads, s["net"].params


def work(c):
    """Each input read once and each output written once; products of the folded Legendre sums and the FFTs."""
    kind = c["kind"]

    def legendre(nlat, nprod):  # nprod complex fields times one table each
        return 2.0 * nlat * (_dims(nlat)[2] / 2) * nprod

    def fft(nlat, nfld):
        return nfld * nlat * 2.5 * 2 * nlat * math.log2(2 * nlat)

    def round_trip(nlat, L):
        nhor, nrsp = 2 * nlat * nlat, _dims(nlat)[2]
        return 2 * (4 * L + 1) * nrsp + (15 * L + 4) * nhor, legendre(nlat, 19 * L + 3) + fft(nlat, 15 * L + 4)

    if kind == "sets":
        nlat, L, n = c["nlat"], c["nlev"], c["ninst"]
        v, f = round_trip(nlat, L)
        v += (8 * L + 1) * (_dims(nlat)[2] + 2 * nlat * nlat)
        f += legendre(nlat, 12 * L + 1) + fft(nlat, 8 * L + 1)
        return {"bytes": float(n * v * ESIZE[c["precision"]]), "flops": float(n * f)}
    if kind == "ensemble":
        w = [round_trip(a, b) for a, b in zip(*ensemble.draw(c["ninst"], seed=c["pick"]))]
        return {"bytes": 4.0 * sum(v for v, _ in w), "flops": float(sum(f for _, f in w))}
    if kind == "output":
        nlat, n = c["nlat"], c["nlev"] * c["ntimes"]
        return {"bytes": 8.0 * n * (4 * _dims(nlat)[2] + 4 * 2 * nlat * nlat),
                "flops": float(n * (legendre(nlat, 6) + fft(nlat, 4)))}
    if kind == "gridpoint":
        ncol, L = c["ninst"] * 2 * c["nlat"] ** 2, c["nlev"]
        return {"bytes": float(ncol * (15 * L + 4) * ESIZE[c["precision"]]), "flops": float(ncol * (3 * L * L + 60 * L))}
    if kind == "radiation":
        ncol, L = 2 * c["nlat"] ** 2, c["nlev"]
        # about 20 columns of L read and written; four absorptivities (a power or a logarithm, about 20 operations) per pair
        return {"bytes": float(ncol * (18 * L + 21) * ESIZE[c["precision"]]), "flops": float(ncol * (40 * L * (L + 1) + 900 * L))}
    if kind == "surrogate":
        ncol = 2 * c["nlat"] ** 2
        return {"bytes": float(ncol * (69 + 2 * 20 + 6) * ESIZE[c["precision"]]), "flops": float(ncol * 2 * _weights(20))}
    n, L = c["batch"], c["nlev"]
    return {"bytes": 4.0 * (n * (4 * L + 13) + 8 * _weights(L)), "flops": 6.0 * n * _weights(L)}


def _weights(L):
    return (3 * L + 9) * 256 + 5 * 256 * 256 + 256 * (L + 4)


# -------------------------------------------------------- in 64 bits, by torch
@functools.lru_cache(maxsize=8)
def _gauss(nlat):
    """sin(lat), north first, and weights of the Gaussian grid."""
    x, w = np.polynomial.legendre.leggauss(nlat)
    return x[::-1].copy(), w[::-1].copy()


@functools.lru_cache(maxsize=2)
def _tables(nlat):
    """Associated Legendre functions P(mode, lat) with unit norm and (1 - mu^2) dP/dmu, modes m-major; m, n of each mode."""
    _, ntru, _ = _dims(nlat)
    mu, _ = _gauss(nlat)
    c = np.sqrt(1.0 - mu * mu)
    ps, qs, ms, ns = [], [], [], []
    pmm = np.full(nlat, math.sqrt(0.5))
    for m in range(ntru + 1):
        if m:
            pmm = -pmm * c * math.sqrt((2 * m + 1) / (2.0 * m))
        eps = lambda n: math.sqrt((n * n - m * m) / (4.0 * n * n - 1.0))  # noqa: B023, E731
        prev, cur = np.zeros(nlat), pmm
        for n in range(m, ntru + 1):
            e = eps(n) if n else 0.0
            ps.append(cur)
            qs.append((2 * n + 1) * e * prev - n * mu * cur)
            ms.append(m)
            ns.append(n)
            prev, cur = cur, (mu * cur - e * prev) / eps(n + 1)
    f = lambda a: torch.as_tensor(np.array(a), dtype=torch.float64, device="cuda")  # noqa: E731
    return f(ps), f(qs), f(ms), f(ns)


def _synth(table, spec):
    """sum over n of table * complex coefficients: (..., modes) -> (..., nlat, NTRU+1)."""
    nlat = table.shape[1]
    ntru = _dims(nlat)[1]
    out, w = [], 0
    for m in range(ntru + 1):
        k = ntru + 1 - m
        out.append(spec[..., w:w + k] @ table[w:w + k].to(spec.dtype))
        w += k
    return torch.stack(out, -1)


def _analyse(table, four):
    """sum over lat of table * Fourier coefficients: (..., nlat, NTRU+1) -> (..., modes)."""
    ntru = _dims(table.shape[1])[1]
    out, w = [], 0
    for m in range(ntru + 1):
        k = ntru + 1 - m
        out.append(four[..., m] @ table[w:w + k].t().to(four.dtype))
        w += k
    return torch.cat(out, -1)


def _complex(x):
    return torch.view_as_complex(x.double().reshape(*x.shape[:-1], -1, 2).contiguous())


def _real(z):
    return torch.view_as_real(z).reshape(*z.shape[:-1], -1)


def _to_grid(four):
    nlon = 2 * four.shape[-2]
    return torch.fft.irfft(torch.nn.functional.pad(four, (0, nlon // 2 + 1 - four.shape[-1])), n=nlon) * nlon


def _to_four(grid):
    nlon = grid.shape[-1]
    return torch.fft.rfft(grid.double())[..., :_dims(grid.shape[-2])[1] + 1] / nlon


def _winds(nlat, d, z, plavor):
    P, Q, m, n = _tables(nlat)
    nn1 = torch.where(n > 0, 1.0 / (n * (n + 1)).clamp(min=1), torch.zeros_like(n))[:, None]
    qu, qv = P * nn1 * m[:, None], Q * nn1
    z = z.clone()
    z[..., 1] -= plavor
    return _synth(qv, z) - 1j * _synth(qu, d), -1j * _synth(qu, z) - _synth(qv, d)


def _exact_inverse(nlat, L, sp, dset):
    P, Q, _, _ = _tables(nlat)
    x = _complex(sp)
    d, t, z, q, lnp = x[:, :L], x[:, L:2 * L], x[:, 2 * L:3 * L], x[:, 3 * L:4 * L], x[:, 4 * L:]
    u, v = _winds(nlat, d, z, EZ)
    gp = _synth(P, lnp)
    if dset:
        f = [u, v, _synth(P, t), _synth(P, q), gp]
    else:
        im = 1j * torch.arange(gp.shape[-1], device="cuda")
        f = [u, v, _synth(P, t), _synth(P, d), _synth(P, z), _synth(P, q), _synth(Q, lnp), im * gp, gp]
    return _to_grid(torch.cat(f, 1))


def _exact_forward(nlat, L, grid, dset):
    P, Q, m, n = _tables(nlat)
    mu, w = (torch.as_tensor(a, device="cuda") for a in _gauss(nlat))
    wc = w / (1 - mu * mu)
    qc, qe, qm, qq = P * w, Q * wc, P * wc * m[:, None], P * wc * (n * (n + 1) / 2)[:, None]
    x = _to_four(grid)
    if dset:
        t, u, v, q = x[:, :L], x[:, L:2 * L], x[:, 2 * L:3 * L], x[:, 3 * L:]
        z = _analyse(qe, u) + 1j * _analyse(qm, v)
        d = 1j * _analyse(qm, u) - _analyse(qe, v)
        return _real(torch.cat([d, _analyse(qc, t), z, _analyse(qc, q)], 1))
    tn, qn, ut, vt, uz, vz, ke = (x[:, k * L:(k + 1) * L] for k in range(7))
    vpp, uq, vq = x[:, 7 * L:7 * L + 1], x[:, 7 * L + 1:8 * L + 1], x[:, 8 * L + 1:]
    d = _analyse(qq, ke) - _analyse(qe, uz) + 1j * _analyse(qm, vz)
    t = _analyse(qe, vt) + _analyse(qc, tn) - 1j * _analyse(qm, ut)
    z = _analyse(qe, vz) + 1j * _analyse(qm, uz)
    q = _analyse(qe, vq) + _analyse(qc, qn) - 1j * _analyse(qm, uq)
    return _real(torch.cat([d, t, z, q, _analyse(qc, vpp)], 1))


def _exact_gridpoint(nlat, p, gin):
    """calcgp and the flux products, one row of columns per level."""
    L = p.nlev
    f = lambda a, k=None: torch.as_tensor(np.array(a[:k or L]), device="cuda")  # noqa: E731
    ds, sh, rds, t0, t01, tkp = (f(a) for a in (p.dsigma, p.sigmah, p.rdsig, p.t0, p.t01s2, p.tkp))
    gm, cm = f(p.g, L * L).reshape(L, L), f(p.c, L * L).reshape(L, L)  # [k][i]: column k of g(i, k), c(i, k)
    x = gin.double()
    u, v, t, d, z, q = (x[:, k * L:(k + 1) * L] for k in range(6))
    pj, pm, gp = x[:, 6 * L, None], x[:, 6 * L + 1, None], x[:, 6 * L + 2, None].exp()
    rc = 1.0 / (1.0 - torch.as_tensor(_gauss(nlat)[0], device="cuda")[:, None] ** 2)
    e = lambda a: a[:, None, None]  # noqa: E731
    zv = rc * (u * pm + v * pj)
    zq = (q / gp).clamp(min=0)
    tv = (t + e(t0)) * (1 + (1 / p.rdbrv - 1) * zq)
    tv1, tv2 = tv - e(t0), tv / (1 + p.adv * zq) - e(t0)
    sd, sv = (d * e(ds)).cumsum(1), (zv * e(ds)).cumsum(1)
    vp = sv[:, -1:]
    dot = (e(sh) * (sd[:, -1:] + vp) - (sd + sv))[:, :-1]
    pad = lambda a: torch.nn.functional.pad(a, (0, 0, 0, 0, 1, 1))  # noqa: E731
    ft, fq, fu, fv = (pad(a) for a in (dot * (t[:, 1:] - t[:, :-1]), dot * (q[:, 1:] + q[:, :-1]),
                                       dot * (u[:, 1:] - u[:, :-1]), dot * (v[:, 1:] - v[:, :-1])))
    low = torch.tril(torch.ones(L, L, device="cuda", dtype=torch.float64))
    mix = lambda m, a: torch.einsum("kj,bjyx->bkyx", m, a)  # noqa: E731
    ta, tb = mix(cm * low, zv), mix(cm * low, zv + d)
    t01m, shm = torch.cat([t01[:1] * 0, t01[:-1]]), torch.cat([sh[:1] * 0, sh[:-1]])
    t01p = torch.cat([t01[:-1], t01[:1] * 0])
    adv = ft[:, 1:] + ft[:, :-1] + vp * e(t01p * sh + t01m * shm) - sv * e(t01m + t01p) + zv * e(ds * t01m)
    tn = t * d + p.akap * tv2 * (zv - tb) + e(tkp) * (zv - ta) - e(rds) * adv
    # the top level's form, and the bottom level's sum up to the level above
    tn[:, 0] = (t * d - p.akap * tv2 * d)[:, 0] - rds[0] * (ft[:, 1] + t01[0] * (sh[0] * vp[:, 0] - sv[:, 0]))
    k = L - 1
    tn[:, k] = (t * d + p.akap * tv2 * (zv - tb) + e(tkp) * (zv - ta))[:, k] \
        - rds[k] * (ft[:, k] + t01[k - 1] * (sh[k - 1] * vp[:, 0] - sv[:, k - 1]))
    qn = -e(rds) * (fq[:, 1:] - fq[:, :-1])
    uz = -u * z - pj * tv1 - e(rds) * (fv[:, 1:] + fv[:, :-1])
    vz = v * z - pm * tv1 - e(rds) * (fu[:, 1:] + fu[:, :-1])
    ke = u * u + v * v + mix(gm, tv1 - t) * 2 / rc
    return torch.cat([tn, qn, u * t, v * t, uz, vz, ke, vp, u * q, v * q], 1)


def _o3_absorbed(x):
    return 0.02118 * x / (1 + 0.042 * x + 0.000323 * x * x) + 1.082 * x / (1 + 138.6 * x) ** 0.805 \
        + 0.0658 * x / (1 + (103.6 * x) ** 3)


def _h2o_absorbed(y):
    return 2.9 * y / ((1 + 141.5 * y) ** 0.635 + 5.925 * y)


def _ozone(p, c, sid):
    """mko3: the ozone profile of each column, (L, n)."""
    L, zfo3 = p.nlev, 100.0 / 2.14
    za = p.a0o3 + p.a1o3 * sid.abs() + p.aco3 * sid * math.cos(2 * 3.14159265359 * (p.zcday - p.toffo3))
    left, h, out = za, torch.zeros_like(za), [None] * L
    for j in range(L - 1, 0, -1):
        h = h - c["dt"][j] * p.gascon / p.ga * math.log(p.sigmah[j - 1] / p.sigmah[j])
        o = -za * (1 + math.exp(-p.bo3 / p.co3)) / (1 + torch.exp((h - p.bo3) / p.co3)) + left
        out[j] = o * p.ga / (zfo3 * p.dsigma[j] * c["dp"])
        left = left - o
    out[0] = left * p.ga / (zfo3 * p.dsigma[0] * c["dp"])
    return torch.stack(out)


def _shortwave(p, c, o3):
    """swr with clouds on, Rayleigh scattering in the lowest layer and the ocean's zenith-dependent albedo."""
    L, ga = p.nlev, p.ga
    z1, z2, rco = c["zsol"]
    mu, dp, cc = c["gmu0"], c["dp"], c["dcc"]
    lit = (z1 + z2) * p.gsol0 * p.gdist2 * mu > 1e-6
    mu = torch.where(lit, mu, torch.ones_like(mu))
    f1, f2 = z1 * p.gsol0 * p.gdist2 * mu, z2 * p.gsol0 * p.gdist2 * mu
    one = torch.ones_like(mu)
    half = 0.5 * one
    # cloud optics and absorber paths, downwards
    optics, paths, clear, pclear = [], [], one, one
    o3t = xo3 = wvt = ywv = torch.zeros_like(mu)
    zm = 35 / torch.sqrt(1 + 1224 * mu * mu)
    for j in range(L):
        lwp = (1000 * c["dql"][j] * dp / ga * p.dsigma[j]).clamp(max=1000)
        tau = 2 * torch.log10(lwp + 1.5) ** 3.9
        zlog = torch.log(1000 / tau)

        def stream(m):
            b2 = p.tswr2 * torch.sqrt(m) / torch.log(3 + 0.1 * tau)  # noqa: B023
            om = (1 - p.tswr3 * m * m * zlog).clamp(max=0.9999)  # noqa: B023
            un = 1 - om
            uz = un + 2 * b2 * om
            w = torch.sqrt(uz / un)
            ex = torch.exp((tau * torch.sqrt(uz * un) / m).clamp(max=25))  # noqa: B023
            r = (w + 1) ** 2 * ex - (w - 1) ** 2 / ex
            r1 = 1 - 1 / (1 + p.tswr1 * torch.sqrt(m) * tau / m)  # noqa: B023
            return r1, 4 * w / r, (w * w - 1) / r * (ex - 1 / ex)

        some = cc[j] > 0
        diffuse = [torch.where(some, a, torch.full_like(a, b)) for a, b in zip(stream(half), (0.0, 1.0, 0.0))]
        direct = [torch.where(some, a, torch.full_like(a, b)) for a, b in zip(stream(mu), (0.0, 1.0, 0.0))]
        optics.append(([clear * a + (1 - clear) * b for a, b in zip(direct, diffuse)], diffuse))
        clear = clear * (1 - cc[j])
        o = 100 / 2.14 * p.dsigma[j] * dp * o3[j] / ga
        wv = 0.1 * p.dsigma[j] * c["dq"][j] * dp / ga * torch.sqrt(273 / c["dt"][j]) * p.sigma[j] * dp / 100000
        o3t, xo3 = o3t + o, xo3 + (pclear * zm + (1 - pclear) * 1.9) * o
        wvt, ywv = wvt + wv, ywv + (pclear * zm + (1 - pclear) * 1.66) * wv
        paths.append((o3t, xo3, wvt, ywv))
        pclear = pclear * (1 - cc[j])
    sc = rco * dp / 101100 * 9.80665 / ga
    ray_u = (1 - torch.exp(sc * math.log(1 - 0.144))) * (1 - cc[L - 1])
    ray = (1 - torch.exp(sc * torch.log(1 - 0.219 / (1 + 0.816 * mu)))) * pclear \
        + (1 - torch.exp(sc * math.log(1 - 0.144))) * (1 - pclear - cc[L - 1])
    # downward adding
    ta1 = ta1s = ta2 = ta2s = to3 = twv = one
    ra1s = ra2s = torch.zeros_like(mu)
    to3u, twvu = 1 - _o3_absorbed(xo3 + 1.9 * o3t) / z1, 1 - _h2o_absorbed(ywv + 1.66 * wvt) / z2
    layers, top = [], []
    for j in range(L):
        (r1, t2, r2), (r1s, t2s, r2s) = optics[j]
        a, xa, w, yw = paths[j]
        top.append((ta1, ta2, ra1s, ra2s))
        rb1 = r1 * cc[j] + (ray if j == L - 1 else 0)
        rb1s = r1s * cc[j] + (ray_u if j == L - 1 else 0)
        n = 1 - _o3_absorbed(xa) / z1
        tr, to3 = n / to3, n
        n = 1 - _o3_absorbed(xo3 + 1.9 * (o3t - a)) / z1
        tru, to3u = to3u / n, n
        tb1 = 1 - (1 - tr) * (1 - cc[j]) - rb1
        tb1u = 1 - (1 - tru) * (1 - cc[j]) - rb1s
        k = 1 / (1 - ra1s * rb1s)
        ta1, ra1s, ta1s = ta1 * tb1 * k, rb1s + tb1u * ra1s * tb1 * k, tb1u * ta1s * k
        rb2, rb2s = r2 * cc[j], r2s * cc[j]
        n = 1 - _h2o_absorbed(yw) / z2
        tr, twv = n / twv, n
        n = 1 - _h2o_absorbed(ywv + 1.66 * (wvt - w)) / z2
        tru, twvu = twvu / n, n
        tb2 = 1 - (1 - tr) * (1 - cc[j]) - (1 - t2) * cc[j]
        tb2u = 1 - (1 - tru) * (1 - cc[j]) - (1 - t2s) * cc[j]
        k = 1 / (1 - ra2s * rb2s)
        ta2, ra2s, ta2s = ta2 * tb2 * k, rb2s + tb2u * ra2s * tb2 * k, tb2u * ta2s * k
        layers.append((rb1, rb1s, tb1, tb1u, rb2, rb2s, tb2, tb2u))
    top.append((ta1, ta2, ra1s, ra2s))
    # the surface, and upward adding
    ls, ice = c["dls"], c["dicec"]
    wet = (1 - ls) * (1 - ice)
    ocean = (0.05 / (mu + 0.15)).clamp(max=0.15)
    dry = ls + (1 - ls) * ice
    alb = dry * c["dalb"] + wet * ocean
    sal = dry[:, None] * c["dsalb"] + (wet * ocean)[:, None]
    a1, a2, a1s, a2s = alb, alb, c["dalb"], c["dalb"]
    low = [None] * L + [(a1, a2, a1s, a2s)]
    for j in range(L - 1, -1, -1):
        rb1, rb1s, tb1, tb1u, rb2, rb2s, tb2, tb2u = layers[j]
        a1 = rb1 + tb1 * a1 * tb1u / (1 - a1s * rb1s)
        a1s = rb1s + tb1u * a1s * tb1u / (1 - a1s * rb1s)
        a2 = rb2 + tb2 * a2 * tb2u / (1 - a2s * rb2s)
        a2s = rb2s + tb2u * a2s * tb2u / (1 - a2s * rb2s)
        low[j] = (a1, a2, a1s, a2s)
    up, down = [], []
    for j in range(L + 1):
        t1, t2, r1, r2 = top[j]
        a1, a2, a1s, a2s = low[j]
        k1, k2 = 1 / (1 - r1 * a1s), 1 / (1 - r2 * a2s)
        up.append(-t1 * a1 * k1 * f1 - t2 * a2 * k2 * f2)
        down.append(t1 * k1 * f1 + t2 * k2 * f2)
    dark = lambda a: torch.where(lit, torch.stack(a), torch.zeros_like(mu))  # noqa: E731
    return dark(up), dark(down), torch.where(lit, alb, c["dalb"]), torch.where(lit[:, None], sal, c["dsalb"])


def _longwave(p, c, o3):
    """lwr: absorptivity fits of H2O, CO2 and O3, random-overlap clouds, effective layer emission."""
    L, ga, dp = p.nlev, p.ga, c["dp"]
    sig, sigh, dsig = (np.array(a[:L]) for a in (p.sigma, p.sigmah, p.dsigma))
    t2 = c["dt"] * c["dt"]
    st = 5.67e-8 * (t2 * t2)  # rounded as the reference rounds it: the branches below compare nearly equal values
    # by tensors: torch multiplies by the reciprocal of a plain number
    sf, sh_ = (torch.as_tensor(a, device="cuda")[:, None] for a in (sig, sigh))
    sh = (st[1:L] * (sf[:-1] - sh_[:-1]) + st[:L - 1] * (sh_[:-1] - sf[1:])) / (sf[:-1] - sf[1:])
    first = st[0] - (st[0] - st[1]) * sf[0] / (sf[0] - sf[1])
    warm = (st[L - 1] - sh[-1]) * (st[L - 1] - st[L]) > 0
    ground = st[L - 1] + (st[L - 1] - st[L - 2]) * (1 - sf[L - 1]) / (sf[L - 1] - sf[L - 2])
    sh = torch.cat([first[None], sh, torch.where(warm, st[L], ground)[None]])
    eps = c["dls"] + 0.98 * (1 - c["dls"])
    fac = torch.as_tensor(sig * dsig, device="cuda")[:, None] / ga / 1e5 * dp * dp
    q, qo3 = 0.1 * fac * c["dq"][:L], 100 / 2.14 * fac * o3
    qco2 = 100 / 1.9635 * (0.0440098 / 0.0289644 * 1e-6) * fac * c["dqco2"]
    cloud = 1 - c["dcc"][:L] * (1 - torch.exp(torch.as_tensor(-1.66 * p.acllwr * 1000 * dsig / ga, device="cuda")[:, None]
                                              * c["dql"][:L] * dp))
    o30, co20, h2oa, h2o0 = 0.209 * 7e-5 ** 0.436, 0.0676 * 0.01022 ** 0.421, 0.846 * 3.59e-5 ** 0.243, 0.832 * 0.0286 ** 0.26
    o3c = 0.209 * (0.01 + 7e-5) ** 0.436 - o30 - 0.0212 * math.log10(0.01)
    co2c = 0.0676 * 1.01022 ** 0.421 - co20
    h2oc = 0.846 * (0.01 + 3.59e-5) ** 0.243 - h2oa - 0.24 * math.log10(0.02)
    th2c = 1 - (0.832 * 2.0286 ** 0.26 - h2o0) + 0.1196 * math.log(2 - 0.6931)

    def trans(w, o, g):
        a = torch.where(w <= 0.01, 0.846 * (w + 3.59e-5) ** 0.243 - h2oa, 0.24 * torch.log10(w + 0.01) + h2oc)
        a = (a + 1 - torch.exp(-p.th2oc * w)).clamp(max=1)
        b = torch.where(g <= 1, 0.0676 * (g + 0.01022) ** 0.421 - co20, 0.0546 * torch.log10(g.clamp(min=1)) + co2c)
        t = torch.where(w <= 2, 1 - (0.832 * (w + 0.0286) ** 0.26 - h2o0),
                        (th2c - 0.1196 * torch.log(w.clamp(min=2) - 0.6931)).clamp(min=0))
        x = torch.where(o <= 0.01, 0.209 * (o + 7e-5) ** 0.436 - o30, 0.0212 * torch.log10(o.clamp(min=0.01)) + o3c)
        return (1 - a - x - b * t).clamp(1e-6, 1 - 1e-6)

    n = dp.shape[0]
    up, down = torch.zeros((L + 1, n), device="cuda", dtype=torch.float64), torch.zeros((L + 1, n), device="cuda", dtype=torch.float64)
    bd, bu = [torch.zeros_like(dp)], [None]
    last = []
    for j in range(L):
        clear = trans(q[j:].cumsum(0), qo3[j:].cumsum(0), qco2[j:].cumsum(0))
        tau = clear * cloud[j:].cumprod(0)
        if j == 0:
            before = torch.cat([torch.full_like(clear[:1], 1 - 1e-6), clear[:-1]])
            t0 = (clear / before * cloud * p.tpofmt).clamp(1e-6, 1 - 1e-6)
            for i in range(L):
                h0, h1 = sh[i], sh[i + 1]
                peak = (st[i] - h0) * (st[i] - h1) > 0
                mean = 0.5 * st[i] + 0.25 * (h0 + h1)
                b = (h1 - t0[i] * h0) / (1 - t0[i]) - (h0 - h1) / torch.log(t0[i])
                bd.append(torch.where(peak, mean, b))
                bu.append(torch.where(peak, mean, h0 + h1 - b))
            bu.append(eps * st[L])
        up[j] -= bu[j + 1]
        down[j] += bd[j]
        for i in range(j, L):
            up[j] -= (bu[i + 2] - bu[i + 1]) * tau[i - j]
            down[i + 1] += (bd[j] - bd[j + 1]) * tau[i - j]
        last.append(tau[-1])
    up[L] -= bu[L + 1]
    down[L] += bd[L]
    up[:L] -= torch.stack(last) * (1 - eps) * down[L]
    return up, down


def _exact_radiation(p, c):
    L = p.nlev
    c = {k: v.double() for k, v in c.items()}
    sid = c["sid"].repeat_interleave(p.nlon)
    o3 = _ozone(p, c, sid)
    fu, fd, alb, sal = _shortwave(p, c, o3)
    tu, td = _longwave(p, c, o3)
    sw, lw = fu + fd, tu + td
    f = lambda a: torch.as_tensor(np.array(a), device="cuda")[:, None]  # noqa: E731
    den = f(p.dsigma[:L]) * c["dp"] * p.acpd * (1 + p.adv * c["dq"][:L])
    rate = lambda a: -p.ga * (a[1:] - a[:-1]) / den  # noqa: E731
    thick = [0.5 * math.log(p.sigma[0] / p.sigmah[0])] + [math.log(p.sigmah[j - 1] / p.sigmah[j]) for j in range(1, L)]
    net = sw + lw
    dz = -c["dt"][:L] * p.gascon / p.ga * f(thick)
    return dict(dfu=fu, dfd=fd, dftu=tu, dftd=td, dswfl=sw, dlwfl=lw, dflux=net, dtdtswr=rate(sw), dtdtlwr=rate(lw),
                dconv=(net[:-1] - net[1:]) / (dz + 1e-9), dqo3=o3, dalb=alb, dsalb=sal, dtdt=c["dtdt"] + rate(net))


def _layers(params, nin, nout):
    """(W, b) of each layer of the packed parameters, in 64 bits."""
    dims, off, got = [nin] + [256] * 6 + [nout], 0, []
    for a, b in zip(dims[:-1], dims[1:]):
        got.append((params[off:off + a * b].reshape(b, a), params[off + a * b:off + a * b + b]))
        off += a * b + b
    return got


def _mlp(layers, x):
    for w, b in layers[:-1]:
        x = torch.nn.functional.silu(x @ w.t() + b)
    w, b = layers[-1]
    return x @ w.t() + b


def _exact_surrogate(net, p, c, out):
    L = p.nlev
    c = {k: v.double() for k, v in c.items()}
    f = [c["dt"][:L + 1], torch.log(c["dq"][:L + 1].clamp(min=1e-12)), c["dcc"][:L], torch.log(c["dp"])[None], c["dalb"][None],
         c["gmu0"][None], torch.log(c["dqco2"][:1]), c["zsol"][:1], c["zsol"][2:], c["sid"].repeat_interleave(p.nlon)[None]]
    n = {k: torch.as_tensor(v, device="cuda").double() for k, v in net.norm.items()}
    x = torch.cat(f).t()
    if bool(((x < n["xlo"]) | (x > n["xhi"])).any()):
        return None  # such columns are radstep's
    y = (_mlp(_layers(net.params.double(), net.nin, net.nout), (x - n["xm"]) / n["xs"]) * n["ys"] + n["ym"]).t()
    got = {k: v.double().clone() for k, v in out.items()}
    for k, r in (("dfd", L), ("dfu", L + 1), ("dftd", L + 2), ("dftu", L + 3)):
        got[k][L] = y[r]
    got["dswfl"][L], got["dlwfl"][L] = y[L] + y[L + 1], y[L + 2] + y[L + 3]
    return dict(got, dtdt=c["dtdt"] + y[:L] / (86400.0 * c["dp"] / 1e5 * (1 + p.adv * c["dq"][:L])))


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind == "sets":
        nlat, L = case["nlat"], case["nlev"]
        return (_exact_inverse(nlat, L, s["sp"], False), _exact_forward(nlat, L, s["ta"], False),
                _exact_inverse(nlat, L, s["sp"], True), _exact_forward(nlat, L, s["td"], True))
    if kind == "ensemble":
        e = s["ens"]
        grid, spec = torch.zeros(s["gout"].shape, device="cuda", dtype=torch.float64), torch.zeros(
            s["spout"].shape, device="cuda", dtype=torch.float64)
        for nlat in sorted(set(e.nlat)):
            for i in (i for i, a in enumerate(e.nlat) if a == nlat):
                L, nrsp = e.nlev[i], e.dims(i)[2]
                x = s["spin"][int(e.spec_off[i]):][:(4 * L + 1) * nrsp].reshape(1, -1, nrsp)
                g = s["gin"][int(e.gin_off[i]):][:(9 * L + 1) * 2 * nlat ** 2].reshape(1, -1, nlat, 2 * nlat)
                a, b = _exact_inverse(nlat, L, x, False).reshape(-1), _exact_forward(nlat, L, g, False).reshape(-1)
                grid[int(e.gout_off[i]):][:a.numel()] = a
                spec[int(e.spec_off[i]):][:b.numel()] = b
        return grid, spec
    if kind == "output":
        nlat, nlon = case["nlat"], 2 * case["nlat"]
        P, _, _, _ = _tables(nlat)
        _, w = _gauss(nlat)
        roll = lambda g: torch.roll(g, nlon // 2, dims=-1)  # noqa: E731
        u, v = _winds(nlat, _complex(s["div"]), _complex(s["zeta"]), 0.0)
        scale = (math.sqrt(2) * RADIUS / torch.cos(torch.as_tensor(np.radians(s["lats"]), device="cuda")))[:, None]
        cloud = _real(_analyse(P * torch.as_tensor(w, device="cuda"), _to_four(s["cloud"]) / math.sqrt(2)))
        return (roll(_to_grid(_synth(P, _complex(s["temp"]))) * math.sqrt(2)), roll(_to_grid(u) * scale),
                roll(_to_grid(v) * scale), cloud.reshape(*cloud.shape[:-1], -1, 2))
    if kind == "gridpoint":
        return _exact_gridpoint(case["nlat"], s["const"].params, s["gin"])
    if kind == "radiation":
        return _exact_radiation(s["params"], s["cols"])
    if kind == "surrogate":
        return _exact_surrogate(s["net"], s["params"], s["cols"], s["out"])
    net = s["net"]
    p = net.params.double().clone().requires_grad_()
    loss = ((_mlp(_layers(p, net.nin, net.nout), s["x"].double()) - s["t"].double()) ** 2).mean()
    g, = torch.autograd.grad(loss, p)
    return loss.detach().reshape(1), g, p.detach() - 1e-4 * g / (g.abs() + 1e-8)
