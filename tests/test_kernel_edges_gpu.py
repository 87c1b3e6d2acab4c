"""The transform, grid-point, radiation and training kernels at the sizes where
their tiles end and their dispatch turns, and the rules of dispatch against the
general path.

Tolerances, fixed beforehand: FP64 against the FP64 oracle 1e-12 per field (the
sums have at most 256 terms of 1.1e-16 each, twice, and the FFT log2(n) stages);
FP32 sets 2e-5 and mixed sets 5e-6, the bars those paths have elsewhere.  A
float FFT 2e-6 (2 log2(n) roundings of 6e-8 are 1.1e-6 at n = 512), a double one
1e-13.  The grid-point step's two forms differ by the
order of no sum, so FP64 outputs agree to a rounding of the quotients, 1e-14;
in FP32, where the compiler may contract differently and nearly equal terms are
subtracted, 1e-4.  Radiation 1e-9: the longwave
effective emission divides by the logarithm of a transmissivity clamped at
1 - 1e-6, which amplifies a few roundings of 1.1e-16 a million times, and a
single column has no larger neighbour to be measured against.  Gradients 1e-4
per tensor."""
import numpy as np
import pytest
import torch

from exoplasim_b200 import gridpoint as GP
from exoplasim_b200 import postprocess as PP
from exoplasim_b200 import pyfft
from exoplasim_b200 import radiation as R
from exoplasim_b200 import surrogate as SG
from exoplasim_b200 import synthetic as S
from exoplasim_b200.ensemble import Ensemble
from exoplasim_b200.transforms import Plan, fc2gp, gp2fc, tc_error
from tests._util import relerr

pytestmark = pytest.mark.gpu

FFTMOD_N = (8, 16, 32, 64, 96, 128, 256, 384, 512)
DT = {"fp64": torch.float64, "fp32": torch.float32, "mixed": torch.float32}
TOL = {"fp64": 1e-12, "fp32": 2e-5, "mixed": 5e-6}


def _cuda(a, dt=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")


class Oracle:
    """The oracle's sets; lengths that neither fftmod nor fft991 transforms pass its FFT untouched, and numpy's
    takes its place."""

    def __init__(self, oracle, nlat):
        self.L, self.n = oracle.Leg(nlat), 2 * nlat
        self.own = self.n in FFTMOD_N + (192, 320)
        self.use991 = self.n not in FFTMOD_N

    def inverse(self, f, sp, nlev):
        rows = getattr(self.L, f)(sp, nlev, plavor=S.EZ, use991=self.use991)
        if self.own:
            return rows
        r = rows.reshape(len(rows), -1, self.n)
        c = np.zeros(r.shape[:-1] + (self.n // 2 + 1,), complex)
        c[..., :-1] = r[..., 0::2] + 1j * r[..., 1::2]
        return (np.fft.irfft(c, n=self.n, axis=-1) * self.n).reshape(len(rows), -1)

    def forward(self, f, g, nlev):
        if not self.own:
            c = np.fft.rfft(g.reshape(len(g), -1, self.n), axis=-1)[..., :-1] / self.n
            g = np.stack((c.real, c.imag), axis=-1).reshape(len(g), -1)
        return getattr(self.L, f)(np.ascontiguousarray(g), nlev, use991=self.use991)


def _worst(a, b):
    return max(relerr(a[f], b[f]) for f in range(len(b)))


# nlat 8 and 16: less than one table tile; 48, 72, 120: latitude pairs past a multiple of 8, an FFT length without a
# kernel of its own; 144, 160, 180, 200: mixed sets on either side of both lines between the FP64 and tcgen05 kernels
@pytest.mark.parametrize("nlat,nlev,ninst,prec", [
    (8, 1, 1, "fp64"), (8, 3, 2, "fp32"), (16, 2, 5, "fp64"), (32, 1, 1, "fp64"), (32, 5, 9, "fp32"), (48, 3, 1, "fp64"),
    (72, 7, 3, "fp64"), (120, 1, 2, "fp32"), (128, 13, 2, "fp64"), (160, 1, 1, "fp64"), (256, 1, 1, "fp64"),
    (32, 1, 1, "mixed"), (48, 3, 2, "mixed"), (128, 3, 3, "mixed"), (144, 1, 2, "mixed"), (160, 3, 1, "mixed"),
    (180, 1, 2, "mixed"), (200, 2, 1, "mixed"), (256, 1, 3, "mixed")])
def test_sets_at_tile_edges(oracle, nlat, nlev, ninst, prec):
    P = Plan(nlat)
    O = Oracle(oracle, nlat)
    kind = "steep" if nlat >= 144 else "nn1"
    spins = [S.transform_state(P.ntru, nlev, seed=3 + i, kind=kind) for i in range(ninst)]
    gins = [S.grid_tendencies(nlat, nlev, seed=30 + i) for i in range(ninst)]
    ts, tg = _cuda(np.stack(spins), DT[prec]), _cuda(np.stack(gins), DT[prec])
    td = tg[:, :4 * nlev].contiguous()
    gp = P.inverse_set_batch(ts, nlev, precision=prec).double().cpu().numpy()
    sp = P.forward_set_batch(tg, nlev, precision=prec).double().cpu().numpy()
    gd = P.inverse_set_d_batch(ts, nlev, precision=prec).double().cpu().numpy()
    sd = P.forward_set_d_batch(td, nlev, precision=prec).double().cpu().numpy()
    for i in {0, ninst - 1}:
        g = gins[i].reshape(9 * nlev + 1, -1)
        assert _worst(gp[i].reshape(6 * nlev + 3, -1), O.inverse("inverse_set", spins[i], nlev)) < TOL[prec]
        assert _worst(sp[i], O.forward("forward_set", g, nlev)) < TOL[prec]
        assert _worst(gd[i].reshape(4 * nlev + 1, -1), O.inverse("inverse_set_d", spins[i], nlev)) < TOL[prec]
        assert _worst(sd[i], O.forward("forward_set_d", g[:4 * nlev], nlev)) < TOL[prec]
    assert tc_error() == 0


# T21 and T42: the global means are warps of the forward launch in both sets; T127: in the gridpointd one
@pytest.mark.parametrize("nlat,nlev,ninst", [(32, 1, 1), (32, 5, 3), (64, 13, 2), (192, 2, 2)])
def test_mixed_global_means_are_rounded_once(oracle, nlat, nlev, ninst):
    # FP64 sums rounded once to float32: half an ulp, and 1e-14 for the order of the sums
    P = Plan(nlat)
    O = Oracle(oracle, nlat)
    gin = np.stack([S.grid_tendencies(nlat, nlev, seed=70 + i) for i in range(ninst)])
    gin[:, :2 * nlev] += 0.3
    gin[:, 3 * nlev:4 * nlev] += 0.2
    g = _cuda(gin, torch.float32)
    sa = P.forward_set_batch(g, nlev, precision="mixed").double().cpu().numpy()
    sd = P.forward_set_d_batch(g[:, :4 * nlev].contiguous(), nlev, precision="mixed").double().cpu().numpy()
    for i in range(ninst):
        rows = g[i].double().cpu().numpy().reshape(9 * nlev + 1, -1)
        for out, ref, top in ((sa[i], O.forward("forward_set", rows, nlev), [4 * nlev]),
                              (sd[i], O.forward("forward_set_d", rows[:4 * nlev], nlev), [])):
            for f in list(range(nlev, 2 * nlev)) + list(range(3 * nlev, 4 * nlev)) + top:
                half = 0.5 * float(np.spacing(np.float32(abs(ref[f][0]))))
                assert abs(out[f][0] - ref[f][0]) <= half + 1e-14 * abs(ref[f][0]) and out[f][1] == 0.0, (i, f)


@pytest.mark.parametrize("nlat,prec", [(32, "fp64"), (64, "fp32"), (64, "mixed"), (192, "mixed")])
def test_sets_on_arrays_aligned_to_their_reals(nlat, prec):
    # a grid that starts on an odd element takes the general FFT, a state the FP64 kernels
    nlev = 3
    P = Plan(nlat)

    def odd(t):
        b = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
        b[1:] = t.reshape(-1)
        return b[1:].view(t.shape)

    ts = _cuda(S.transform_state(P.ntru, nlev, seed=1)[None], DT[prec])
    tg = _cuda(S.grid_tendencies(nlat, nlev, seed=2)[None], DT[prec])
    for f, t in ((P.inverse_set_batch, ts), (P.forward_set_batch, tg)):
        a = f(t, nlev, precision=prec).double().cpu().numpy()[0]
        b = f(odd(t), nlev, precision=prec).double().cpu().numpy()[0]
        assert _worst(b.reshape(len(b), -1), a.reshape(len(a), -1)) < TOL[prec]


@pytest.mark.parametrize("n", [64, 128, 192, 256, 320, 384, 512])
@pytest.mark.parametrize("dt,tol", [(torch.float64, 1e-13), (torch.float32, 2e-6)])
def test_fft_ragged_row_counts(n, dt, tol):
    # the register-resident kernels' last block, against numpy and against the general kernel
    for lot in (1, 3, 17, 65):
        x = np.random.default_rng(n + lot).standard_normal((lot, n))
        x = _cuda(x, dt).double().cpu().numpy()
        ref = np.zeros_like(x)
        c = np.fft.rfft(x, axis=-1) / n
        ref[:, 0::2], ref[:, 1::2] = c.real[:, :n // 2], c.imag[:, :n // 2]
        ref[:, 1] = 0
        a = _cuda(x, dt)
        b = torch.empty(x.size + 1, dtype=dt, device="cuda")[1:].view(lot, n)
        b.copy_(a)
        for t in (a, b):
            gp2fc(t)
            assert relerr(t.double().cpu().numpy(), ref) < tol
        c[:, n // 2] = 0
        for t in (a, b):
            t.copy_(_cuda(ref, dt))
            fc2gp(t)
            assert relerr(t.double().cpu().numpy(), np.fft.irfft(c * n, n=n, axis=-1)) < tol


def test_ensemble_of_both_kernel_families():
    nlat, nlev = [32, 160, 192, 256, 32, 128], [1, 3, 2, 1, 5, 2]
    E = Ensemble(nlat, nlev)
    spins = [_cuda(S.transform_state((2 * n - 1) // 3, L, seed=i, kind="nn1"), torch.float32)
             for i, (n, L) in enumerate(zip(nlat, nlev))]
    gins = [_cuda(S.grid_tendencies(n, L, seed=50 + i), torch.float32) for i, (n, L) in enumerate(zip(nlat, nlev))]
    _, gout, _, spout = E.buffers()
    E.inverse(E.pack("spec", spins), gout)
    E.forward(E.pack("gin", gins), spout)
    gouts, spouts = E.unpack("gout", gout), E.unpack("spec", spout)
    for i, (n, L) in enumerate(zip(nlat, nlev)):
        P = Plan(n)
        g = P.inverse_set_batch(spins[i][None].contiguous(), L, precision="mixed")[0].double().cpu().numpy()
        s = P.forward_set_batch(gins[i][None].contiguous(), L, precision="mixed")[0].double().cpu().numpy()
        assert _worst(gouts[i].double().cpu().numpy().reshape(len(g), -1), g.reshape(len(g), -1)) < TOL["mixed"]
        assert _worst(spouts[i].double().cpu().numpy().reshape(len(s), -1), s) < TOL["mixed"]
    assert tc_error() == 0


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_sets_under_capture(prec):
    # a batch captured where one state's call sized the work buffer, and a graph
    # whose plan has grown its work buffer since
    nlev, ninst = 4, 6
    P = Plan(32)
    sp = _cuda(np.stack([S.transform_state(P.ntru, nlev, seed=i) for i in range(ninst)]), DT[prec])
    gi = _cuda(np.stack([S.grid_tendencies(32, nlev, seed=i) for i in range(ninst)]), DT[prec])
    ref = Plan(32)
    rg, rs = ref.inverse_set_batch(sp, nlev, precision=prec), ref.forward_set_batch(gi, nlev, precision=prec)
    P.inverse_set(sp[0].contiguous(), nlev, precision=prec)
    P.forward_set(gi[0].contiguous(), nlev, precision=prec)
    og, os_ = torch.zeros_like(rg), torch.zeros_like(rs)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        og.copy_(P.inverse_set_batch(sp, nlev, precision=prec))
        os_.copy_(P.forward_set_batch(gi, nlev, precision=prec))
    P.inverse_set_batch(sp.repeat(8, 1, 1), nlev, precision=prec)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(og, rg) and torch.equal(os_, rs)


# either side of each unrolled level count, and past the last
@pytest.mark.parametrize("nlev", [2, 7, 8, 10, 11, 13, 14, 16, 17, 20, 21, 25, 26])
@pytest.mark.parametrize("nqspec", [1, 0])
def test_gridpoint_forms_agree(nlev, nqspec):
    # a g with one entry above its diagonal, too small to count, takes the general form
    nlat, ninst = 8, 3
    P = Plan(nlat)
    p = GP.default_params(nlev, nqspec=nqspec)
    q = GP.default_params(nlev, nqspec=nqspec)
    q.g[nlev * (nlev - 1)] = 1e-300       # g(0, nlev - 1)
    rng = np.random.default_rng(nlev)
    gin = rng.standard_normal((ninst, 6 * nlev + 3, nlat, 2 * nlat)) * 1e-2
    dq = np.abs(rng.standard_normal((ninst, nlev, nlat, 2 * nlat))) * 1e-3
    for dt, tol in ((torch.float64, 1e-14), (torch.float32, 1e-4)):
        o = []
        for c in (p, q):
            dw = torch.zeros((ninst, nlev, nlat, 2 * nlat), dtype=dt, device="cuda")
            out = GP.gridpoint(P, GP.GpConst(c), _cuda(gin, dt), dw=dw, dq=None if nqspec else _cuda(dq, dt))
            o.append((out.double().cpu().numpy(), dw.double().cpu().numpy()))
        for i in range(ninst):
            assert _worst(o[0][0][i], o[1][0][i]) < tol
        assert relerr(o[0][1], o[1][1]) < tol


@pytest.mark.parametrize("ncol", [1, 7, 15, 16, 17, 33])
@pytest.mark.parametrize("nlev", [5, 13, 25])
def test_radstep_partial_blocks(oracle, ncol, nlev):
    cols, g = S.radiation_columns(8, nlev, seed=ncol)
    nhor = g["nhor"]
    pick = np.random.default_rng(ncol).permutation(nhor)[:ncol]
    cols = {k: v if k in ("sid", "cola") else np.ascontiguousarray(v[pick] if k == "dsalb" else v[..., pick])
            for k, v in cols.items()}
    params = R.default_params(nlev, ncol, ncol, nsol=0)   # one latitude
    sig = [np.array(getattr(params, k)[:nlev]) for k in ("sigma", "sigmah", "dsigma")]
    ref = oracle.radstep(oracle.radpar(nlev, ncol, ncol, *sig, nsol=0), cols["sid"], cols["cola"],
                         {k: v.copy() for k, v in cols.items()})
    dev = {k: _cuda(v) for k, v in cols.items()}
    out = R.radstep(params, dev)
    for k in ("dfu", "dfd", "dftu", "dftd", "dswfl", "dlwfl", "dflux", "dtdtswr", "dtdtlwr"):
        assert relerr(out[k].cpu().numpy(), ref[k]) < 1e-9, k


# batches about a tile of 128 rows and a range of 256; input widths that are no multiple of four
@pytest.mark.parametrize("nlev,width,nhid,n", [(5, 32, 1, 1), (5, 96, 2, 129), (10, 128, 7, 255), (13, 64, 3, 257)])
def test_training_tiles(nlev, width, nhid, n):
    from oracle import mlp_oracle as MO
    nin, nout = SG.nin_for(nlev), SG.nout_for(nlev)
    net = SG.Mlp(nin, nout, width=width, nhidden=nhid, max_batch=n + 3)
    net.init(seed=1)
    g = np.random.default_rng(n)
    X, T = (g.standard_normal((n, w)).astype(np.float32) for w in (nin, nout))
    params = net.params.cpu().numpy()
    loss = torch.zeros(1, device="cuda")
    Y = net.forward(_cuda(X, torch.float32)).cpu().numpy()
    net.backward(_cuda(X, torch.float32), _cuda(T, torch.float32), loss)
    assert relerr(Y, MO.forward(params, net.layers, X)[0]) < 1e-4
    gref = MO.loss_and_grads(params, net.layers, X, T)[1]
    G = net.grads.cpu().numpy()
    for wo, bo, di, do in net.layers:
        assert relerr(G[wo:wo + di * do], gref[wo:wo + di * do]) < 1e-4
        assert relerr(G[bo:bo + do], gref[bo:bo + do]) < 1e-4


@pytest.mark.parametrize("nlat,ntimes,nlev", [(32, 1, 1), (48, 2, 3), (64, 3, 5), (96, 1, 7)])
@pytest.mark.parametrize("nfs", [0, 1])
def test_output_transforms_equal_their_parts(nlat, ntimes, nlev, nfs):
    # one call per variable against sp2fc / dv2uv, the FFT, scaling and roll
    P = Plan(nlat, pyfft_nfs=nfs, plavor=0.0)
    nlon, nrsp = 2 * nlat, (P.ntru + 1) * (P.ntru + 2)
    rng = np.random.default_rng(nlat)
    a, b = (rng.standard_normal((ntimes, nlev, nrsp)) for _ in range(2))
    odd = torch.empty(a.size + 1, dtype=torch.float64, device="cuda")[1:].view(a.shape)
    odd.copy_(_cuda(a))
    fc = P.sp2fc(_cuda(a).reshape(-1, nrsp))
    fc2gp(fc)
    grid = torch.roll(fc * pyfft.SQRT2, nlat, dims=-1).reshape(ntimes, nlev, nlat, nlon)
    args = (nlat, nlon, nlev, P.ntru)
    for v in (_cuda(a), odd, _cuda(a).transpose(0, 1).contiguous().transpose(0, 1)):
        assert relerr(PP.transformvar(v, *args, physfilter=nfs).cpu().numpy(), grid.cpu().numpy()) < 1e-13
    u, v = P.dv2uv(_cuda(a).reshape(-1, nrsp), _cuda(b).reshape(-1, nrsp))
    lats = np.arcsin(P.gauss()[0])
    sc = _cuda(PP.SQRT2 * 6371220.0 / np.cos(lats)).view(1, nlat, 1)
    got = PP.transformvectorvar(_cuda(a), _cuda(b), lats, nlon, nlev, P.ntru, physfilter=nfs)
    for x, y in zip((u, v), got):
        fc2gp(x)
        ref = torch.roll(x * sc, nlat, dims=-1).reshape(ntimes, nlev, nlat, nlon)
        assert relerr(y.cpu().numpy(), ref.cpu().numpy()) < 1e-13
    rows = (grid / pyfft.SQRT2).reshape(-1, nlat, nlon).contiguous()
    gp2fc(rows)
    ref = P.fc2sp(rows).reshape(ntimes, nlev, nrsp // 2, 2)
    goff = torch.empty(grid.numel() + 1, dtype=torch.float64, device="cuda")[1:].view(grid.shape)
    goff.copy_(grid)
    for v in (grid, goff):
        keep = v.clone()
        assert relerr(PP.transformvar(v, *args, mode="spectral", physfilter=nfs).cpu().numpy(), ref.cpu().numpy()) < 1e-13
        assert torch.equal(v, keep)
    with pytest.raises(ValueError):
        PP.transformvar(_cuda(a), nlat, nlon + 2, nlev, P.ntru)
    with pytest.raises(ValueError):
        pyfft.sp2gp(_cuda(a[0].T[:-2]), nlat, nlon, P.ntru)
    with pytest.raises(ValueError):
        pyfft.gp2sp(torch.zeros((nlon, nlat + 2, 1), dtype=torch.float64, device="cuda"), nlat, nlon, P.ntru)
