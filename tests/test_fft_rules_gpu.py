"""The FFT forms on either side of the row counts where the dispatch changes between them.

Tolerances, fixed beforehand: a double transform 1e-13, a float one 2e-6 (2 log2(n) roundings of 6e-8 are 1.1e-6 at
n = 512)."""
import numpy as np
import pytest
import torch

from exoplasim_b200 import synthetic as S
from exoplasim_b200.ensemble import Ensemble
from exoplasim_b200.transforms import Plan, fc2gp, gp2fc
from tests._util import relerr

pytestmark = pytest.mark.gpu


# the rows of the forward and the inverse line (0: one form at every count)
@pytest.mark.parametrize("dt,tol,n,lines", [
    (torch.float64, 1e-13, 64, (32768, 32768)), (torch.float64, 1e-13, 128, (2048, 1024)),
    (torch.float64, 1e-13, 192, (5120, 10240)), (torch.float64, 1e-13, 256, (4608, 1152)),
    (torch.float64, 1e-13, 320, (16384, 16384)), (torch.float64, 1e-13, 384, (2560, 5120)),
    (torch.float64, 1e-13, 512, (4096, 4096)), (torch.float32, 2e-6, 64, (4096, 4096)),
    (torch.float32, 2e-6, 128, (0, 0)), (torch.float32, 2e-6, 192, (2560, 0)),
    (torch.float32, 2e-6, 256, (2048, 0)), (torch.float32, 2e-6, 320, (16384, 16384)),
    (torch.float32, 2e-6, 384, (0, 0)), (torch.float32, 2e-6, 512, (2048, 0))])
def test_rows_about_the_line(dt, tol, n, lines):
    for edge in set(lines):
        for lot in {max(1, edge - 1), edge + 1, edge + 18}:
            x = torch.randn((lot, n), generator=torch.Generator().manual_seed(lot), dtype=torch.float64).to(dt)
            c = np.fft.rfft(x.double().numpy(), axis=-1) / n
            ref = np.zeros((lot, n))
            ref[:, 0::2], ref[:, 1::2] = c.real[:, :n // 2], c.imag[:, :n // 2]
            ref[:, 1] = 0
            a = x.cuda()
            gp2fc(a)
            assert relerr(a.double().cpu().numpy(), ref) < tol
            a.copy_(torch.as_tensor(ref))
            fc2gp(a)
            c[:, n // 2] = 0
            assert relerr(a.double().cpu().numpy(), np.fft.irfft(c * n, n=n, axis=-1)) < tol


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
def test_t106_states_have_their_bits_in_any_batch(prec):
    # eight states of 320-point rows and one take two forms of the inverse; an ensemble a third, and its own forward one
    nlat, nlev, ninst = 160, 6, 8
    P, dt = Plan(nlat), torch.float64 if prec == "fp64" else torch.float32
    sp = torch.as_tensor(np.stack([S.transform_state(P.ntru, nlev, seed=i, kind="steep") for i in range(ninst)]), dtype=dt).cuda()
    gi = torch.as_tensor(np.stack([S.grid_tendencies(nlat, nlev, seed=i) for i in range(ninst)]), dtype=dt).cuda()
    td = gi[:, :4 * nlev].contiguous()
    one = {}
    for f, x in ((P.inverse_set_batch, sp), (P.forward_set_batch, gi), (P.inverse_set_d_batch, sp), (P.forward_set_d_batch, td)):
        many = f(x, nlev, precision=prec)
        for i in (0, ninst - 1):
            one[f.__name__] = f(x[i:i + 1].contiguous(), nlev, precision=prec)[0]
            assert torch.equal(many[i], one[f.__name__])
    if prec == "mixed":
        E = Ensemble([nlat, 32], [nlev, 5])
        spin, gout, gin, spout = E.buffers()
        spin.zero_(), gin.zero_()
        spin[int(E.spec_off[0]):][:sp[0].numel()] = sp[-1].reshape(-1)
        gin[int(E.gin_off[0]):][:gi[0].numel()] = gi[-1].reshape(-1)
        E.inverse(spin, gout)
        E.forward(gin, spout)
        assert torch.equal(E.unpack("gout", gout)[0].reshape(-1), one["inverse_set_batch"].reshape(-1))
        assert torch.equal(E.unpack("spec", spout)[0].reshape(-1), one["forward_set_batch"].reshape(-1))
