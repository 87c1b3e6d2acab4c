"""The FFT forms on either side of the row counts where the dispatch changes between them.

Tolerances, fixed beforehand: a double transform 1e-13, a float one 2e-6 (2 log2(n) roundings of 6e-8 are 1.1e-6 at
n = 512); sets FP64 1e-12, FP32 2e-5, mixed 5e-6, the bars those paths have elsewhere."""
import numpy as np
import pytest
import torch

from exoplasim_b200 import synthetic as S
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


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 2e-5), ("mixed", 5e-6)])
def test_t106_batch_and_states(prec, tol):
    # eight states of 320-point rows take the many-row form, one the other
    nlat, nlev, ninst = 160, 6, 8
    P, dt = Plan(nlat), torch.float64 if prec == "fp64" else torch.float32
    sp = torch.as_tensor(np.stack([S.transform_state(P.ntru, nlev, seed=i, kind="steep") for i in range(ninst)]), dtype=dt).cuda()
    gi = torch.as_tensor(np.stack([S.grid_tendencies(nlat, nlev, seed=i) for i in range(ninst)]), dtype=dt).cuda()
    td = gi[:, :4 * nlev].contiguous()
    for f, x in ((P.inverse_set_batch, sp), (P.forward_set_batch, gi), (P.inverse_set_d_batch, sp), (P.forward_set_d_batch, td)):
        many = f(x, nlev, precision=prec).double().cpu().numpy()
        for i in (0, ninst - 1):
            one = f(x[i:i + 1].contiguous(), nlev, precision=prec).double().cpu().numpy()[0]
            for a, b in zip(many[i].reshape(len(one), -1), one.reshape(len(one), -1)):
                assert relerr(a, b) < tol
