"""Launches: their count, and the grid of a launch over a column list."""
import numpy as np
import pytest
import torch

from exoplasim_b200 import radiation as R
from exoplasim_b200 import surrogate as SG
from exoplasim_b200 import synthetic as S
from exoplasim_b200.transforms import launch_count

pytestmark = pytest.mark.gpu


def _columns(nlat, nlev, dt):
    cols, g = S.radiation_columns(nlat, nlev, seed=1, teff=True)
    zsol = SG.zsol_for(cols.pop("teff"))
    dev = {k: torch.as_tensor(np.ascontiguousarray(v), dtype=dt, device="cuda") for k, v in dict(cols, zsol=zsol).items()}
    params = R.default_params(nlev, g["nhor"], g["nlon"], nsol=0)
    return params, dev, R.alloc_outputs(params, dt)


@pytest.mark.parametrize("nhid,n", [(1, 5), (6, 300)])
def test_training_launches_are_counted(nhid, n):
    net = SG.Mlp(SG.nin_for(10), SG.nout_for(10), width=64, nhidden=nhid, max_batch=n)
    net.init(seed=1)
    x, t = torch.randn((n, net.nin), device="cuda"), torch.randn((n, net.nout), device="cuda")
    loss, nl = torch.zeros(1, device="cuda"), nhid + 1
    c0 = launch_count()
    net.forward(x)
    c1 = launch_count()
    assert c1 - c0 == nl                 # one GEMM per layer
    net.backward(x, t, loss)
    c2 = launch_count()
    # a GEMM per layer forward, the loss, a GEMM per layer below the last, all layers' weights and their sum
    assert c2 - c1 == nl + 1 + (nl - 1) + 2
    net.adam(1e-4, 1)
    assert launch_count() - c2 == 1


def _time(f, reps=5):
    f()
    best = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        best.append(a.elapsed_time(b))
    return min(best)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_column_list_fills_the_gpu(prec):
    # 32768 columns that all leave the network's training range take its own time and
    # radstep's over as many columns; half of that to spare
    dt = torch.float32 if prec == "fp32" else torch.float64
    net = SG.Mlp.load(SG.DEFAULT_NET)
    params, cols, out = _columns(128, 20, dt)
    inside = _time(lambda: SG.surrogate_step(net, params, cols, out, prec))
    cols["dt"] *= 3.0
    assert SG.surrogate_step(net, params, cols, out, prec, count=True) == params.nhor
    listed = _time(lambda: SG.surrogate_step(net, params, cols, out, prec))
    whole = _time(lambda: R.radstep(params, cols, out, prec))
    assert listed < inside + 1.5 * whole, (inside, listed, whole)
