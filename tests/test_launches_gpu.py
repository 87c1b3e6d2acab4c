"""Launches: the grid of a launch over a column list."""
import numpy as np
import pytest
import torch

from exoplasim_b200 import radiation as R
from exoplasim_b200 import surrogate as SG
from exoplasim_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def _columns(nlat, nlev, dt):
    cols, g = S.radiation_columns(nlat, nlev, seed=1, teff=True)
    zsol = SG.zsol_for(cols.pop("teff"))
    dev = {k: torch.as_tensor(np.ascontiguousarray(v), dtype=dt, device="cuda") for k, v in dict(cols, zsol=zsol).items()}
    params = R.default_params(nlev, g["nhor"], g["nlon"], nsol=0)
    return params, dev, R.alloc_outputs(params, dt)


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
