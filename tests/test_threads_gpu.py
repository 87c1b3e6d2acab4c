"""Calls of several host threads, each with its own plan, arrays and stream."""
import threading

import numpy as np
import pytest
import torch

from exoplasim_b200 import _lib
from exoplasim_b200 import gridpoint as GP
from exoplasim_b200 import radiation as R
from exoplasim_b200 import synthetic as S
from exoplasim_b200 import transforms as TR

pytestmark = pytest.mark.gpu


def _fft(n, dt, name):
    a = torch.zeros((2, n), dtype=dt, device="cuda")
    return TR, lambda: getattr(TR, name)(a)


def _set(nlat):
    P = TR.Plan(nlat)
    sp = torch.zeros((1, 5, P.nrsp), device="cuda")
    out = torch.zeros((1, 9, nlat, 2 * nlat), device="cuda")
    return TR, lambda: P.inverse_set_batch(sp, 1, precision="fp32", out=out)


def _rad(nlev, prec):
    dt = torch.float64 if prec == "fp64" else torch.float32
    cols, g = S.radiation_columns(8, nlev, seed=1)
    dev = {k: torch.as_tensor(np.ascontiguousarray(v), dtype=dt, device="cuda") for k, v in cols.items()}
    p = R.default_params(nlev, g["nhor"], g["nlon"], nsol=0)
    out = R.alloc_outputs(p, dt)
    return R, lambda: R.radstep(p, dev, out, prec)


def _gp(nlev):
    P, c = TR.Plan(8), GP.GpConst(GP.default_params(nlev))
    gin = torch.zeros((1, 6 * nlev + 3, 8, 16), device="cuda")
    out = torch.zeros((1, 9 * nlev + 1, 8, 16), device="cuda")
    return GP, lambda: GP.gridpoint(P, c, gin, out)


def _bare(module, f, monkeypatch):
    """f's call of the library alone, for a loop that spends its time there."""
    got = []
    with monkeypatch.context() as m:
        m.setattr(module, "call", lambda *a: (got.append(a), _lib.call(*a)))
        f()
    (name, *args), = got
    entry = getattr(_lib.load(), name)
    return lambda: entry(*args)


# calls that launch one kernel with different amounts of shared memory, above the default limit
@pytest.mark.parametrize("make", [
    lambda: (_fft(384, torch.float32, "fc2gp"), _set(192)),
    lambda: (_fft(4096, torch.float64, "gp2fc"), _fft(3200, torch.float64, "gp2fc")),
    lambda: (_fft(4096, torch.float64, "fc2gp"), _fft(3200, torch.float64, "fc2gp")),
    lambda: (_rad(25, "fp64"), _rad(20, "fp64")),
    lambda: (_rad(25, "fp32"), _rad(20, "fp32")),
    lambda: (_gp(40), _gp(30))], ids=["fft384", "gp2fc", "fc2gp", "rad64", "rad32", "gridpoint"])
def test_two_threads_on_one_kernel(make, monkeypatch):
    device, calls = torch.cuda.current_device(), []
    pair = make()
    for module, f in pair:
        with torch.cuda.stream(torch.cuda.Stream()):
            f()                                  # modules, tables and buffers
            calls.append(_bare(module, f, monkeypatch))
    torch.cuda.synchronize()
    failed = [0, 0]

    def work(i):
        torch.cuda.set_device(device)
        for _ in range(10000):
            failed[i] += calls[i]() != 0

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failed == [0, 0]
