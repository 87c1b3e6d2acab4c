"""Device memory of a plan: what its sets allocate goes back when it goes, and a
request that no GPU can meet leaves the plan usable."""
import gc

import pytest
import torch

from exoplasim_b200._lib import ExotxError, FP64, call
from exoplasim_b200.transforms import Plan, _ptr, _stream

pytestmark = pytest.mark.gpu

NLAT, NLEV, NINST = 64, 20, 8
FIELDS = NLAT * (2 * NLAT // 3 + 1) * 16   # bytes of Fourier intermediate per FP64 field
BLOCK = 4 << 20                            # two 2 MiB blocks, in which the driver hands out memory
HUGE = 1 << 22                             # levels whose intermediate, over 200 GB a state, no GPU holds


def _used():
    gc.collect()
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


class Sets:
    """A plan with the arrays of both sets: torch allocates nothing during a call."""

    def __init__(self, nlat=NLAT, nlev=NLEV, ninst=NINST):
        self.p, self.nlev = Plan(nlat), nlev
        g = torch.Generator(device="cuda").manual_seed(nlat)
        f = lambda n, *s: torch.randn((ninst, n, *s), generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
        self.sp, self.gi = f(4 * nlev + 1, self.p.nrsp), f(9 * nlev + 1, nlat, 2 * nlat)
        self.gp, self.so = torch.zeros_like(f(6 * nlev + 3, nlat, 2 * nlat)), torch.zeros_like(self.sp)

    def inverse(self, n=None):
        return self.p.inverse_set_batch(self.sp[:n], self.nlev, precision="fp64", out=self.gp[:n])

    def forward(self, n=None):
        return self.p.forward_set_batch(self.gi[:n], self.nlev, precision="fp64", out=self.so[:n])

    def beyond_memory(self):
        with pytest.raises(ExotxError) as e:
            call("exotx_inverse_set", self.p._h, FP64, _ptr(self.sp), _ptr(self.gp), HUGE, _stream())
        assert e.value.code == 5   # out of device memory


def test_destroyed_plan_gives_its_memory_back():
    s = Sets()
    s.inverse(), s.forward()   # modules and FFT tables
    s.p = None
    before = _used()
    for _ in range(3):
        s.p = Plan(NLAT)
        s.inverse()
        s.forward()            # more fields: outgrows the inverse set's buffer, 8 x 123 of them
        s.p = None
    assert _used() - before < BLOCK


def test_requests_beyond_memory_leave_the_plan_usable():
    s = Sets()
    ref = (s.inverse().clone(), s.forward().clone())
    torch.cuda.synchronize()
    for _ in range(3):         # each after the buffer has grown again
        s.beyond_memory()
        s.inverse(2)
        s.beyond_memory()
        s.gp.zero_(), s.so.zero_()
        assert torch.equal(s.inverse(), ref[0]) and torch.equal(s.forward(), ref[1])
    torch.cuda.synchronize()


def test_outgrown_buffer_is_given_back_at_once():
    # where no captured graph uses it, a plan holds what its largest call needs
    s = Sets()
    s.inverse(), s.forward()
    s.p = None
    s.p = Plan(NLAT)
    tables = _used()
    s.inverse()
    s.forward()
    assert _used() - tables < NINST * (9 * NLEV + 1) * FIELDS + BLOCK


def test_captured_graphs_keep_their_buffers():
    s = Sets()
    ref = s.inverse(2).clone()
    torch.cuda.synchronize()
    s.p = None
    s.p = Plan(NLAT)
    s.inverse(2)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        s.inverse(2)
    held = _used()
    full = s.forward().clone()             # outgrows the graph's buffer
    s.beyond_memory()                      # and gives its own back in vain
    other = torch.full((NINST * (9 * NLEV + 1) * FIELDS // 8,), 7.0, device="cuda", dtype=torch.float64)
    s.gp.zero_()
    graph.replay()                         # writes to no memory but the graph's
    torch.cuda.synchronize()
    assert torch.equal(s.gp[:2], ref) and bool((other == 7.0).all())
    assert torch.equal(s.forward(), full)
    del graph, other, full, ref
    s.p = None
    torch.cuda.empty_cache()
    assert _used() <= held
