"""Compensated accumulation where both planes of FP64 sums do not fit (the
allocation is made to fail): the decision is kept, so a warmed-up call
allocates nothing and can be captured; the sums are allocated last and give
way to what the call cannot do without.  Results against the two-plane job:
FP64 sums in another order, rounded to FP32 once (relative RMS <= 2e-7)."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import _lib, workloads as W

pytestmark = pytest.mark.gpu

G, OS = 500, 4
COMP = dict(accum_mode=_lib.ACCUM_COMPENSATED)


def _fail(after):
    assert fg.load().oskar_b200_testing_fail_allocation(after) == _lib.OK


class Job:
    def __init__(self, n):
        rng = np.random.default_rng(n)
        self.support = np.asarray([2, 4, 2], np.int32)
        self.csh = W.min_conv_size_half(self.support, OS) + 1
        f = lambda a: torch.as_tensor(np.asarray(a, np.float32)).cuda()
        pos = rng.uniform(-200.0, 200.0, (2, n))
        # (the same kernels for every job)
        self.conv = np.random.default_rng(1).normal(
            size=2 * 3 * self.csh ** 2).astype(np.float32)
        self.args = [f(-pos[0] / G), f(pos[1] / G), f(rng.uniform(-6, 6, n)),
                     f(rng.normal(size=2 * n)), None, 1.0, 1.0, G]

    def new(self):
        ws = fg.Workspace(0)
        return ws, fg.Cube(ws, self.support, OS, self.csh, self.conv, False)

    def grid(self, ws, cube, stream=None, grid=None, **opts):
        if grid is None:
            grid = torch.zeros(2 * G * G, device="cuda")
            torch.cuda.synchronize()
        fg.grid_device(ws, cube, *self.args, grid, opts=fg.options(**opts),
                       stream=stream)
        if stream is None:
            torch.cuda.synchronize()
            assert ws.stats().status == 0
        return grid

    def reference(self):
        ws, cube = self.new()
        out = self.grid(ws, cube, **COMP)
        cube.close()
        ws.close()
        return out


def _close(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm()) <= 2e-7


@pytest.fixture
def disarm():
    yield
    _fail(-1)


def test_second_call_allocates_nothing(disarm):
    job = Job(3000)
    ref = job.reference()
    ws, cube = job.new()
    job.grid(ws, cube)              # sizes everything but the sums
    _fail(0)
    assert _close(job.grid(ws, cube, **COMP), ref)
    held = ws.bytes
    _fail(0)
    assert _close(job.grid(ws, cube, **COMP), ref)
    assert ws.bytes == held
    # the failure is still waiting for an allocation
    ws2, cube2 = fg.Workspace(0), None
    with pytest.raises(fg.GridderError) as e:
        cube2 = fg.Cube(ws2, job.support, OS, job.csh, job.conv, False)
    assert e.value.status == _lib.ERR_OUT_OF_MEMORY and cube2 is None
    # captured and replayed, with a call beside the graph in between
    s = torch.cuda.Stream()
    grid = torch.zeros(2 * G * G, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        job.grid(ws, cube, stream=s, grid=grid, **COMP)
    assert _close(job.grid(ws, cube, **COMP), ref)
    with torch.cuda.stream(s):
        graph.replay()
    torch.cuda.synchronize()
    assert _close(grid, ref)
    del graph
    cube.close()
    ws.close()
    ws2.close()


def test_sums_are_allocated_last(disarm):
    """A compensated call on a new workspace whose last allocation fails gets
    by with one plane."""
    job = Job(3000)
    ref = job.reference()
    for after in range(40):         # allocations of a plain call
        ws, cube = job.new()
        _fail(after)
        try:
            job.grid(ws, cube)
            done = True
        except fg.GridderError as e:
            assert e.status == _lib.ERR_OUT_OF_MEMORY
            done = False
        _fail(-1)
        cube.close()
        ws.close()
        if done:
            break
    assert done and after > 0
    ws, cube = job.new()
    _fail(after)
    assert _close(job.grid(ws, cube, **COMP), ref)
    cube.close()
    ws.close()


def test_second_plane_gives_way(disarm):
    """Both planes are held when a larger call's keys do not fit: the call
    gives one of them up instead of failing."""
    small, large = Job(3000), Job(600000)
    ref = large.reference()
    ws, cube = small.new()
    small.grid(ws, cube, **COMP)
    _fail(0)
    assert _close(large.grid(ws, cube, **COMP), ref)
    assert _close(small.grid(ws, cube, **COMP), small.reference())
    cube.close()
    ws.close()
