"""Degridding takes smaller chunks for smaller calls.  A visibility's value does
not depend on its chunk: one call over all points (chunks of 256) and calls
over pieces of 1 to 100 000 points (chunks of 32, 64, 128) give the same bits."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("piece", [1, 31, 33, 18943, 18944, 37889, 75777,
                                   100000])
def test_pieces(piece, single):
    rng = np.random.default_rng(piece)
    n, g, os_ = 200_000, 400, 4
    support = np.asarray([2, 5, 8, 8], np.int32)
    csh = W.min_conv_size_half(support, os_) + 1
    real = np.float32 if single else np.float64
    f = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=real)).cuda()
    ws = fg.Workspace(0)
    cube = fg.Cube(ws, support, os_, csh,
                   rng.normal(size=2 * 4 * csh * csh).astype(real), not single)
    pos = rng.uniform(-60.0, 60.0, (2, n))
    uu, vv = f(-pos[0] / g), f(pos[1] / g)
    ww = f(rng.uniform(0, 4, n) ** 2 * rng.choice([-1.0, 1.0], n))
    grid = f(rng.normal(size=2 * g * g))
    whole = torch.zeros(2 * n, dtype=uu.dtype, device="cuda")
    torch.cuda.synchronize()
    fg.degrid_device(ws, cube, uu, vv, ww, None, 1.0, 1.0, g, grid, whole,
                     None)
    begin = 50_001
    part = torch.zeros(2 * piece, dtype=uu.dtype, device="cuda")
    at = slice(begin, begin + piece)
    pu, pv, pw = (a[at].clone() for a in (uu, vv, ww))
    torch.cuda.synchronize()
    fg.degrid_device(ws, cube, pu, pv, pw, None, 1.0, 1.0, g, grid, part, None)
    torch.cuda.synchronize()
    assert ws.stats().status == 0
    assert torch.equal(part, whole[2 * begin:2 * (begin + piece)])
    cube.close()
    ws.close()
