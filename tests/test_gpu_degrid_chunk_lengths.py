"""Degridding in chunks of 64, 128 and 256 visibilities, for narrow, wide and
the widest footprints: calls just large enough for each length, in cells so
dense that equal placements and pairs reach across the warps of a chunk, and in
sparser ones.  A sample against the CPU oracle (FP64: relative RMS <= 1e-12,
FP32: <= 1e-5), and pieces of the call, which run in chunks of 32, bit for
bit."""
import math

import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import workloads as W

pytestmark = pytest.mark.gpu

SUPPORTS = {"narrow": [0, 3, 3, 7, 7], "wide": [8, 8, 15, 16, 23, 24, 24],
            "widest": [39, 40, 40, 60]}
G, OS = 400, 4


def _points(chunk, support, single):
    """The fewest points that take this chunk (degrid_plan.h)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    taps = chunk * (2 * max(support) + 1) ** 2
    n = 4 * sms * chunk
    if taps > 300000:
        n = max(n, math.ceil(taps / (0.75 if single else 0.6)))
    return n + 13


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("spread", [0.4, 6.0])
@pytest.mark.parametrize("name,chunk", [
    ("narrow", 64), ("narrow", 128), ("narrow", 256), ("wide", 64),
    ("wide", 128), ("wide", 256), ("widest", 64), ("widest", 128)])
def test_chunk(oracle, name, chunk, spread, single):
    rng = np.random.default_rng(chunk)
    support = np.asarray(SUPPORTS[name], np.int32)
    p, n = len(support), _points(chunk, SUPPORTS[name], single)
    csh = W.min_conv_size_half(support, OS) + 1
    real = np.float32 if single else np.float64
    pos = rng.uniform(-spread, spread, (2, n))
    ww = rng.uniform(0, p, n) ** 2 * rng.choice([-1.0, 1.0], n)
    src = rng.integers(0, n, n)
    pos[:, ::3] = pos[:, src[::3]]
    ww[::3] = ww[src[::3]]
    f = lambda a: np.ascontiguousarray(a, dtype=real)
    conv, grid = f(rng.normal(size=2 * p * csh * csh)), \
        f(rng.normal(size=2 * G * G))
    uu, vv, ww = f(-pos[0] / G), f(pos[1] / G), f(ww)
    ws = fg.Workspace(0)
    cube = fg.Cube(ws, support, OS, csh, conv, not single)
    tg = torch.as_tensor(grid).cuda()

    def degrid(at):
        a = [torch.as_tensor(x[at]).cuda() for x in (uu, vv, ww)]
        out = torch.zeros(2 * a[0].numel(), dtype=a[0].dtype, device="cuda")
        torch.cuda.synchronize()
        fg.degrid_device(ws, cube, *a, None, 1.0, 1.0, G, tg, out)
        torch.cuda.synchronize()
        assert ws.stats().status == 0
        return out.cpu().numpy().reshape(-1, 2)
    whole = degrid(slice(None))
    for begin in (0, n // 2 + 1, n - 5000):
        at = slice(begin, begin + 5000)
        assert np.array_equal(degrid(at), whole[at])
    some = rng.integers(0, n, 2000)
    w = dict(num_w_planes=p, support=support, oversample=OS,
             conv_size_half=csh, conv_func=conv.astype(np.float64),
             uu=uu[some].astype(np.float64), vv=vv[some].astype(np.float64),
             ww=ww[some].astype(np.float64), vis=np.zeros(4000),
             weight=np.ones(2000), cell_size_rad=1.0, w_scale=1.0,
             grid_size=G)
    res = oracle.degrid_d(w, grid.astype(np.float64), np.zeros(4000))
    ref = [a for a in res if isinstance(a, np.ndarray)][0]
    assert oracle.rel_rms(whole[some].reshape(-1), ref) <= (
        1e-5 if single else 1e-12)
    cube.close()
    ws.close()
