"""Degridding of chunks in which visibilities share their placement or their
cell: repeated positions (written to each of them), several planes and offsets
in a cell (gathered two at a time), supports on both sides of the widths at
which the walk changes, chunk sizes around 256, weights, against the CPU
oracle (FP64: relative RMS <= 1e-12, FP32: <= 1e-5)."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import workloads as W

pytestmark = pytest.mark.gpu

SUPPORTS = {"narrow": [0, 3, 3, 7, 7], "wide": [8, 8, 15, 16, 23, 24, 24],
            "widest": [39, 40, 40, 60]}


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("spread", [0.4, 3.0, 60.0])
@pytest.mark.parametrize("n", [1, 255, 257, 5000])
@pytest.mark.parametrize("name", list(SUPPORTS))
def test_chunks(oracle, name, n, spread, single):
    rng = np.random.default_rng(n)
    g, os_ = 400, 4
    support = np.asarray(SUPPORTS[name], np.int32)
    p = len(support)
    csh = W.min_conv_size_half(support, os_) + 1
    real = np.float32 if single else np.float64
    pos = rng.uniform(-spread, spread, (2, n))
    src = rng.integers(0, n, n)
    pos[:, ::3] = pos[:, src[::3]]
    ww = rng.uniform(0, p, n) ** 2 * rng.choice([-1.0, 1.0], n)
    ww[::3] = ww[src[::3]]
    f = lambda a: np.ascontiguousarray(a, dtype=real)
    w = dict(num_w_planes=p, support=support, oversample=os_,
             conv_size_half=csh,
             conv_func=f(rng.normal(size=2 * p * csh * csh)),
             uu=f(-pos[0] / g), vv=f(pos[1] / g), ww=f(ww),
             vis=np.zeros(2 * n), weight=f(rng.uniform(0.5, 2, n)),
             cell_size_rad=1.0, w_scale=1.0, grid_size=g)
    grid = f(rng.normal(size=2 * g * g))
    ref = {k: np.asarray(v, np.float64)
           if isinstance(v, np.ndarray) and v.dtype == real else v
           for k, v in w.items()}
    res = oracle.degrid_d(ref, grid.astype(np.float64), np.zeros(2 * n))
    vis_ref = [a for a in res if isinstance(a, np.ndarray)][0]
    vis_ref = vis_ref * np.repeat(ref["weight"], 2)
    ws = fg.Workspace(0)
    cube = fg.Cube(ws, support, os_, csh, w["conv_func"], not single)
    t = {k: torch.as_tensor(w[k]).cuda() for k in ("uu", "vv", "ww", "weight")}
    out = torch.zeros(2 * n, dtype=t["uu"].dtype, device="cuda")
    tg = torch.as_tensor(grid).cuda()
    torch.cuda.synchronize()
    fg.degrid_device(ws, cube, t["uu"], t["vv"], t["ww"], t["weight"], 1.0,
                     1.0, g, tg, out, None, fg.options(apply_weight=1))
    torch.cuda.synchronize()
    assert ws.stats().status == 0
    assert oracle.rel_rms(out.cpu().numpy(), vis_ref) <= (1e-5 if single
                                                          else 1e-12)
    cube.close()
    ws.close()
