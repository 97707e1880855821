"""The gridding kernel walks a task's visibilities with a branch for those at the
cell of the one before, or straight where most lie at another cell: one, two
and three different placements per cell (all move, half of them, a third), a
mixture of them in one call, narrow to wide footprints, kernel values through
L1 and staged, calls small enough for the kernel with the branch alone and larger
ones, against the CPU oracle (FP32: relative RMS <= 1e-5, FP64:
<= 1e-12)."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import _lib, workloads as W

pytestmark = pytest.mark.gpu

G, OS = 700, 8


@pytest.mark.parametrize("cells", [1500, 17000])
@pytest.mark.parametrize("kw", [{}, dict(staging=1),
                                dict(accum_mode=_lib.ACCUM_COMPENSATED)])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("per_cell", [(1,), (2,), (3,), (1, 3), (1, 2, 3)])
@pytest.mark.parametrize("support", [[0], [1], [2, 2], [8, 8, 3], [30, 30]])
def test_tasks(oracle, support, per_cell, single, kw, cells):
    if kw.get("accum_mode") and not single:
        kw = dict(classes_per_thread=4)      # (compensation is FP32 only)
    if kw.get("staging") and not single and max(support) > 20:
        kw = dict(tile_shift=6)              # (the rows do not fit on chip)
    rng = np.random.default_rng(len(per_cell))
    support = np.asarray(support, np.int32)
    p = len(support)
    csh = W.min_conv_size_half(support, OS) + 1
    real = np.float32 if single else np.float64
    # distinct cells, each with so many different offsets inside it
    side = 2 * 150
    cells = rng.choice(side * side, cells, replace=False)
    count = np.resize(per_cell, cells.size)
    cell = np.repeat(cells, count)
    first = np.repeat(np.cumsum(count) - count, count)
    k = np.arange(cell.size) - first
    off = (-0.25 + 0.25 * k, rng.choice([-0.25, 0.25], cell.size))
    pos = np.stack([cell % side - side // 2 + off[0],
                    cell // side - side // 2 + off[1]])
    n = cell.size
    mix = rng.permutation(n)
    f = lambda a: np.ascontiguousarray(a, dtype=real)
    w = dict(num_w_planes=p, support=support, oversample=OS,
             conv_size_half=csh,
             conv_func=f(rng.normal(size=2 * p * csh * csh)),
             uu=f(-pos[0][mix] / G), vv=f(pos[1][mix] / G),
             ww=f(rng.uniform(0, p, n) ** 2 * rng.choice([-1.0, 1.0], n)),
             vis=f(rng.normal(size=2 * n)), weight=f(np.ones(n)),
             cell_size_rad=1.0, w_scale=1.0, grid_size=G)
    ref = {a: np.asarray(v, np.float64)
           if a in ("conv_func", "uu", "vv", "ww", "vis", "weight") else v
           for a, v in w.items()}
    s1, _, g1 = oracle.grid_d(ref, threads=8)
    ws = fg.Workspace(0)
    cube = fg.Cube(ws, support, OS, csh, w["conv_func"], not single)
    t = [torch.as_tensor(w[a]).cuda() for a in ("uu", "vv", "ww", "vis")]
    grid = torch.zeros(2 * G * G, dtype=t[0].dtype, device="cuda")
    skipped = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    fg.grid_device(ws, cube, *t, None, 1.0, 1.0, G, grid, skipped,
                   opts=fg.options(**kw))
    torch.cuda.synchronize()
    assert ws.stats().status == 0
    assert int(skipped) == s1 == 0
    assert oracle.rel_rms(grid.cpu().numpy(), g1) <= (1e-5 if single
                                                      else 1e-12)
    cube.close()
    ws.close()
