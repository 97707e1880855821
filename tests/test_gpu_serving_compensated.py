"""A server with compensated accumulation takes one plane of FP64 sums where both
would exceed its memory budget: it stays within the budget, with the results of
the two-plane job (FP64 sums rounded to FP32 once: relative RMS <= 2e-7)."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import _lib, workloads as W
from fpga_gridding_b200.serving import Server

pytestmark = pytest.mark.gpu

N, G, OS = 5000, 2048, 4          # 32 MiB of grid and of sums per plane


@pytest.mark.parametrize("budget_mib,planes", [(100, 1), (256, 2)])
def test_budget(budget_mib, planes):
    rng = np.random.default_rng(4)
    support = np.asarray([2, 4, 6], np.int32)
    csh = W.min_conv_size_half(support, OS) + 1
    conv = rng.normal(size=2 * 3 * csh * csh).astype(np.float32)
    f = lambda a: torch.as_tensor(np.asarray(a, np.float32)).cuda()
    pos = rng.uniform(-900.0, 900.0, (2, N))
    uu, vv, ww = f(-pos[0] / G), f(pos[1] / G), f(rng.uniform(-5, 5, N))
    vis, weight = f(rng.normal(size=2 * N)), f(np.ones(N))
    opts = fg.options(accum_mode=_lib.ACCUM_COMPENSATED)
    ws = fg.Workspace(0)
    cube = fg.Cube(ws, support, OS, csh, conv, False)
    ref = torch.zeros(2 * G * G, device="cuda")
    torch.cuda.synchronize()
    fg.grid_device(ws, cube, uu, vv, ww, vis, None, 1.0, 1.0, G, ref,
                   opts=opts)
    torch.cuda.synchronize()
    srv = Server(0, budget_bytes=budget_mib << 20, slots=1, max_batch=1,
                 opts=opts)
    used = []
    for tag in range(3):
        srv.submit(tag, cube, uu, vv, ww, vis, weight, 1.0, 1.0, G)
        done = []
        for _ in range(120):
            done = srv.poll(timeout=1.0)
            if done:
                break
        assert len(done) == 1 and done[0]["status"] == 0
        got = srv.grid(done[0]).clone()
        assert float((got - ref).norm() / ref.norm()) <= 2e-7
        used.append(srv.memory()[0])
        srv.release(tag)
    assert used[0] == used[1] == used[2] <= budget_mib << 20
    # grid, sums and 20 MiB of the smallest buffers
    assert (32 + 32 * planes) << 20 <= used[0] <= (56 + 32 * planes) << 20
    srv.close()
    cube.close()
    ws.close()
