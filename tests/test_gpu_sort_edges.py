"""Sort and task list at the edges of their tiles (4096 positions): the
ordered weights write, whose sums depend on a stable sort, and a gridding job
whose points are one per task, many per task, all skipped or all in one cell.
Weights bit for bit, gridding FP64 to relative RMS <= 1e-12."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 255, 4095, 4096, 4097, 8192, 12289, 300001]


@pytest.mark.parametrize("real", [np.float32, np.float64])
@pytest.mark.parametrize("n", SIZES)
def test_ordered_weights(oracle, n, real):
    rng = np.random.default_rng(n)
    g = 300
    pos = rng.normal(scale=30.0, size=(2, n))
    pos[:, ::17] *= 40.0        # some outside
    uu, vv = (-pos[0] / g).astype(real), (pos[1] / g).astype(real)
    w = rng.uniform(0.1, 3.0, n).astype(real)
    ref = rng.uniform(0, 1, g * g).astype(real)
    got = torch.as_tensor(ref.copy()).cuda()
    sk, ref, _, _ = oracle.weights(uu, vv, w, 1.0, g, ref, np.zeros(n, real),
                                   single=real is np.float32)
    ws = fg.Workspace(0)
    skipped = torch.zeros(1, dtype=torch.int64, device="cuda")
    tu, tv, tw = (torch.as_tensor(a).cuda() for a in (uu, vv, w))
    torch.cuda.synchronize()
    fg.weights_write_device(ws, tu, tv, tw, 1.0, g, got, skipped)
    torch.cuda.synchronize()
    assert int(skipped) == sk
    assert np.array_equal(got.cpu().numpy(), ref)
    ws.close()


@pytest.mark.parametrize("spread", [0.2, 20.0, 1000.0, 1e7])
@pytest.mark.parametrize("n", SIZES)
def test_task_list(oracle, n, spread):
    rng = np.random.default_rng(n)
    g, os_ = 1100, 4
    support = np.array([2, 3, 2, 6], np.int32)
    csh = W.min_conv_size_half(support, os_) + 1
    pos = rng.uniform(-spread, spread, (2, n))
    if spread > 1e6:
        pos += 2 * spread       # every point outside
    w = dict(num_w_planes=4, support=support, oversample=os_,
             conv_size_half=csh,
             conv_func=rng.normal(size=2 * 4 * csh * csh), uu=-pos[0] / g,
             vv=pos[1] / g, ww=rng.uniform(-9.0, 9.0, n),
             vis=rng.normal(size=2 * n), weight=np.ones(n),
             cell_size_rad=1.0, w_scale=1.0, grid_size=g)
    s1, _, g1 = oracle.grid_d(w, threads=8)
    s2, _, g2 = fg.grid_workload(w, single=False)
    assert s1 == s2
    if s1 == n:
        assert not g2.any()
    else:
        assert oracle.rel_rms(g2, g1) <= 1e-12
