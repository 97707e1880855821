"""Ordered weights write: runs of equal cells around the lengths at which the
summing changes (a window of 32 positions and the next, 256 at a time), at
shifting offsets in the sorted order.  Bit for bit: the additions are the
reference's, in its order."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 31, 32, 33, 47, 63, 64, 65, 95, 96, 97, 255, 256, 257,
           288, 511, 512, 513, 1025]


@pytest.mark.parametrize("outside", [0, 700])
@pytest.mark.parametrize("shift", [0, 1, 30, 33, 191])
@pytest.mark.parametrize("real", [np.float32, np.float64])
def test_run_lengths(oracle, real, shift, outside):
    rng = np.random.default_rng(shift)
    g = 64
    counts = [1] * shift + LENGTHS + LENGTHS[::-1] + [20000]
    cell = np.repeat(np.arange(len(counts)) * 13 % (g * g), counts)
    cell = np.concatenate([cell, np.full(outside, -1)])
    rng.shuffle(cell)
    iv, iu = np.divmod(cell, g)
    n = cell.size
    uu = (-(iu - g // 2) / g).astype(real)
    vv = ((iv - g // 2) / g).astype(real)
    uu[cell < 0] = 5.0
    w = rng.uniform(0.1, 3.0, n).astype(real)
    start = rng.uniform(0, 1, g * g).astype(real)
    sk, ref, _, _ = oracle.weights(uu, vv, w, 1.0, g, start.copy(),
                                   np.zeros(n, real),
                                   single=real is np.float32)
    assert sk == outside
    ws = fg.Workspace(0)
    got = torch.as_tensor(start).cuda()
    skipped = torch.zeros(1, dtype=torch.int64, device="cuda")
    tu, tv, tw = (torch.as_tensor(a).cuda() for a in (uu, vv, w))
    torch.cuda.synchronize()
    fg.weights_write_device(ws, tu, tv, tw, 1.0, g, got, skipped)
    torch.cuda.synchronize()
    assert int(skipped) == outside
    assert np.array_equal(got.cpu().numpy(), ref)
    assert torch.equal(tw.cpu(), torch.as_tensor(w))
    ws.close()
