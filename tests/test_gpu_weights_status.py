"""An ordered weights write whose sort gives up a bounded wait (made to, at one
tile) reports it: on device arrays through the workspace's statistics, with a
skip count or without, and through the host call's status.  The weights grid
keeps its bits, and a good call clears what it reported."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import _lib, workloads as W

pytestmark = pytest.mark.gpu

N, G = 20000, 300                 # five tiles of 4096 positions


def _arm(handle, stage, tile):
    assert fg.load().oskar_b200_testing_expire_wait(handle, stage,
                                                    tile) == _lib.OK


def _inputs(real):
    rng = np.random.default_rng(3)
    pos = rng.normal(scale=30.0, size=(2, N))
    return ((-pos[0] / G).astype(real), (pos[1] / G).astype(real),
            rng.uniform(0.1, 3.0, N).astype(real),
            rng.uniform(0, 1, G * G).astype(real))


@pytest.mark.parametrize("with_count", [True, False])
@pytest.mark.parametrize("real", [np.float32, np.float64])
@pytest.mark.parametrize("tile", [0, 2, 4])
def test_device_write(oracle, tile, real, with_count):
    uu, vv, w, start = _inputs(real)
    ws = fg.Workspace(0)
    tu, tv, tw, grid = (torch.as_tensor(a).cuda() for a in (uu, vv, w, start))
    count = torch.zeros(1, dtype=torch.int64, device="cuda") \
        if with_count else None

    def write():
        torch.cuda.synchronize()
        fg.weights_write_device(ws, tu, tv, tw, 1.0, G, grid, count)
        torch.cuda.synchronize()
        return ws.stats().status
    _arm(ws.handle, 1, tile)
    assert write() == _lib.ERR_TIMEOUT
    assert np.array_equal(grid.cpu().numpy(), start)
    if with_count:
        assert int(count) == -1         # UINT64_MAX
    _arm(ws.handle, 0, 0)
    assert write() == _lib.OK
    skipped, ref, _, _ = oracle.weights(uu, vv, w, 1.0, G, start.copy(),
                                        np.zeros(N, real),
                                        single=real is np.float32)
    assert np.array_equal(grid.cpu().numpy(), ref)
    if with_count:
        assert int(count) == skipped
    ws.close()


def test_status_beside_gridding():
    """A failed gridding call stays visible behind a good write; a gridding
    call after a failed write reports its own outcome."""
    uu, vv, w, start = _inputs(np.float32)
    support = np.asarray([2, 3], np.int32)
    csh = W.min_conv_size_half(support, 4) + 1
    ws = fg.Workspace(0)
    cube = fg.Cube(ws, support, 4, csh,
                   np.ones(2 * 2 * csh * csh, np.float32), False)
    tu, tv, tw, grid = (torch.as_tensor(a).cuda() for a in (uu, vv, w, start))
    vis = torch.ones(2 * N, device="cuda")
    image = torch.zeros(2 * G * G, device="cuda")

    def call(kind, tile=None):
        torch.cuda.synchronize()
        _arm(ws.handle, 0 if tile is None else 1, tile or 0)
        if kind == "grid":
            fg.grid_device(ws, cube, tu, tv, tw, vis, None, 1.0, 1.0, G, image)
        else:
            fg.weights_write_device(ws, tu, tv, tw, 1.0, G, grid)
        torch.cuda.synchronize()
        return ws.stats().status
    assert call("grid", 1) == _lib.ERR_TIMEOUT
    assert call("write") == _lib.ERR_TIMEOUT
    assert call("grid") == _lib.OK
    assert call("write", 1) == _lib.ERR_TIMEOUT
    assert call("grid") == _lib.OK
    assert call("write") == _lib.OK
    cube.close()
    ws.close()


@pytest.mark.parametrize("single", [False, True])
def test_host_write(single):
    real = np.float32 if single else np.float64
    uu, vv, w, start = _inputs(real)
    write = fg.gridder.oskar_grid_weights_write_f if single \
        else fg.gridder.oskar_grid_weights_write_d
    grid = start.copy()
    fg.load().oskar_grid_wproj_b200_release_thread_cache()
    _arm(None, 1, 0)
    try:
        with pytest.raises(fg.GridderError) as e:
            write(N, uu, vv, w, 1.0, G, grid)
    finally:
        _arm(None, 0, 0)
    assert e.value.status == _lib.ERR_TIMEOUT
    assert np.array_equal(grid, start)
    write(N, uu, vv, w, 1.0, G, grid)
    assert not np.array_equal(grid, start)
