"""A bounded wait between the blocks of the sort or of the task list that
expires (made to, at one tile): the call reports a timeout and takes nothing
from the unfinished lists, so grids and visibilities keep their bits, and the
next call on the same workspace is right."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import _lib, workloads as W

pytestmark = pytest.mark.gpu

N, G, OS = 20000, 600, 4          # five tiles of 4096 positions
SUPPORT = np.asarray([2, 5, 2, 8, 5], np.int32)
SORT, TASKS = 1, 2


def _inputs(real, seed=1):
    rng = np.random.default_rng(seed)
    csh = W.min_conv_size_half(SUPPORT, OS) + 1
    pos = rng.uniform(-250.0, 250.0, (2, N))
    w = dict(num_w_planes=5, support=SUPPORT, oversample=OS,
             conv_size_half=csh, conv_func=rng.normal(size=2 * 5 * csh * csh),
             uu=-pos[0] / G, vv=pos[1] / G, ww=rng.uniform(-20.0, 20.0, N),
             vis=rng.normal(size=2 * N), weight=np.ones(N),
             cell_size_rad=1.0, w_scale=1.0, grid_size=G)
    for k in ("conv_func", "uu", "vv", "ww", "vis", "weight"):
        w[k] = np.ascontiguousarray(w[k], dtype=real)
    return w, rng.normal(size=2 * G * G).astype(real)


def _arm(handle, stage, tile):
    assert fg.load().oskar_b200_testing_expire_wait(handle, stage,
                                                    tile) == _lib.OK


def _jobs(ws, count, real):
    jobs = []
    for i in range(count):
        w, start = _inputs(real, i + 1)
        cube = fg.Cube(ws, SUPPORT, OS, w["conv_size_half"], w["conv_func"],
                       real is np.float64)
        t = {k: torch.as_tensor(w[k]).cuda()
             for k in ("uu", "vv", "ww", "vis", "weight")}
        jobs.append(dict(cube=cube, cell_size_rad=1.0, w_scale=1.0,
                         grid_size=G, grid=torch.as_tensor(start).cuda(),
                         start=torch.as_tensor(start).cuda(), **t))
    return jobs


@pytest.mark.parametrize("jobs,real,kw", [
    (1, np.float32, {}), (1, np.float64, {}), (3, np.float32, {}),
    (1, np.float32, dict(staging=1)),
    (1, np.float32, dict(accum_mode=_lib.ACCUM_COMPENSATED))])
@pytest.mark.parametrize("stage,tile", [(SORT, 0), (SORT, 3), (TASKS, 0),
                                        (TASKS, 2), (TASKS, 4)])
def test_gridding(jobs, real, kw, stage, tile):
    opts = fg.options(**kw)
    ws = fg.Workspace(0)        # its task list has never been written
    batch = _jobs(ws, jobs, real)
    torch.cuda.synchronize()
    _arm(ws.handle, stage, tile)
    fg.grid_batch_device(ws, batch, opts)
    torch.cuda.synchronize()
    assert ws.stats().status == _lib.ERR_TIMEOUT
    for j in batch:
        assert torch.equal(j["grid"], j["start"])
    _arm(ws.handle, 0, 0)
    fg.grid_batch_device(ws, batch, opts)
    torch.cuda.synchronize()
    assert ws.stats().status == 0
    ws2 = fg.Workspace(0)
    for j in batch:
        fg.grid_device(ws2, j["cube"], j["uu"], j["vv"], j["ww"], j["vis"],
                       None, 1.0, 1.0, G, j["start"], opts=opts)
    torch.cuda.synchronize()
    for j in batch:
        a, b = j["grid"].double(), j["start"].double()
        # two summation orders of the same terms
        assert float((a - b).norm() / b.norm()) <= (
            2e-6 if real is np.float32 else 1e-13)
        j["cube"].close()
    ws.close()
    ws2.close()


@pytest.mark.parametrize("real", [np.float32, np.float64])
def test_degridding(real):
    ws = fg.Workspace(0)
    (j,) = _jobs(ws, 1, real)
    before = j["vis"].clone()

    def degrid(vis):
        fg.degrid_device(ws, j["cube"], j["uu"], j["vv"], j["ww"], None, 1.0,
                         1.0, G, j["grid"], vis)
        torch.cuda.synchronize()
    torch.cuda.synchronize()
    _arm(ws.handle, SORT, 2)
    degrid(j["vis"])
    assert ws.stats().status == _lib.ERR_TIMEOUT
    assert torch.equal(j["vis"], before)
    _arm(ws.handle, 0, 0)
    degrid(j["vis"])
    assert ws.stats().status == 0
    assert not torch.equal(j["vis"], before)
    j["cube"].close()
    ws.close()


@pytest.mark.parametrize("stage,tile", [(SORT, 1), (TASKS, 0), (TASKS, 3)])
@pytest.mark.parametrize("single", [False, True])
def test_drop_in(oracle, single, stage, tile):
    """Band after band is gridded there; the caller's arrays keep their
    values."""
    w, start = _inputs(np.float32 if single else np.float64)
    grid = start.copy()
    fg.load().oskar_grid_wproj_b200_release_thread_cache()
    _arm(None, stage, tile)
    try:
        with pytest.raises(fg.GridderError) as e:
            fg.grid_workload(w, single, grid, 1.5)
    finally:
        _arm(None, 0, 0)
    assert e.value.status == _lib.ERR_TIMEOUT
    assert np.array_equal(grid, start)
    skipped, _, grid = fg.grid_workload(w, single)
    ref = {k: np.asarray(v, np.float64)
           if k in ("conv_func", "uu", "vv", "ww", "vis", "weight") else v
           for k, v in w.items()}
    s1, _, g1 = oracle.grid_d(ref, threads=8)
    assert skipped == s1
    assert oracle.rel_rms(grid, g1) <= (1e-5 if single else 1e-12)


def test_bad_stage_is_refused():
    ws = fg.Workspace(0)
    for stage in (-1, 3):
        assert fg.load().oskar_b200_testing_expire_wait(
            ws.handle, stage, 0) == _lib.ERR_INVALID_ARGUMENT
    ws.close()
