"""Tasks hold points of every w-plane of one support: cubes whose planes
repeat supports in any order, cells in which many planes and offsets meet,
points spread over a whole coarse tile, and oversampling from 1 to 32,
against the CPU oracle (FP64: relative RMS <= 1e-12; FP32 on the same float
inputs: <= 1e-5)."""
import numpy as np
import pytest
import torch

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import _lib, workloads as W

pytestmark = pytest.mark.gpu

SUPPORTS = {
    "constant": [5] * 40,
    "mixed": [7, 2, 7, 3, 12, 3, 2, 12, 7, 0, 3, 7],
    "one": [9],
    "wide": [40, 1, 40, 17, 40],
}


def _job(name, oversample, spread, n=3000, grid=500):
    rng = np.random.default_rng(7)
    support = np.asarray(SUPPORTS[name], np.int32)
    p = len(support)
    csh = W.min_conv_size_half(support, oversample) + 1
    conv = rng.normal(size=2 * p * csh * csh)
    # Repeated positions (every third point copies an earlier one), plane
    # and sign of w varying independently of the position.
    pos = rng.uniform(-spread, spread, (2, n))
    src = rng.integers(0, n, n)
    pos[:, ::3] = pos[:, src[::3]]
    ww = rng.uniform(0, p, n) ** 2 * rng.choice([-1.0, 1.0], n)
    ww[::3] = ww[src[::3]]
    return dict(num_w_planes=p, support=support, oversample=oversample,
                conv_size_half=csh, conv_func=conv, uu=-pos[0] / grid,
                vv=pos[1] / grid, ww=ww, vis=rng.normal(size=2 * n),
                weight=np.ones(n), cell_size_rad=1.0, w_scale=1.0,
                grid_size=grid)


@pytest.mark.parametrize("accum", [_lib.ACCUM_PLAIN, _lib.ACCUM_COMPENSATED])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("spread", [1.5, 30.0, 205.0])
@pytest.mark.parametrize("name,oversample", [
    ("constant", 4), ("mixed", 1), ("mixed", 5), ("mixed", 8), ("one", 32),
    ("wide", 4)])
def test_groups_match_oracle(oracle, name, oversample, spread, single, accum):
    if accum == _lib.ACCUM_COMPENSATED and not single:
        pytest.skip("compensated accumulation is FP32 only")
    _check(oracle, _job(name, oversample, spread), oversample, single, accum)


@pytest.mark.parametrize("single,accum", [
    (False, _lib.ACCUM_PLAIN), (True, _lib.ACCUM_PLAIN),
    (True, _lib.ACCUM_COMPENSATED)])
@pytest.mark.parametrize("spread", [1.5, 6.0, 205.0])
@pytest.mark.parametrize("name", ["constant", "mixed", "one"])
def test_batches_match_oracle(oracle, name, spread, single, accum):
    """Enough points that a task holds several batches: all merged into a few
    records, some, none."""
    _check(oracle, _job(name, 4, spread, n=80000), 4, single, accum)


def _check(oracle, w, oversample, single, accum):
    real = np.float32 if single else np.float64
    ref = dict(w)
    for k in ("conv_func", "uu", "vv", "ww", "vis", "weight"):
        ref[k] = np.asarray(w[k], real).astype(np.float64)
    s1, n1, g1 = oracle.grid_d(ref, threads=8)
    ws = fg.Workspace(0)
    t = {k: torch.as_tensor(np.asarray(w[k], real)).cuda()
         for k in ("uu", "vv", "ww", "vis")}
    cube = fg.Cube(ws, w["support"], oversample, w["conv_size_half"],
                   np.asarray(w["conv_func"], real), not single)
    grid = torch.zeros(2 * w["grid_size"] ** 2, dtype=t["uu"].dtype,
                       device="cuda")
    skipped = torch.zeros(1, dtype=torch.int64, device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    fg.grid_device(ws, cube, t["uu"], t["vv"], t["ww"], t["vis"], None, 1.0,
                   1.0, w["grid_size"], grid, skipped, norm,
                   fg.options(accum_mode=accum))
    torch.cuda.synchronize()
    assert ws.stats().status == 0
    assert int(skipped) == s1
    assert oracle.rel_rms(grid.cpu().numpy(), g1) <= (1e-5 if single
                                                      else 1e-12)
    # norm: random kernel values cancel, so its scale is the sum of |terms|
    assert abs(float(norm) - n1) <= 1e-12 * max(
        abs(n1), float(np.abs(ref["conv_func"]).max()) * w["uu"].size * 100)
    cube.close()
    ws.close()


def test_compensated_with_one_plane_of_sums(oracle):
    """No memory for both planes of FP64 sums (the allocation is made to
    fail): the job runs twice with one plane and gives the same result, with
    compensation everywhere and within a radius."""
    w = _job("mixed", 4, 100.0)
    ref = dict(w)
    for k in ("conv_func", "uu", "vv", "ww", "vis", "weight"):
        ref[k] = np.asarray(w[k], np.float32).astype(np.float64)
    _, _, g1 = oracle.grid_d(ref, threads=8)
    t = {k: torch.as_tensor(np.asarray(w[k], np.float32)).cuda()
         for k in ("uu", "vv", "ww", "vis")}
    lib = fg.load()
    for radius in (0, 40):
        ws = fg.Workspace(0)
        cube = fg.Cube(ws, w["support"], 4, w["conv_size_half"],
                       np.asarray(w["conv_func"], np.float32), False)
        out = []
        for accum, fail in ((_lib.ACCUM_PLAIN, -1),
                            (_lib.ACCUM_COMPENSATED, 0),
                            (_lib.ACCUM_COMPENSATED, -1)):
            grid = torch.zeros(2 * w["grid_size"] ** 2, device="cuda")
            torch.cuda.synchronize()
            # (the plain job has sized everything but the sums)
            assert lib.oskar_b200_testing_fail_allocation(fail) == _lib.OK
            try:
                fg.grid_device(ws, cube, t["uu"], t["vv"], t["ww"], t["vis"],
                               None, 1.0, 1.0, w["grid_size"], grid,
                               opts=fg.options(accum_mode=accum,
                                               compensate_radius=radius))
                torch.cuda.synchronize()
            finally:
                lib.oskar_b200_testing_fail_allocation(-1)
            assert ws.stats().status == 0
            out.append(grid.cpu().numpy())
            assert oracle.rel_rms(out[-1], g1) <= 1e-5
        # FP64 sums of FP32-rounded products, rounded to FP32 once: the two
        # ways differ by the FP64 summation order before that rounding.
        if radius == 0:
            assert oracle.rel_rms(out[1], out[2]) <= 2e-7
        cube.close()
        ws.close()
