"""Performance cases of the B200 W-projection gridder.

Each case is one call (or one write + read pair) of the framework through its
public Python entry points, on synthetic observations of the kinds the
repository's own configurations describe: Earth-rotation-synthesis uvw tracks
of a uniform-disk or log-radial station layout, complex visibilities, an
analytic W-kernel cube whose support grows with the w-plane.

What the ranges stand for:
  * points 1e4 .. 4e7 per job, grids 512^2 .. 8192^2 (also sizes that are no
    power of two), 8 .. 256 w-planes, support 3 .. 36, oversample 4 or 8:
    the span of the plain, batching, precision and serving configurations;
  * `kind` grid / batch / degrid / weights run on device-resident tensors,
    dropin is the reference's own call on host arrays;
  * `flag` removes that fraction of the samples at random (ragged counts),
    `extent` is how far the longest baseline reaches towards the grid edge
    (above 1 some points fall outside and are skipped).
"""
import math

import numpy as np
import torch

from fpga_gridding_b200 import _lib
from fpga_gridding_b200 import gridder as fg
from fpga_gridding_b200 import workloads as W

DEC = math.radians(-30.0)
KERNEL = {"native": _lib.KERNEL_NATIVE, "f16": _lib.KERNEL_F16,
          "bf16": _lib.KERNEL_BF16}
COST_LIMIT = 1.2e10      # taps (weighted by type) a drawn case may have


def _case(kind, name=None, layout="log", stations=128, radius=30000.0,
          times=60, freq=150e6, grid=2048, planes=64, s_lo=4, s_hi=24,
          oversample=4, dtype="f32", kernel="native", compensated=False,
          weighted=False, flag=0.0, extent=1.0, channels=1):
    c = dict(kind=kind, layout=layout, stations=stations, radius=radius,
             times=times, freq=freq, grid=grid, planes=planes, s_lo=s_lo,
             s_hi=s_hi, oversample=oversample, dtype=dtype, kernel=kernel,
             compensated=compensated, weighted=weighted, flag=flag,
             extent=extent, channels=channels)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A snapshot of a small array, the smallest job a server is sent:
        # launches and latency.
        _case("grid", "snapshot_f32", "disk", 32, 1000.0, 20, grid=512,
              planes=8, s_lo=3, s_hi=8),
        # The reference-checkable job: short baselines around the uv origin,
        # many visibilities with the same placement.
        _case("grid", "small_f32", "disk", 64, 1000.0, 120, 100e6, 1024, 16,
              4, 16, extent=0.1),
        # One spectral channel of a mid-size array with visibility weights
        # and flags, a grid that is no power of two, some points outside it.
        _case("grid", "mid_weighted_f32", "log", 200, 30000.0, 157, grid=3000,
              planes=97, s_lo=3, s_hi=27, weighted=True, flag=0.3,
              extent=1.03),
        # The large single job: 39.2 M visibilities on 8192^2, 256 planes.
        _case("grid", "large_f32", "log", 512, 30000.0, 300, grid=8192,
              planes=256, s_lo=4, s_hi=36),
        # FP64 imaging of a compact array with finely oversampled kernels.
        _case("grid", "mid_f64", "disk", 160, 5000.0, 151, grid=2048,
              planes=64, s_lo=4, s_hi=24, oversample=8, dtype="f64"),
        # Compensated FP32 accumulation on a dense core (deep integrations).
        _case("grid", "compensated_f32", "disk", 300, 5000.0, 75, grid=4096,
              planes=128, s_lo=4, s_hi=32, oversample=8, compensated=True),
        # Reduced-precision kernel storage, as the resident server offers.
        _case("grid", "mid_f16_kernels", "log", 256, 30000.0, 101, grid=4096,
              planes=128, s_lo=3, s_hi=32, kernel="f16"),
        # Channels of one observation in one batched call, flagged unevenly.
        _case("batch", "channels_f32", "disk", 128, 5000.0, 60, grid=2048,
              planes=64, s_lo=3, s_hi=24, flag=0.7, channels=24),
        # Prediction: a model grid degridded to every visibility, large...
        _case("degrid", "degrid_large_f32", "log", 512, 30000.0, 120,
              grid=8192, planes=256, s_lo=4, s_hi=36),
        # ...and small.
        _case("degrid", "degrid_small_f32", "disk", 64, 1000.0, 120, 100e6,
              1024, 16, 4, 16, extent=0.1),
        # Uniform weighting of the large job: ordered write, then read.
        _case("weights", "weights_large_f32", "log", 512, 30000.0, 300,
              grid=8192),
        # The reference's own call on host arrays, mid-size.
        _case("dropin", "dropin_f32", "disk", 160, 5000.0, 100, grid=2048,
              planes=64, s_lo=4, s_hi=24),
    ]


def _cost(c):
    nb = c["stations"] * (c["stations"] - 1) // 2
    n = nb * c["times"] * c["channels"] * (1 - 0.5 * c["flag"])
    if c["kind"] == "weights":
        return n * 50
    mean = 2 * (c["s_lo"] + 0.45 * (c["s_hi"] - c["s_lo"])) + 1
    return n * mean * mean * (2 if c["dtype"] == "f64" else 1) * \
        (2 if c["compensated"] else 1)


def draw(rng):
    while True:
        kind = rng.choice(["grid", "grid", "grid", "grid", "batch", "degrid",
                           "degrid", "weights", "dropin"])
        layout = rng.choice(["log", "disk"])
        stations = int(round(math.exp(rng.uniform(math.log(24),
                                                  math.log(512)))))
        nb = stations * (stations - 1) // 2
        top = 4.0e7 if kind in ("grid", "degrid", "weights") else 4.0e6
        n = math.exp(rng.uniform(math.log(1.0e4), math.log(top)))
        times = max(1, int(round(n / nb)))
        if times > 600:
            continue
        grid = rng.choice([512, 1024, 2048, 4096, 8192,
                           2 * rng.randint(256, 2048)])
        s_lo = rng.randint(3, 6)
        s_hi = rng.randint(s_lo + 2, 36)
        dtype = "f64" if kind != "batch" and rng.random() < 0.2 else "f32"
        kernel = rng.choice(["native", "native", "f16", "bf16"]) \
            if kind == "grid" and dtype == "f32" else "native"
        c = _case(kind, None, layout, stations,
                  round(math.exp(rng.uniform(math.log(1000), math.log(30000)))),
                  times, rng.choice([100e6, 150e6, 200e6]), grid,
                  rng.randint(8, 256), s_lo, s_hi, rng.choice([4, 4, 8]),
                  dtype, kernel,
                  kind == "grid" and dtype == "f32" and rng.random() < 0.15,
                  kind in ("grid", "degrid") and rng.random() < 0.3,
                  round(rng.choice([0.0, rng.uniform(0.05, 0.7)]), 3),
                  round(rng.choice([1.0, 1.0, 1.04, rng.uniform(0.1, 0.95)]),
                        3),
                  rng.randint(4, 24) if kind == "batch" else 1)
        if grid <= 1024 and s_hi > 30:
            continue
        if kind == "dropin" and grid > 4096:
            continue
        if kind == "batch" and (grid > 2048 or n * c["channels"] > 3.0e7):
            continue
        if _cost(c) <= COST_LIMIT:
            return c


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _observation(c, seed, channel=0):
    """uvw (wavelengths), cell size, w_scale, supports: FP64, on the device,
    values rounded to the case's data type."""
    dev = _device()
    g = torch.Generator().manual_seed(1000003 * seed + 7)
    enu = (W.stations_log_radial(c["stations"], 20.0, c["radius"], g)
           if c["layout"] == "log"
           else W.stations_uniform_disk(c["stations"], c["radius"], g))
    bxyz = W.baselines_xyz(enu, DEC)
    nch = c["channels"]
    freq = c["freq"]
    if nch > 1:
        freq = 50e6 + 300e6 * channel / (nch - 1)
    uu, vv, ww = W.earth_rotation_uvw(bxyz, c["times"], 10.0, freq, DEC, dev)
    s_hi = c["s_hi"]
    fmax = 1.0
    if nch > 1:
        fmax = 350e6 / freq
        s_hi = int(round(c["s_lo"] + (s_hi - c["s_lo"]) * freq / 350e6))
    support = W.support_ramp(c["planes"], c["s_lo"], s_hi)
    uv_max = float(torch.maximum(uu.abs().max(), vv.abs().max())) * fmax
    cell = c["extent"] * (c["grid"] // 2 - c["s_hi"] - 2) / (c["grid"] * uv_max)
    w_scale = (c["planes"] - 1) ** 2 / float(ww.abs().max())
    gd = torch.Generator(device=dev).manual_seed(1000003 * seed + 13 + channel)
    if c["flag"] > 0:
        # Which samples are flagged depends on the seed, how many does not;
        # uneven over the channels of a batch (up to `flag`).
        n = uu.numel()
        frac = c["flag"] * (0.5 + 0.5 * math.sin(5.0 * channel + 1.0)
                            if nch > 1 else 1.0)
        lost = torch.randperm(n, generator=gd, device=dev)[:int(frac * n)]
        keep = torch.ones(n, dtype=torch.bool, device=dev)
        keep[lost] = False
        uu, vv, ww = uu[keep], vv[keep], ww[keep]
    if c["dtype"] == "f32":
        uu, vv, ww = (t.float() for t in (uu, vv, ww))
    return dict(uu=uu, vv=vv, ww=ww, support=support,
                cell=float(np.float32(cell)), w_scale=float(np.float32(w_scale)),
                csh=W.min_conv_size_half(support, c["oversample"]) + 1, gen=gd)


def _real(c):
    return torch.float64 if c["dtype"] == "f64" else torch.float32


def _inputs(c, seed, channel=0):
    o = _observation(c, seed, channel)
    dev, real, gd, n = _device(), _real(c), o["gen"], o["uu"].numel()
    # A few point sources' worth of flux with phases that turn along the
    # tracks, plus noise.
    ph = (o["uu"] * 0.011 + o["vv"] * 0.007).to(real)
    vis = torch.randn(n, 2, generator=gd, device=dev, dtype=real).mul_(0.1)
    vis[:, 0] += 3 * torch.cos(ph) + 1
    vis[:, 1] += 3 * torch.sin(ph)
    o["vis"] = vis.reshape(-1)
    o["weight"] = torch.rand(n, generator=gd, device=dev,
                             dtype=real).mul_(3.75).add_(0.25)
    if c["kind"] != "weights":
        o["conv"] = W.analytic_kernel_cube(o["support"], c["oversample"],
                                           o["csh"], device=dev).to(real)
    return o


_STREAM = None


def _stream():
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def prepare(case, seed):
    c = case
    kind, real, g = c["kind"], _real(c), c["grid"]
    if kind == "dropin":
        o = _inputs(c, seed)
        np_real = np.float64 if c["dtype"] == "f64" else np.float32
        host = {k: o[k].cpu().pin_memory().numpy()
                for k in ("uu", "vv", "ww", "vis", "conv")}
        grid = torch.zeros(2 * g * g, dtype=real).pin_memory().numpy()
        assert grid.dtype == np_real
        return dict(case=c, o=o, host=host, grid=grid)
    st = dict(case=c, ws=fg.Workspace(0), stream=_stream())
    if kind == "weights":
        st["o"] = _inputs(c, seed)
        st["grid"] = torch.zeros(g * g, dtype=real, device="cuda")
        st["out"] = torch.zeros_like(st["o"]["weight"])
        st["skipped"] = torch.zeros(2, dtype=torch.int64, device="cuda")
        return st
    st["opts"] = fg.options(
        kernel_type=KERNEL[c["kernel"]],
        accum_mode=(_lib.ACCUM_COMPENSATED if c["compensated"]
                    else _lib.ACCUM_PLAIN),
        apply_weight=int(c["weighted"]))
    jobs = []
    st["norm"] = torch.zeros(c["channels"], dtype=torch.float64, device="cuda")
    st["skipped"] = torch.zeros(c["channels"], dtype=torch.int64,
                                device="cuda")
    for ch in range(c["channels"]):
        o = _inputs(c, seed, ch)
        cube = fg.Cube(st["ws"], o["support"], c["oversample"], o["csh"],
                       o.pop("conv"), c["dtype"] == "f64", KERNEL[c["kernel"]])
        j = dict(cube=cube, cell_size_rad=o["cell"], w_scale=o["w_scale"],
                 grid_size=g, uu=o["uu"], vv=o["vv"], ww=o["ww"],
                 vis=o["vis"], weight=o["weight"],
                 grid=torch.zeros(2 * g * g, dtype=real, device="cuda"),
                 d_num_skipped=st["skipped"][ch:ch + 1],
                 d_norm=st["norm"][ch:ch + 1])
        if kind == "degrid":
            j["grid"] = torch.randn(2 * g * g, generator=o["gen"],
                                    device="cuda", dtype=real)
            j["vis"] = torch.zeros_like(j["vis"])
        jobs.append(j)
    st["jobs"] = jobs
    return st


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------

def run(state):
    c = state["case"]
    kind, g = c["kind"], c["grid"]
    if kind == "dropin":
        o, h = state["o"], state["host"]
        fn = fg.oskar_grid_wproj_d if c["dtype"] == "f64" \
            else fg.oskar_grid_wproj_f
        grid = state["grid"]   # accumulates, as over visibility blocks
        skipped, norm = fn(c["planes"], o["support"], c["oversample"],
                           o["csh"], h["conv"], h["uu"].size, h["uu"],
                           h["vv"], h["ww"], h["vis"], None, o["cell"],
                           o["w_scale"], g, 0.0, grid)
        return dict(grid=grid, norm=norm, skipped=skipped)
    ws, stream = state["ws"], state["stream"]
    with torch.cuda.stream(stream):
        if kind == "weights":
            o, grid, sk = state["o"], state["grid"], state["skipped"]
            grid.zero_()
            fg.weights_write_device(ws, o["uu"], o["vv"], o["weight"],
                                    o["cell"], g, grid, sk[0:1],
                                    stream=stream)
            fg.weights_read_device(ws, o["uu"], o["vv"], o["weight"],
                                   state["out"], o["cell"], g, grid, sk[1:2],
                                   stream=stream)
            return dict(grid=grid, out=state["out"], skipped=sk)
        jobs, opts = state["jobs"], state["opts"]
        if kind == "degrid":
            j = jobs[0]
            fg.degrid_device(ws, j["cube"], j["uu"], j["vv"], j["ww"],
                             j["weight"], j["cell_size_rad"], j["w_scale"], g,
                             j["grid"], j["vis"], j["d_num_skipped"], opts,
                             stream)
            return dict(vis=j["vis"], skipped=j["d_num_skipped"])
        state["norm"].zero_()
        for j in jobs:
            j["grid"].zero_()
        if kind == "batch":
            fg.grid_batch_device(ws, jobs, opts, stream)
        else:
            j = jobs[0]
            fg.grid_device(ws, j["cube"], j["uu"], j["vv"], j["ww"], j["vis"],
                           j["weight"], j["cell_size_rad"], j["w_scale"], g,
                           j["grid"], j["d_num_skipped"], j["d_norm"], opts,
                           stream)
        return dict(grids=[j["grid"] for j in jobs], norm=state["norm"],
                    skipped=state["skipped"])


# --------------------------------------------------------------------------
# Work and 64-bit results
# --------------------------------------------------------------------------

def _round(x):
    """C's round(): half away from zero."""
    t = torch.trunc(x)
    return t + torch.where((x - t).abs() >= 0.5, torch.sign(x),
                           torch.zeros_like(x))


def _place(c, o):
    g = c["grid"]
    scale = float(g) * o["cell"]
    u, v, w = (o[k].double() for k in ("uu", "vv", "ww"))
    pu, pv = -u * scale, v * scale
    plane = _round((w * o["w_scale"]).abs().sqrt()).clamp_(
        max=c["planes"] - 1).long()
    ru, rv = _round(pu), _round(pv)
    ou = _round((ru - pu) * c["oversample"]).long()
    ov = _round((rv - pv) * c["oversample"]).long()
    gu, gv = ru.long() + g // 2, rv.long() + g // 2
    s = torch.as_tensor(o["support"], device=u.device).long()[plane]
    keep = (gu - s >= 0) & (gu + s < g) & (gv - s >= 0) & (gv + s < g)
    return gu, gv, plane, ou, ov, w > 0, keep


def _weight_cells(c, o):
    """Cell of each point in the data type's own arithmetic."""
    g, real = c["grid"], _real(c)
    if c["dtype"] == "f64":
        scale = float(g) * o["cell"]
    else:
        scale = float(np.float32(g) * np.float32(o["cell"]))
    scale = torch.tensor(scale, dtype=real, device=o["uu"].device)
    gu = _round(-o["uu"] * scale).long() + g // 2
    gv = _round(o["vv"] * scale).long() + g // 2
    keep = (gu >= 0) & (gu < g) & (gv >= 0) & (gv < g)
    return gv * g + gu, keep


def work(case):
    c = case
    bytes_, flops = 0.0, 0.0
    es = 8 if c["dtype"] == "f64" else 4
    g = c["grid"]
    for ch in range(c["channels"]):
        o = _observation(c, 0, ch)
        n = o["uu"].numel()
        if c["kind"] == "weights":
            return {"bytes": 4.0 * es * n + es * g * g, "flops": 2.0 * n}
        plane, keep = _place(c, o)[2::4]
        side = 2 * torch.as_tensor(o["support"], device=plane.device).long() + 1
        taps = float((side[plane[keep]].double() ** 2).sum())
        kb = 2 * es if c["kernel"] == "native" else 4
        cube = float(c["planes"]) * o["csh"] ** 2 * kb
        bytes_ += (5 + int(c["weighted"])) * es * n + 2.0 * es * g * g + cube
        flops += 8.0 * taps
    return {"bytes": bytes_, "flops": flops}


def _taps(c, o):
    """Per plane, in chunks: (point indices, kernel values [m, k, k], flat
    grid cells [m, k, k]) of the kept points."""
    gu, gv, plane, ou, ov, conj, keep = _place(c, o)
    cube = o["conv"].double().view(c["planes"], o["csh"], o["csh"], 2)
    cube = torch.view_as_complex(cube)
    idx = torch.nonzero(keep).squeeze(1)
    idx = idx[torch.argsort(plane[idx])]
    counts = torch.bincount(plane[idx], minlength=c["planes"]).tolist()
    start = 0
    for p, m in enumerate(counts):
        s = int(o["support"][p])
        k = torch.arange(-s, s + 1, device=idx.device)
        step = max(1, 60_000_000 // k.numel() ** 2)
        for b in range(start, start + m, step):
            i = idx[b:min(b + step, start + m)]
            ru = (ou[i, None] + k * c["oversample"]).abs()
            rv = (ov[i, None] + k * c["oversample"]).abs()
            kv = cube[p].reshape(-1)[rv[:, :, None] * o["csh"] + ru[:, None, :]]
            kv = torch.where(conj[i, None, None], kv.conj(), kv)
            cells = (gv[i, None] + k)[:, :, None] * c["grid"] + \
                (gu[i, None] + k)[:, None, :]
            yield i, kv, cells
        start += m


def exact(case, seed):
    c = case
    g = c["grid"]
    if c["kind"] != "weights" and work(case)["flops"] / 8 > 6.0e9:
        return None
    grids, norms, skips = [], [], []
    for ch in range(c["channels"]):
        o = _inputs(c, seed, ch)
        dev = o["uu"].device
        if c["kind"] == "weights":
            cell, keep = _weight_cells(c, o)
            w = o["weight"].double()
            grid = torch.zeros(g * g, dtype=torch.float64, device=dev)
            grid.index_add_(0, cell[keep], w[keep])
            out = torch.zeros_like(w)
            out[keep] = w[keep] / grid[cell[keep]]
            sk = int((~keep).sum())
            return dict(grid=grid, out=out,
                        skipped=torch.tensor([sk, sk]))
        keep = _place(c, o)[6]
        skipped = torch.tensor([int((~keep).sum())])
        wt = o["weight"].double() if c["weighted"] else None
        if c["kind"] == "degrid":
            gen = o["gen"]
            grid = torch.view_as_complex(
                torch.randn(2 * g * g, generator=gen, device=dev,
                            dtype=_real(c)).double().view(-1, 2))
            vis = torch.zeros(o["uu"].numel(), dtype=torch.complex128,
                              device=dev)
            for i, kv, cells in _taps(c, o):
                vis[i] = (grid[cells] * kv.conj()).sum((1, 2))
            if wt is not None:
                vis = vis * wt
            return dict(vis=torch.view_as_real(vis).reshape(-1),
                        skipped=skipped)
        vis = torch.view_as_complex(o["vis"].double().view(-1, 2))
        if wt is not None:
            vis = vis * wt
        grid = torch.zeros(g * g, 2, dtype=torch.float64, device=dev)
        norm = torch.zeros(1, dtype=torch.float64, device=dev)
        for i, kv, cells in _taps(c, o):
            t = kv.real.sum((1, 2))
            norm += (t * wt[i] if wt is not None else t).sum()
            grid.index_add_(0, cells.reshape(-1), torch.view_as_real(
                kv * vis[i, None, None]).reshape(-1, 2))
        grid = grid.reshape(-1)
        if c["kind"] == "dropin":
            return dict(grid=grid.cpu().numpy(), norm=float(norm),
                        skipped=int(skipped))
        grids.append(grid)
        norms.append(norm)
        skips.append(skipped)
    return dict(grids=grids, norm=torch.cat(norms), skipped=torch.cat(skips))
