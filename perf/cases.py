"""Workloads for timing the framework through its public entry points.

A case is a dict of plain values: the operation (`op`), the data type, how
the visibilities are distributed (`sky`), their number and the shape of the
grid and the kernel stack.  `listed()` holds the standing cases, `draw(rng)`
makes further ones of the same ranges, `prepare` builds the inputs on the GPU
from a seed, `run` makes one pass and returns its outputs whole, `work` says
what a pass cannot do without, and `exact` gives the outputs in 64 bits from
plain torch operations.

Two distributions of visibilities occur in real use:

* "uniform": radially concentrated (u, v), w uniform in +-w_max, in no
  particular order -- the synthetic-challenge shape;
* "tracks": Earth-rotation tracks of an SKA-LOW-like array (log-normal
  station radii), time-major, w growing with the baseline.

The kernels are a Gaussian taper times a chirp, plane p's support rising
linearly with p.
"""
import importlib
import math

import numpy as np
import torch

gridder = importlib.import_module("gpu-gridding_gb300")

DEVICE = "cuda"
SPEED_OF_LIGHT = 299792458.0
LATITUDE = math.radians(-26.82)
DECLINATION = math.radians(-27.0)
TRACK_HOURS = 4.0
W_MAX = 5000.0          # wavelengths, "uniform"
UV_SIGMA, UV_CLIP = 0.12, 0.45   # fractions of the grid's extent, "uniform"
TAPS_AT_ONCE = 1 << 25  # footprint taps held at once by exact()


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _uniform(name, op, n, grid_size, planes, s_min, s_max, dtype="float32",
             oversample=4):
    return {"name": name, "op": op, "dtype": dtype, "sky": "uniform",
            "n": n, "grid_size": grid_size, "planes": planes, "s_min": s_min,
            "s_max": s_max, "oversample": oversample}


def _tracks(name, op, stations, times, grid_size, planes, s_min, s_max,
            dtype="float32", oversample=4, channels=1):
    return {"name": name, "op": op, "dtype": dtype, "sky": "tracks",
            "stations": stations, "times": times, "channels": channels,
            "grid_size": grid_size, "planes": planes, "s_min": s_min,
            "s_max": s_max, "oversample": oversample}


def listed():
    return [
        # One correlator dump of a small array on a quick-look grid: the
        # launches and the host path are what it costs.
        _uniform("grid_small", "grid", 4000, 256, 16, 2, 8),
        # A short snapshot at ordinary size.
        _uniform("grid_2048", "grid", 200_000, 2048, 128, 4, 24),
        # The synthetic-challenge dataset: 8192^2, 714 planes, random order.
        _uniform("grid_synthetic_8192", "grid", 2_152_800, 8192, 714, 4, 36),
        # A quarter of an SKA-LOW EL82-70 observation, 339 planes.
        _tracks("grid_el82_70", "grid", 512, 60, 8192, 339, 8, 44),
        # A whole SKA-LOW EL56-82 observation: the largest call.
        _tracks("grid_el56_82", "grid", 512, 240, 8192, 601, 4, 72),
        # The same gridder in double precision, at ordinary size.
        _uniform("grid_2048_f64", "grid", 200_000, 2048, 128, 4, 24,
                 dtype="float64"),
        # Predicting visibilities from a model grid (a major cycle's other
        # half), at ordinary size and on a quarter of an observation.
        _uniform("degrid_2048", "degrid", 200_000, 2048, 128, 4, 24),
        _tracks("degrid_el56_82", "degrid", 512, 60, 8192, 601, 4, 72),
        # A training step through the autograd function: gridding forward,
        # gradients of amplitudes and weights backward.
        _uniform("train_synthetic_8192", "train", 2_152_800, 8192, 714, 4,
                 36),
        # Sixteen channels of a 128-station array, each 0-60 % flagged, onto
        # grids of their own in one call.
        _tracks("batched_16x2048", "batched", 128, 120, 2048, 339, 8, 44,
                channels=16),
        # Uniform weighting of an observation: the density grid, then the
        # re-weighted visibilities.
        _tracks("weights_8192", "weights", 512, 60, 8192, 16, 4, 8),
        # The drop-in call on numpy arrays, adding to the caller's grid.
        _uniform("host_2048", "host", 200_000, 2048, 128, 4, 24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("grid", "grid", "grid", "degrid", "degrid", "train",
                     "batched", "weights", "host"))
    grid_size = _log_int(rng, 200, 8192)
    if rng.random() < 0.5:
        grid_size = max(200, grid_size // 64 * 64)
    s_min = rng.randint(2, 8)
    s_max = min(_log_int(rng, s_min + 1, 72), grid_size // 8)
    planes = _log_int(rng, 8, 714)
    oversample = rng.choice((4, 4, 4, 4, 2, 3, 8))
    if oversample > 4:
        s_max = min(s_max, 36)
    dtype = "float32"
    if op in ("grid", "degrid") and rng.random() < 0.2:
        dtype = "float64"
    if op == "batched" or (op in ("grid", "degrid", "weights") and
                           rng.random() < 0.4):
        stations = _log_int(rng, 24, 96 if dtype == "float64" else 512)
        baselines = stations * (stations - 1) // 2
        most = 400_000 if dtype == "float64" else 8_000_000
        times = min(240, max(4, _log_int(rng, 4, 240)), most // baselines)
        channels = 1
        if op == "batched":
            grid_size = min(grid_size, 4096)
            s_max = min(s_max, grid_size // 8)
            channels = rng.randint(2, 24)
            times = max(4, min(times, most // (baselines * channels)))
        return _unnamed(_tracks("", op, stations, times, grid_size, planes,
                                s_min, s_max, dtype, oversample, channels))
    most = 300_000 if dtype == "float64" else 2_500_000
    n = _log_int(rng, 2000, most)
    if s_max > 36:
        n = min(n, most // 4)
    return _unnamed(_uniform("", op, n, grid_size, planes, s_min, s_max,
                             dtype, oversample))


def _unnamed(case):
    return {k: v for k, v in case.items() if k != "name"}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _supports(case):
    p = np.arange(case["planes"], dtype=np.float64)
    span = max(case["planes"] - 1, 1)
    s = case["s_min"] + (case["s_max"] - case["s_min"]) * p / span
    return np.rint(s).astype(np.int32)


def _conv_size_half(case):
    return (int(_supports(case).max()) + 1) * case["oversample"]


def _cube(case):
    """The kernel quadrants [P, csh, csh, 2] of the case's stack."""
    dtype = getattr(torch, case["dtype"])
    csh, planes = _conv_size_half(case), case["planes"]
    s = torch.from_numpy(_supports(case)).to(DEVICE, torch.float64)
    w = 8.0 * torch.arange(planes, device=DEVICE, dtype=torch.float64) / max(
        planes - 1, 1)
    r = torch.arange(csh, device=DEVICE, dtype=torch.float64)
    taper = torch.exp(-2.0 * (r / case["oversample"]) ** 2 /
                      (s.clamp(min=1)[:, None] ** 2))
    side = torch.polar(taper, math.pi * w[:, None] * r ** 2 / csh ** 2)
    # The taps at zero offset sum to one over the whole footprint.
    lattice = side[:, :: case["oversample"]].clone()
    m = torch.arange(lattice.shape[1], device=DEVICE)
    lattice[m > s[:, None]] = 0
    total = 2 * lattice.sum(1) - lattice[:, 0]
    side = side / total[:, None]
    out = torch.empty((planes, csh, csh, 2), dtype=dtype, device=DEVICE)
    for a in range(0, planes, 64):
        k = side[a:a + 64]
        out[a:a + 64] = torch.view_as_real(k[:, :, None] * k[:, None, :])
    return out


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, device=DEVICE,
                      dtype=torch.float64)


def _randn(gen, *shape, dtype=torch.float32):
    return torch.randn(shape, generator=gen, device=DEVICE, dtype=dtype)


def _uniform_uvw(case, gen):
    n, cell = case["n"], 0.16384 / case["grid_size"]
    extent = 1.0 / cell
    r = (_randn(gen, n, dtype=torch.float64).abs() * UV_SIGMA).clamp(
        max=UV_CLIP) * extent
    theta = 2 * math.pi * _rand(gen, n)
    w = W_MAX * (2 * _rand(gen, n) - 1)
    return r * torch.cos(theta), r * torch.sin(theta), w, cell, W_MAX


def _baselines(stations, rng):
    """Baselines (X, Y, Z) in metres of an array with log-normal station
    radii: median 1 km, 70 % within 2 km, none past 65 km."""
    r = np.empty(0)
    while r.shape[0] < stations:
        c = np.exp(rng.normal(math.log(1000.0), math.log(2.0) / 0.5244,
                              stations))
        r = np.concatenate([r, c[c <= 65000.0]])
    r, az = r[:stations], rng.uniform(0, 2 * math.pi, stations)
    east, north = r * np.sin(az), r * np.cos(az)
    xyz = np.stack([-math.sin(LATITUDE) * north, east,
                    math.cos(LATITUDE) * north])
    i, j = np.triu_indices(stations, k=1)
    return xyz[:, j] - xyz[:, i]


def _track_uvw(case, xyz, times):
    """(u, v, w) in metres, time-major, as a [3, times * baselines] tensor."""
    x, y, z = (torch.from_numpy(a).to(DEVICE)[None, :] for a in xyz)
    ha = torch.linspace(-0.5, 0.5, times, device=DEVICE,
                        dtype=torch.float64) * TRACK_HOURS * math.pi / 12
    sh, ch = torch.sin(ha)[:, None], torch.cos(ha)[:, None]
    sd, cd = math.sin(DECLINATION), math.cos(DECLINATION)
    u = sh * x + ch * y
    v = -sd * ch * x + sd * sh * y + cd * z
    w = cd * ch * x - cd * sh * y + sd * z
    return torch.stack([u.reshape(-1), v.reshape(-1), w.reshape(-1)])


def _tracks_uvw(case, gen, seed):
    """u, v, w in wavelengths, channel by channel, and each channel's first
    visibility.  Several channels span 100-200 MHz and lose 0-60 % each."""
    rng = np.random.default_rng(seed)
    uvw = _track_uvw(case, _baselines(case["stations"], rng), case["times"])
    channels = case["channels"]
    freqs = np.linspace(1e8, 2e8, channels) if channels > 1 else [1e8]
    top = freqs[-1] / SPEED_OF_LIGHT
    u_max, w_max = float(uvw[:2].abs().max()) * top, float(
        uvw[2].abs().max()) * top
    G = case["grid_size"]
    cell = (G / 2 - case["s_max"] - 2) / (G * u_max)
    parts, offsets = [], [0]
    for f in freqs:
        part = uvw * (f / SPEED_OF_LIGHT)
        if channels > 1:
            keep = 1.0 - rng.uniform(0, 0.6)
            part = part[:, _rand(gen, part.shape[1]) < keep]
        parts.append(part)
        offsets.append(offsets[-1] + part.shape[1])
    u, v, w = torch.cat(parts, 1) if channels > 1 else parts[0]
    return u, v, w, cell, w_max, offsets


def _inputs(case, seed):
    """What the caller holds: coordinates, amplitudes, weights, the cube."""
    dtype = getattr(torch, case["dtype"])
    gen = torch.Generator(DEVICE).manual_seed(seed)
    offsets = None
    if case["sky"] == "tracks":
        u, v, w, cell, w_max, offsets = _tracks_uvw(case, gen, seed)
    else:
        u, v, w, cell, w_max = _uniform_uvw(case, gen)
    n = u.shape[0]
    x = {"n": n, "offsets": offsets, "grid_size": case["grid_size"],
         "uu": u.to(dtype).contiguous(), "vv": v.to(dtype).contiguous(),
         "ww": w.to(dtype).contiguous(),
         "cell_size_rad": float(np.float32(cell)),
         "w_scale": float(np.float32((case["planes"] - 1) ** 2 / w_max))}
    del u, v, w
    op = case["op"]
    x["weight"] = (1.5 - _rand(gen, n)).to(dtype)
    if op in ("grid", "batched", "train", "host"):
        x["vis"] = _randn(gen, n, 2, dtype=dtype)
    if op in ("degrid", "train"):
        G = case["grid_size"]
        x["model"] = _randn(gen, G, G, 2, dtype=dtype)
    if op != "weights":
        x["cube"] = _cube(case)
    return x


def prepare(case, seed):
    """The inputs on the GPU and what a program keeps: plan, kernel stack and
    output arrays (for the drop-in call: numpy arrays on the host)."""
    x = _inputs(case, seed)
    s = {"op": case["op"], "x": x}
    dtype, G = getattr(torch, case["dtype"]), case["grid_size"]
    precision = "d" if case["dtype"] == "float64" else "f"
    if case["op"] == "host":
        s["stack"] = (case["planes"], _supports(case), case["oversample"],
                      _conv_size_half(case), x.pop("cube").cpu().numpy())
        for k in ("uu", "vv", "ww", "vis", "weight"):
            x[k] = x[k].cpu().numpy()
        s["grid"] = np.zeros((G, G, 2), case["dtype"])
        s["grid"].fill(0)
        return s
    s["plan"] = gridder.Plan()
    if case["op"] == "weights":
        s["density"] = torch.zeros((G, G), dtype=dtype, device=DEVICE)
        s["weight_out"] = torch.zeros(x["n"], dtype=dtype, device=DEVICE)
        s["skipped"] = torch.zeros(2, dtype=torch.int64, device=DEVICE)
        return s
    s["stack"] = gridder.KernelStack(
        case["planes"], _supports(case), case["oversample"],
        _conv_size_half(case), x.pop("cube"), precision)
    if case["op"] == "degrid":
        s["out"] = torch.zeros((x["n"], 2), dtype=dtype, device=DEVICE)
    elif case["op"] == "train":
        x["vis"].requires_grad_(True)
        x["weight"].requires_grad_(True)
    else:
        c = case.get("channels", 1)
        s["grid"] = torch.zeros((c, G, G, 2), dtype=dtype, device=DEVICE)
        s["norm"] = torch.zeros(c, dtype=torch.float64, device=DEVICE)
        s["skipped"] = torch.zeros(c, dtype=torch.int64, device=DEVICE)
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    x, op = s["x"], s["op"]
    geometry = (x["cell_size_rad"], x["w_scale"], x["grid_size"])
    if op == "grid":
        s["grid"].zero_()
        s["norm"].zero_()
        gridder.grid_wproj_device(
            s["plan"], s["stack"], x["uu"], x["vv"], x["ww"], x["vis"],
            x["weight"], *geometry, s["grid"], s["norm"], s["skipped"])
        return {k: s[k] for k in ("grid", "norm", "skipped")}
    if op == "batched":
        s["grid"].zero_()
        s["norm"].zero_()
        gridder.grid_wproj_batched_device(
            s["plan"], s["stack"], x["offsets"], x["uu"], x["vv"], x["ww"],
            x["vis"], x["weight"], *geometry, s["grid"], s["norm"],
            s["skipped"])
        return {k: s[k] for k in ("grid", "norm", "skipped")}
    if op == "degrid":
        gridder.degrid_wproj_device(s["plan"], s["stack"], x["uu"], x["vv"],
                                    x["ww"], *geometry, x["model"], s["out"])
        return {"vis": s["out"]}
    if op == "train":
        grid = gridder.GridWproj.apply(
            x["vis"], x["weight"], x["uu"], x["vv"], x["ww"], s["stack"],
            s["plan"], *geometry)
        d_vis, d_weight = torch.autograd.grad(
            grid, (x["vis"], x["weight"]), grad_outputs=x["model"])
        return {"grid": grid.detach(), "d_vis": d_vis, "d_weight": d_weight}
    if op == "weights":
        s["density"].zero_()
        cell, _, G = geometry
        gridder.grid_weights_write_device(
            s["plan"], x["uu"], x["vv"], x["weight"], cell, G, s["density"],
            s["skipped"][:1])
        gridder.grid_weights_read_device(
            s["plan"], x["uu"], x["vv"], x["weight"], s["weight_out"], cell,
            G, s["density"], s["skipped"][1:])
        return {k: s[k] for k in ("density", "weight_out", "skipped")}
    # The drop-in call adds to the grid that the caller holds.
    skipped, norm = gridder.oskar_grid_wproj_f(
        *s["stack"], x["n"], x["uu"], x["vv"], x["ww"], x["vis"],
        x["weight"], *geometry, s["grid"], 0.0)
    return {"grid": s["grid"], "norm": norm, "skipped": skipped}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _points(case):
    if case["sky"] == "uniform":
        return case["n"]
    kept = 0.7 if case["channels"] > 1 else 1.0
    return int(case["stations"] * (case["stations"] - 1) // 2 *
               case["times"] * case["channels"] * kept)


def _taps_per_point(case):
    """Mean footprint taps of a visibility."""
    if case["sky"] == "uniform":
        p = np.sqrt((np.arange(4096) + 0.5) / 4096)
    else:
        x, y, z = _baselines(case["stations"], np.random.default_rng(0))
        ws = []
        for h in np.linspace(-0.5, 0.5, 5) * TRACK_HOURS * math.pi / 12:
            ws.append(np.abs(math.cos(DECLINATION) * (
                math.cos(h) * x - math.sin(h) * y) +
                math.sin(DECLINATION) * z))
        w = np.concatenate(ws)
        scale = 0.75 if case["channels"] > 1 else 1.0
        p = np.sqrt(w / w.max() * scale)
    s = _supports(case)[np.rint(p * (case["planes"] - 1)).astype(int)]
    return float(np.mean((2.0 * s + 1) ** 2))


def work(case):
    n, G = _points(case), case["grid_size"]
    real = 8 if case["dtype"] == "float64" else 4
    op = case["op"]
    if op == "weights":
        # Coordinates and weights in, density and new weights out.
        return {"bytes": real * (4 * n + G * G), "flops": 2 * n}
    grids = 2 * real * G * G * case.get("channels", 1)
    quadrant = float(np.sum((_supports(case) * case["oversample"] + 1.0) ** 2))
    taps = 2 * real * quadrant
    flops = 8 * n * _taps_per_point(case)
    if op == "degrid":
        return {"bytes": real * 5 * n + grids + taps, "flops": flops}
    if op == "train":
        return {"bytes": real * 9 * n + 2 * grids + taps, "flops": 2 * flops}
    return {"bytes": real * 6 * n + grids + taps, "flops": flops}


# ---------------------------------------------------------------------------
# The outputs in 64 bits
# ---------------------------------------------------------------------------
def _round(a):
    """Half away from zero, as C's round()."""
    t = torch.trunc(a)
    return t + torch.where((a - t).abs() >= 0.5, torch.sign(a), 0.0).to(
        a.dtype)


def _scalar(value, dtype):
    return (np.float32 if dtype == torch.float32 else np.float64)(value)


def _placed(x, case, a, b):
    """Cells, offsets, planes and conjugation of the points a..b that lie on
    the grid (by the gridder's definition, in the inputs' own precision), as
    tensors, with their indices."""
    dtype, G = x["uu"].dtype, case["grid_size"]
    scale = float(_scalar(G, dtype) * _scalar(x["cell_size_rad"], dtype))
    pu, pv = -x["uu"][a:b] * scale, x["vv"][a:b] * scale
    ru, rv = _round(pu), _round(pv)
    ww = x["ww"][a:b]
    plane = _round(torch.sqrt((ww * float(_scalar(x["w_scale"], dtype))).abs())
                   ).to(torch.int64).clamp(max=case["planes"] - 1)
    s = torch.from_numpy(_supports(case)).to(DEVICE, torch.int64)[plane]
    gu, gv = ru.to(torch.int64) + G // 2, rv.to(torch.int64) + G // 2
    os = case["oversample"]
    ou = _round((ru - pu) * os).to(torch.int64)
    ov = _round((rv - pv) * os).to(torch.int64)
    on = (gu + s < G) & (gu - s >= 0) & (gv + s < G) & (gv - s >= 0)
    i = torch.nonzero(on).reshape(-1)
    i = i[torch.argsort(plane[i], stable=True)]
    return (i + a, gu[i], gv[i], ou[i], ov[i], plane[i], ww[i] > 0,
            (b - a) - int(on.sum()))


def _footprints(x, case, cube, a, b):
    """Pieces of the points a..b, plane by plane: point indices, flat grid
    cells [m, F, F] and complex taps [m, F, F] with the conjugation in."""
    i, gu, gv, ou, ov, plane, neg, _ = _placed(x, case, a, b)
    G, os = case["grid_size"], case["oversample"]
    supports = _supports(case)
    counts = torch.bincount(plane, minlength=case["planes"]).tolist()
    at = 0
    for p, count in enumerate(counts):
        s = int(supports[p])
        k = torch.arange(-s, s + 1, device=DEVICE)
        step = max(1, TAPS_AT_ONCE // (2 * s + 1) ** 2)
        for lo in range(at, at + count, step):
            q = slice(lo, min(lo + step, at + count))
            rows = (ov[q, None] + k * os).abs()
            cols = (ou[q, None] + k * os).abs()
            taps = torch.view_as_complex(
                cube[p][rows[:, :, None], cols[:, None, :]].double())
            taps = torch.where(neg[q, None, None], taps.conj(), taps)
            cells = ((gv[q, None] + k) * G)[:, :, None] + (
                gu[q, None] + k)[:, None, :]
            yield i[q], cells, taps
        at += count


def _exact_grid(x, case, cube, a, b):
    """Grid [G, G, 2], norm and skips of the points a..b."""
    G = case["grid_size"]
    grid = torch.zeros((G * G, 2), dtype=torch.float64, device=DEVICE)
    norm = torch.zeros((), dtype=torch.float64, device=DEVICE)
    w = x["weight"].detach().double()
    vis = torch.view_as_complex(x["vis"].detach().double())
    for i, cells, taps in _footprints(x, case, cube, a, b):
        value = taps * (w[i] * vis[i])[:, None, None]
        grid.index_add_(0, cells.reshape(-1),
                        torch.view_as_real(value).reshape(-1, 2))
        norm += (taps.real.sum((1, 2)) * w[i]).sum()
    return grid.reshape(G, G, 2), norm, _placed(x, case, a, b)[-1]


def _exact_degrid(x, case, cube):
    model = torch.view_as_complex(x["model"].double()).reshape(-1)
    out = torch.zeros(x["n"], dtype=torch.complex128, device=DEVICE)
    for i, cells, taps in _footprints(x, case, cube, 0, x["n"]):
        out[i] = (taps.conj() * model[cells]).sum((1, 2))
    return out


def _exact_weights(x, case):
    dtype, G = x["uu"].dtype, case["grid_size"]
    scale = float(_scalar(G, dtype) * _scalar(x["cell_size_rad"], dtype))
    gu = _round(-x["uu"] * scale).to(torch.int64) + G // 2
    gv = _round(x["vv"] * scale).to(torch.int64) + G // 2
    on = (gu >= 0) & (gu < G) & (gv >= 0) & (gv < G)
    cell = (gv * G + gu)[on]
    w = x["weight"].double()
    density = torch.zeros(G * G, dtype=torch.float64, device=DEVICE)
    density.index_add_(0, cell, w[on])
    out = torch.zeros_like(w)
    d = density[cell]
    out[on] = torch.where(d != 0, w[on] / d, 0.0)
    skipped = torch.full((2,), int((~on).sum()), dtype=torch.int64)
    return {"density": density.reshape(G, G), "weight_out": out,
            "skipped": skipped}


def exact(case, seed):
    op = case["op"]
    x = _inputs(case, seed)
    if op == "weights":
        return _exact_weights(x, case)
    if _points(case) * _taps_per_point(case) > 1.1e10:
        return None
    cube = x["cube"]
    if op == "degrid":
        return {"vis": torch.view_as_real(_exact_degrid(x, case, cube))}
    if op == "train":
        grid, _, _ = _exact_grid(x, case, cube, 0, x["n"])
        u = _exact_degrid(x, case, cube)
        vis = torch.view_as_complex(x["vis"].double())
        return {"grid": grid,
                "d_vis": torch.view_as_real(x["weight"].double() * u),
                "d_weight": (vis.conj() * u).real}
    offsets = x["offsets"] or [0, x["n"]]
    if op == "host":
        grid, norm, skipped = _exact_grid(x, case, cube, 0, x["n"])
        return {"grid": grid, "norm": float(norm), "skipped": skipped}
    parts = [_exact_grid(x, case, cube, a, b)
             for a, b in zip(offsets, offsets[1:])]
    return {"grid": torch.stack([p[0] for p in parts]),
            "norm": torch.stack([p[1] for p in parts]),
            "skipped": torch.tensor([p[2] for p in parts])}
