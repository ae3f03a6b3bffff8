"""GPU tests of the adjoint (degridding) kernel and the autograd binding.

* dot-product identity <G x, y> = <x, G^H y>: relative 1e-6 in FP32,
  1e-12 in FP64;
* degridding against the FP64 oracle adjoint: max-rel 1e-5 (FP32);
* torch.autograd.gradcheck in FP64 on a small case, and FP64 central
  finite differences of L = ||grid - target||^2 along a random direction on
  a 20,000-visibility subset of the synthetic-challenge shape: relative 1e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import load_golden, max_rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


def _setup(pkg, torch, wl, prec):
    dt = torch.float32 if prec == "f" else torch.float64
    cast = np.float32 if prec == "f" else float
    d = dict(
        stack=pkg.KernelStack.from_workload(wl, prec), plan=pkg.Plan(),
        uu=torch.from_numpy(wl.uu).to(dt).cuda(),
        vv=torch.from_numpy(wl.vv).to(dt).cuda(),
        ww=torch.from_numpy(wl.ww).to(dt).cuda(),
        cell=cast(wl.cell_size_rad), ws=cast(wl.w_scale), G=wl.grid_size,
        dt=dt)
    return d


def _forward(pkg, torch, s, vis, weight):
    G = s["G"]
    grid = torch.zeros((G, G, 2), dtype=s["dt"], device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    ns = torch.zeros(1, dtype=torch.int64, device="cuda")
    pkg.grid_wproj_device(s["plan"], s["stack"], s["uu"], s["vv"], s["ww"],
                          vis.contiguous(), weight.contiguous(), s["cell"],
                          s["ws"], G, grid, norm, ns)
    return grid


def _adjoint(pkg, torch, s, grid):
    out = torch.empty((s["uu"].shape[0], 2), dtype=s["dt"], device="cuda")
    pkg.degrid_wproj_device(s["plan"], s["stack"], s["uu"], s["vv"], s["ww"],
                            s["cell"], s["ws"], s["G"], grid.contiguous(),
                            out)
    return out


def _cdot(a, b):
    """Complex inner product sum(conj(a) * b) of (.., 2) real tensors."""
    re = (a[..., 0] * b[..., 0] + a[..., 1] * b[..., 1]).sum()
    im = (a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]).sum()
    return complex(re.item(), im.item())


@pytest.mark.parametrize("prec,tol,phases", [("f", 1e-6, 0), ("d", 1e-12, 0),
                                             ("f", 1e-6, 2), ("d", 1e-12, 4)])
def test_dot_product_identity(pkg, synthetic, torch, prec, tol, phases):
    """<G x, y> = <x, G^H y>, also with the gridding and the degridding on
    two and four tile phases."""
    wl = synthetic.config0().subset(60_000)
    s = _setup(pkg, torch, wl, prec)
    s["plan"].set_tuning({"tile_phases": phases})
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((wl.num_points, 2), generator=g, device="cuda",
                    dtype=s["dt"])
    y = torch.randn((wl.grid_size, wl.grid_size, 2), generator=g,
                    device="cuda", dtype=s["dt"])
    ones = torch.ones(wl.num_points, dtype=s["dt"], device="cuda")
    gx = _forward(pkg, torch, s, x, ones)
    ghy = _adjoint(pkg, torch, s, y)
    lhs = _cdot(gx.double(), y.double())
    rhs = _cdot(x.double(), ghy.double())
    rel = abs(lhs - rhs) / abs(lhs)
    print(f"dot-product test ({prec}): relative mismatch {rel:.2e}")
    assert rel <= tol


def test_dot_product_identity_cfg1_shape(pkg, synthetic, torch):
    """The FP32 dot-product identity on the whole synthetic-challenge shape
    the gridding/degridding pair is stated on (2,152,800 visibilities,
    8192^2 grid, 714 w-planes, support 4..36): relative 1e-6."""
    wl = synthetic.config1()
    s = _setup(pkg, torch, wl, "f")
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn((wl.num_points, 2), generator=g, device="cuda",
                    dtype=torch.float32)
    y = torch.randn((wl.grid_size, wl.grid_size, 2), generator=g,
                    device="cuda", dtype=torch.float32)
    ones = torch.ones(wl.num_points, dtype=torch.float32, device="cuda")
    gx = _forward(pkg, torch, s, x, ones)
    ghy = _adjoint(pkg, torch, s, y)
    lhs = _cdot(gx.double(), y.double())
    rhs = _cdot(x.double(), ghy.double())
    rel = abs(lhs - rhs) / abs(lhs)
    print(f"dot-product test (cfg1 shape, FP32): relative mismatch "
          f"{rel:.2e}")
    assert rel <= 1e-6


@pytest.mark.parametrize("phases", [0, 1, 2, 4])
def test_degrid_matches_fp64_oracle(pkg, oracle_mod, torch, phases):
    wl, _ = load_golden("small_f")
    s = _setup(pkg, torch, wl, "f")
    s["plan"].set_tuning({"tile_phases": phases})
    rng = np.random.default_rng(3)
    y = rng.standard_normal((wl.grid_size, wl.grid_size, 2))
    out = _adjoint(pkg, torch, s, torch.from_numpy(
        y.astype(np.float32)).cuda()).cpu().numpy()
    ref = oracle_mod.degrid_fp64(wl, y.astype(np.float32).astype(np.float64))
    assert max_rel(out, ref) <= 1e-5
    p = oracle_mod.place(wl)
    assert not out[p["skipped"] == 1].any()   # skipped points get 0


def test_gradcheck_fp64_small(pkg, synthetic, torch):
    wl = synthetic.random_uniform_workload("gc", 40, 48, 6, 1, 4, seed=9,
                                           cell_size_rad=4e-3)
    s = _setup(pkg, torch, wl, "d")
    vis = torch.from_numpy(wl.vis).double().cuda().requires_grad_(True)
    w = torch.from_numpy(wl.weight).double().cuda().requires_grad_(True)

    def fn(v, ww):
        return pkg.GridWproj.apply(v, ww, s["uu"], s["vv"], s["ww"],
                                   s["stack"], s["plan"], s["cell"], s["ws"],
                                   s["G"])

    assert torch.autograd.gradcheck(fn, (vis, w), eps=1e-6, atol=1e-8,
                                    rtol=1e-6, fast_mode=True)


def test_finite_differences_fp64_cfg1_subset(pkg, synthetic, torch):
    """Central differences of L = ||grid - target||^2 along a random
    direction in (vis, weight) on 20,000 visibilities of the
    synthetic-challenge shape, against the autograd gradient."""
    wl = synthetic.config1().subset(20_000)
    s = _setup(pkg, torch, wl, "d")
    gen = torch.Generator(device="cuda").manual_seed(4)
    vis0 = torch.from_numpy(wl.vis).double().cuda()
    w0 = torch.from_numpy(wl.weight).double().cuda()
    target = torch.randn((wl.grid_size, wl.grid_size, 2), generator=gen,
                         device="cuda", dtype=torch.float64) * 1e-3
    dv = torch.randn(vis0.shape, generator=gen, device="cuda",
                     dtype=torch.float64)
    dw = torch.randn(w0.shape, generator=gen, device="cuda",
                     dtype=torch.float64)

    def loss(v, w):
        g = pkg.GridWproj.apply(v, w, s["uu"], s["vv"], s["ww"], s["stack"],
                                s["plan"], s["cell"], s["ws"], s["G"])
        return ((g - target) ** 2).sum()

    v = vis0.clone().requires_grad_(True)
    w = w0.clone().requires_grad_(True)
    L = loss(v, w)
    L.backward()
    analytic = (v.grad * dv).sum().item() + (w.grad * dw).sum().item()
    h = 1e-4
    with torch.no_grad():
        lp = loss(vis0 + h * dv, w0 + h * dw).item()
        lm = loss(vis0 - h * dv, w0 - h * dw).item()
    numeric = (lp - lm) / (2 * h)
    rel = abs(numeric - analytic) / abs(analytic)
    print(f"finite differences: analytic {analytic:.9e} numeric "
          f"{numeric:.9e} rel {rel:.2e}")
    assert rel <= 1e-6


def test_degrid_fp64_matches_fp64_oracle(pkg, oracle_mod, synthetic, torch):
    """FP64 degridding against the FP64 adjoint (FP64 placement and cube)."""
    wl = synthetic.random_uniform_workload("degrid_d", 3_000, 512, 16, 2, 10,
                                           seed=21, cell_size_rad=8e-5)
    s = _setup(pkg, torch, wl, "d")
    rng = np.random.default_rng(5)
    y = rng.standard_normal((wl.grid_size, wl.grid_size, 2))
    out = _adjoint(pkg, torch, s, torch.from_numpy(y).cuda()).cpu().numpy()
    ref = oracle_mod.degrid_d(wl, y)
    assert max_rel(out, ref) <= 1e-12
    p = oracle_mod.place(wl, "d")
    assert p["num_skipped"] < wl.num_points
    assert not out[p["skipped"] == 1].any()


DEGRID_TUNINGS = [{"plane_group_mb": 1}, {"items_per_cta": 1},
                  {"items_per_cta": 64}, {"sort_detail": 0},
                  {"sort_detail": 1, "ctas_per_sm": 1}]


def test_degrid_bit_identical_across_tunings(pkg, synthetic, torch):
    """Each record's partial result is formed the same way whichever CTA
    takes it, and each visibility adds its records in emission order, so
    plane groups, work-item splitting, record order and CTA count leave
    the output bit for bit unchanged (tile phases change which tiles a
    visibility's sum is cut into, so they are held at the default)."""
    wl = synthetic.config0().subset(40_000)
    s = _setup(pkg, torch, wl, "f")
    g = torch.Generator(device="cuda").manual_seed(7)
    y = torch.randn((wl.grid_size, wl.grid_size, 2), generator=g,
                    device="cuda", dtype=torch.float32)
    base = _adjoint(pkg, torch, s, y).cpu().numpy()
    again = _adjoint(pkg, torch, s, y).cpu().numpy()
    assert np.array_equal(base.view(np.uint32), again.view(np.uint32))
    for t in DEGRID_TUNINGS:
        plan = pkg.Plan()
        plan.set_tuning(t)
        s2 = dict(s, plan=plan)
        got = _adjoint(pkg, torch, s2, y).cpu().numpy()
        if t.get("plane_group_mb") == 1:
            assert plan.stats()["num_plane_groups"] > 1
        assert np.array_equal(got.view(np.uint32), base.view(np.uint32)), t


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("n,size,s_min,s_max,phases", [
    (30, 200, 2, 6, 1),          # less than one unit of records
    (600, 2048, 4, 20, 0),       # a record or two a tile
    (5_000, 333, 31, 41, 4),     # footprints wider than a tile and phases
    (900_000, 512, 1, 3, 0),     # every unit length, tiles of many units
    (20_000, 1000, 2, 16, 2)])   # units across several tiles
def test_degrid_units(pkg, oracle_mod, synthetic, torch, prec, n, size, s_min,
                      s_max, phases):
    """Degridding over units of records shorter and longer than a tile's, with
    grid values per tile and per record.  Each result passes at most 36 rounded
    additions in FP32 (8 rows, 5 lane steps, 8 bands, up to 15 records) and 150
    in FP64 (128 cells of a lane, 5 lane steps, up to 15 records); the sum of
    its terms' moduli is taken as up to 2 s_max + 1 times the largest result,
    as for terms of random phase."""
    wl = synthetic.random_uniform_workload("units", n, size, 16, s_min, s_max,
                                           seed=n)
    s = _setup(pkg, torch, wl, prec)
    s["plan"].set_tuning({"tile_phases": phases})
    rng = np.random.default_rng(n)
    y = rng.standard_normal((wl.grid_size, wl.grid_size, 2)).astype(np.float32)
    out = _adjoint(pkg, torch, s, torch.from_numpy(y).cuda().to(s["dt"]))
    oracle = oracle_mod.degrid_fp64 if prec == "f" else oracle_mod.degrid_d
    tol = 36 * 2.0**-24 if prec == "f" else 150 * 2.0**-53
    assert max_rel(out.cpu().numpy(), oracle(wl, y.astype(np.float64))) <= \
        tol * (2 * s_max + 1)


@pytest.mark.parametrize("n,size", [(20_000, 8192), (4_000, 4099)])
def test_gridding_and_degridding_in_turn_on_one_plan(pkg, synthetic, torch, n,
                                                     size):
    """A plan that grids (one tile phase) and degrids (four) in turn, as a
    training step does, gives what plans of their own give, in about their
    time: nothing that depends on the geometry is worked out anew each time.
    (The margin is half as much again and 0.2 ms: the tiles' order alone took
    a millisecond a call.)"""
    wl = synthetic.random_uniform_workload("turns", n, size, 32, 2, 8, seed=n)
    G = wl.grid_size
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    stack = pkg.KernelStack.from_workload(wl, "f")
    uvw = (dev(wl.uu), dev(wl.vv), dev(wl.ww))
    vis, weight = dev(wl.vis), dev(wl.weight)
    geometry = (np.float32(wl.cell_size_rad), np.float32(wl.w_scale), G)
    grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")
    y = dev(np.random.default_rng(1).standard_normal((G, G, 2),
                                                     dtype=np.float32))

    def step(forward, backward):
        out = torch.empty((n, 2), dtype=torch.float32, device="cuda")
        grid.zero_()
        pkg.grid_wproj_device(forward, stack, *uvw, vis, weight, *geometry,
                              grid, norm, skip)
        pkg.degrid_wproj_device(backward, stack, *uvw, *geometry, y, out)
        return grid.cpu(), out.cpu()

    def ms(forward, backward):
        best = float("inf")
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            for _ in range(4):
                grid.zero_()
                pkg.grid_wproj_device(forward, stack, *uvw, vis, weight,
                                      *geometry, grid, norm, skip)
                pkg.degrid_wproj_device(backward, stack, *uvw, *geometry, y,
                                        out)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) / 4)
        return best

    out = torch.empty((n, 2), dtype=torch.float32, device="cuda")
    one, two, three = pkg.Plan(), pkg.Plan(), pkg.Plan()
    for _ in range(2):
        for got, want in zip(step(one, one), step(two, three)):
            assert torch.equal(got, want)
    assert ms(one, one) <= 1.5 * ms(two, three) + 0.2


@pytest.mark.parametrize("s_min,s_max", [(4, 12), (30, 60)])
def test_degrid_fp64_rounding(pkg, synthetic, torch, s_min, s_max):
    """FP64 degridding's rounding stays that of short chains: eight of a lane's
    cells, at most eight such sums, the five steps of the warp's sum and a
    visibility's few tiles add, as random signs do, some sqrt(8/2 + 8/2 + 5 +
    4) = 4.1 roundings of 0.58 units each, 2.4 units of 2^-53.  One chain over
    both products of a lane's forty cells on the wide footprints would add
    sqrt(80/2 + 5 + 4) of them, 4.1 units.  The root mean square over the
    visibilities, against sums in extended precision, lies below the geometric
    mean of the two, 3.1."""
    n, G = 400, 512
    wl = synthetic.random_uniform_workload("rounding", n, G, 16, s_min, s_max,
                                           seed=s_max)
    s = _setup(pkg, torch, wl, "d")
    y = np.random.default_rng(7).standard_normal((G, G, 2))
    out = _adjoint(pkg, torch, s, torch.from_numpy(y).cuda()).cpu().numpy()
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).double().cuda()
    place = pkg.place_wproj_device(
        pkg.KernelStack.from_workload(wl, "d"), dev(wl.uu), dev(wl.vv),
        dev(wl.ww), float(wl.cell_size_rad), float(wl.w_scale),
        G).cpu().numpy()
    err = total = 0.0
    for i, (gu, gv, ou, ov, plane, flags) in enumerate(place):
        if flags & 1:
            assert not out[i].any()
            continue
        sup = int(wl.support[plane])
        k = np.arange(-sup, sup + 1)
        t = wl.conv_func[plane][np.abs(ov + k * wl.oversample)[:, None],
                                np.abs(ou + k * wl.oversample)[None, :]]
        t = t.astype(np.longdouble)
        g = y[gv - sup:gv + sup + 1, gu - sup:gu + sup + 1].astype(
            np.longdouble)
        im = -t[..., 1] if flags & 2 else t[..., 1]
        re = (t[..., 0] * g[..., 0] + im * g[..., 1]).sum()
        ima = (t[..., 0] * g[..., 1] - im * g[..., 0]).sum()
        err += float((out[i, 0] - re) ** 2 + (out[i, 1] - ima) ** 2)
        total += float(re * re + ima * ima)
    assert np.sqrt(err / total) <= 3.1 * 2.0**-53
