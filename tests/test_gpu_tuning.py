"""GPU tests of the plan's tuning settings and of the autotuner.

Every setting changes speed only: num_skipped and norm stay identical to
the default plan's, the grid stays within 1e-5 (max |err| / max |grid|) of
the FP64-accumulating oracle.  The autotuner applies what it found, stores
it in its cache and takes it from there on the next call.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import pytest

from conftest import max_rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


@pytest.fixture(scope="module")
def wl(synthetic):
    """60,000 visibilities on a 1024^2 grid, 32 planes, support 2..16."""
    return synthetic.random_uniform_workload("tuning_1024", 60_000, 1024, 32,
                                             2, 16, seed=7)


@pytest.fixture(scope="module")
def fp64(oracle_mod, wl):
    return oracle_mod.grid_f_fp64acc(wl)


def _grid(pkg, torch, wl, plan, stack):
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    G = wl.grid_size
    grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")
    pkg.grid_wproj_device(plan, stack, dev(wl.uu), dev(wl.vv), dev(wl.ww),
                          dev(wl.vis), dev(wl.weight),
                          np.float32(wl.cell_size_rad), np.float32(wl.w_scale),
                          G, grid, norm, skip)
    torch.cuda.synchronize()
    return grid.cpu().numpy(), float(norm.item()), int(skip.item())


TUNINGS = [
    {"tile_u": 32, "slice_staging": 1, "items_per_cta": 1, "sort_detail": 2},
    {"tile_u": 16, "slice_staging": 0, "items_per_cta": 16, "sort_detail": 1},
    {"tile_u": 8, "slice_staging": 1, "items_per_cta": 64, "sort_detail": 0},
    {"tile_u": 0, "slice_staging": -1, "items_per_cta": 8, "ctas_per_sm": 1},
    {"tile_u": 32, "slice_staging": 0, "items_per_cta": 4, "plane_group_mb": 1},
    {"tile_u": 8, "slice_staging": 1, "items_per_cta": 2, "plane_group_mb": 1},
    {"tile_u": 32, "slice_staging": 0, "items_per_cta": 4, "tile_order": 1},
    {"tile_u": 16, "slice_staging": 0, "items_per_cta": 2, "plane_group_mb": 1,
     "tile_order": 1},
    {"tile_u": 32, "slice_staging": 0, "items_per_cta": 4, "lane_groups": 1},
    {"tile_u": 32, "slice_staging": 0, "items_per_cta": 2, "lane_groups": 2,
     "plane_group_mb": 1},
    {"tile_u": 32, "slice_staging": 0, "items_per_cta": 4, "tile_phases": 2},
    {"tile_u": 32, "slice_staging": 1, "items_per_cta": 8, "tile_phases": 4,
     "plane_group_mb": 1},
    {"tile_u": 16, "slice_staging": 0, "items_per_cta": 2, "tile_phases": 4},
    {"tile_u": 8, "slice_staging": 1, "items_per_cta": 4, "tile_phases": 2,
     "plane_group_mb": 1},
    {"tile_u": 32, "slice_staging": 0, "items_per_cta": 2, "lane_groups": 2,
     "tile_phases": 2},
    {"tile_u": 32, "slice_staging": 0, "items_per_cta": 4, "tile_phases": 8},
    {"tile_u": 8, "slice_staging": 0, "items_per_cta": 4, "tile_phases": 8,
     "plane_group_mb": 1},
]


@pytest.mark.parametrize("tuning", TUNINGS)
def test_tuning_changes_speed_only(pkg, torch, wl, fp64, tuning):
    stack = pkg.KernelStack.from_workload(wl, "f")
    base = _grid(pkg, torch, wl, pkg.Plan(), stack)
    plan = pkg.Plan()
    plan.set_tuning(tuning)
    got = _grid(pkg, torch, wl, plan, stack)
    st = plan.stats()
    if tuning["tile_u"]:
        assert st["tile_u"] == tuning["tile_u"]
    if tuning.get("plane_group_mb") == 1:
        assert st["num_plane_groups"] > 1
    else:
        assert st["num_plane_groups"] == 1
    if tuning.get("ctas_per_sm") == 1:
        assert st["num_ctas"] == torch.cuda.get_device_properties(
            0).multi_processor_count
    assert got[2] == base[2] == fp64[1]
    assert got[1] == base[1]
    assert max_rel(got[0], fp64[0]) <= 1e-5


def test_tuning_rejects_bad_values(pkg, torch):
    plan = pkg.Plan()
    before = plan.tuning()
    for bad in ({"tile_u": 12}, {"slice_staging": 2}, {"items_per_cta": 0},
                {"items_per_cta": 65}, {"sort_detail": 3},
                {"ctas_per_sm": -1}, {"tile_order": 2}, {"lane_groups": 3},
                {"tile_phases": 3}, {"tile_phases": 16}):
        with pytest.raises(pkg.GridError):
            plan.set_tuning(bad)
        assert plan.tuning() == before


def test_autotune_applies_and_caches(pkg, torch, wl, fp64, tmp_path):
    at = importlib.import_module(pkg.__name__ + ".autotune")
    cache = at.TuningCache(str(tmp_path / "tuning.json"))
    stack = pkg.KernelStack.from_workload(wl, "f")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = (dev(wl.uu), dev(wl.vv), dev(wl.ww), dev(wl.vis), dev(wl.weight),
            wl.cell_size_rad, wl.w_scale, wl.grid_size)
    plan = pkg.Plan()
    r1 = at.autotune(pkg, plan, stack, *args, cache=cache, steps=1)
    assert r1["cached"] is False and r1["trials"] >= 10
    applied = plan.tuning()
    assert applied == {k: r1[k] for k in at.DEFAULT_TUNING}
    got = _grid(pkg, torch, wl, plan, stack)
    assert got[2] == fp64[1]
    assert max_rel(got[0], fp64[0]) <= 1e-5
    plan2 = pkg.Plan()
    r2 = at.autotune(pkg, plan2, stack, *args,
                     cache=at.TuningCache(cache.path))
    assert r2["cached"] is True and plan2.tuning() == applied


def test_plane_groups_deterministic(pkg, torch, wl):
    """Gridding in several plane-group passes is reproducible bit for bit."""
    stack = pkg.KernelStack.from_workload(wl, "f")
    plan = pkg.Plan()
    plan.set_tuning({"plane_group_mb": 1})
    a = _grid(pkg, torch, wl, plan, stack)
    b = _grid(pkg, torch, wl, plan, stack)
    assert plan.stats()["num_plane_groups"] > 1
    assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))


def test_host_tuning_applies_to_dropin(pkg, torch, wl, fp64):
    """The host-pointer entry points take a tuning like a plan does: the
    getter returns it, results stay within the bars, and None restores the
    defaults."""
    default = pkg.host_tuning()
    tuned = {"tile_u": 16, "slice_staging": 0, "items_per_cta": 8,
             "sort_detail": 1, "ctas_per_sm": 0, "plane_group_mb": 1,
             "tile_order": 1, "lane_groups": 1, "tile_phases": 2}
    try:
        pkg.set_host_tuning(tuned)
        assert pkg.host_tuning() == tuned
        g, ns, nm = pkg.grid_f(wl)
        assert ns == fp64[1]
        assert max_rel(g, fp64[0]) <= 1e-5
        with pytest.raises(pkg.GridError):
            pkg.set_host_tuning({"items_per_cta": 0})
        assert pkg.host_tuning() == tuned
    finally:
        pkg.set_host_tuning(None)
    assert pkg.host_tuning() == default
    g2, ns2, nm2 = pkg.grid_f(wl)
    assert ns2 == ns and nm2 == nm


@pytest.mark.parametrize("tile_u", [32, 16, 8])
def test_stack_beyond_4_gib(pkg, torch, tile_u):
    """A stack whose taps pass 4 GiB (64-bit tap offsets in the kernels)
    grids and degrids bit for bit like a small one with the same kernels:
    every plane of both has the same support and chirp, and all points fall
    on the last."""
    G, s, n = 512, 100, 600
    rng = np.random.default_rng(3)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    uu, vv = (dev(rng.uniform(-130.0, 130.0, n)) for _ in range(2))
    ww = dev(np.full(n, 1.0e6) * rng.choice([-1.0, 1.0], n))
    vis, weight = dev(rng.standard_normal((n, 2))), dev(rng.uniform(1, 2, n))
    y = dev(rng.standard_normal((G, G, 2)))
    outs = []
    for planes in (2, 1500):
        stack = pkg.KernelStack.generate(
            planes, np.full(planes, s, np.int32), 4, 4 * (s + 1),
            np.full(planes, 3.0))
        plan = pkg.Plan()
        plan.set_tuning({"tile_u": tile_u, "plane_group_mb": 1048576})
        grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        skip = torch.zeros(1, dtype=torch.int64, device="cuda")
        pkg.grid_wproj_device(plan, stack, uu, vv, ww, vis, weight, 0.002,
                              np.float32(1.0e6), G, grid, norm, skip)
        out = torch.empty((n, 2), dtype=torch.float32, device="cuda")
        pkg.degrid_wproj_device(plan, stack, uu, vv, ww, 0.002,
                                np.float32(1.0e6), G, y, out)
        outs.append([t.cpu().numpy() for t in (grid, norm, skip, out)])
        del stack
    assert int(outs[0][2][0]) < n // 2 and np.abs(outs[0][0]).max() > 0
    for a, b in zip(*outs):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("tuning", [
    {"tile_u": 32, "tile_phases": 1}, {"tile_u": 32, "tile_phases": 4},
    {"tile_u": 16, "items_per_cta": 64}, {"tile_u": 8, "tile_phases": 2},
    {"tile_u": 32, "tile_phases": 2, "plane_group_mb": 1}])
@pytest.mark.parametrize("s_min,s_max", [(1, 2), (3, 17), (31, 48)])
def test_fp64_footprints_packed_over_lanes(pkg, oracle_mod, synthetic, torch,
                                           s_min, s_max, tuning):
    """FP64 gridding packs each footprint's cells inside a band over the
    lanes: footprints below, at and above a tile's width and a band's height,
    over every tile shape.  A cell sums at most n = 4000 visibilities, on each
    side in n rounded steps of partial sums no larger than the grid's maximum:
    2 n 2^-53 < 1e-12 of it."""
    n = 4000
    wl = synthetic.random_uniform_workload("packed", n, 512, 24, s_min, s_max,
                                           seed=s_max)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).double().cuda()
    G = wl.grid_size
    plan = pkg.Plan()
    plan.set_tuning(tuning)
    grid = torch.zeros((G, G, 2), dtype=torch.float64, device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")
    pkg.grid_wproj_device(plan, pkg.KernelStack.from_workload(wl, "d"),
                          dev(wl.uu), dev(wl.vv), dev(wl.ww), dev(wl.vis),
                          dev(wl.weight), float(wl.cell_size_rad),
                          float(wl.w_scale), G, grid, norm, skip)
    want, skipped, _ = oracle_mod.grid_d(wl)
    assert int(skip.item()) == skipped
    assert max_rel(grid.cpu().numpy(), want) <= 1e-12


@pytest.mark.parametrize("phases", [1, 4])
@pytest.mark.parametrize("chunks", [1, 2, 15, 16, 17, 41])
def test_chunks_of_one_tile(pkg, oracle_mod, synthetic, torch, chunks,
                            phases):
    """A tile cut into `chunks` chunks of 64 records, whose partial sums are
    added sixteen at a time as (hi, lo) pairs: below, at and above one and two
    such groups.  Each partial is rounded once, the products of weights and
    visibilities once, the sum once: 3 * 2^-24 of the sum of moduli, here up to
    5 times the largest cell."""
    wl = synthetic.random_uniform_workload("chunks", 64 * chunks, 256, 4, 2, 3,
                                           seed=chunks)
    # All centres inside the tile to the right of and above the grid's centre.
    extent = 1.0 / wl.cell_size_rad / 256
    rng = np.random.default_rng(chunks)
    wl.uu[:] = rng.uniform(12.0, 20.0, wl.num_points) * extent
    wl.vv[:] = rng.uniform(12.0, 20.0, wl.num_points) * extent
    plan = pkg.Plan()
    plan.set_tuning({"tile_u": 32, "tile_phases": phases})
    got = _grid(pkg, torch, wl, plan, pkg.KernelStack.from_workload(wl, "f"))
    want = oracle_mod.grid_f_fp64acc(wl)
    assert plan.stats()["chunk_records"] == 64
    assert got[2] == want[1] == 0
    assert max_rel(got[0], want[0]) <= 3 * 2.0**-24 * 5


@pytest.mark.parametrize("n,top,groups", [
    (20_000, 600, 4),      # planes used evenly: the whole stack of 350 MB
    (20_000, 120, 1),      # the lowest fifth: 5.6 MB
    (300, 600, 3),         # 245 MB
    (1, 1, 1),
    (5_000, 0, 1)])        # all outside the grid: none used
def test_plane_groups_by_use(pkg, torch, n, top, groups):
    """The automatic number of plane groups follows the bytes of the planes
    that the points use, and changes the grid by rounding only (the tuning
    tests' bound)."""
    G, planes = 512, 601
    sup = np.rint(np.linspace(4, 72, planes)).astype(np.int32)
    stack = pkg.KernelStack.generate(planes, sup, 4, 4 * 73,
                                     np.full(planes, 3.0))
    rng = np.random.default_rng(n + top)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    far = 1e6 if top == 0 else 1.0
    uu, vv = (dev(far * rng.uniform(60.0, 150.0, n)) for _ in range(2))
    p = np.rint(top * np.sqrt(rng.random(n)))
    args = (stack, uu, vv, dev(p * p), dev(rng.standard_normal((n, 2))),
            dev(rng.uniform(1, 2, n)), 0.002, np.float32(1.0), G)
    outs = []
    for tuning in ({}, {"plane_group_mb": 1048576}):
        plan = pkg.Plan()
        plan.set_tuning(tuning)
        grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        skip = torch.zeros(1, dtype=torch.int64, device="cuda")
        pkg.grid_wproj_device(plan, *args, grid, norm, skip)
        outs.append((grid.cpu().numpy(), float(norm.item()),
                     int(skip.item()), plan.stats()["num_plane_groups"]))
    assert outs[0][3] == groups and outs[1][3] == 1
    assert outs[0][1:3] == outs[1][1:3]
    if outs[0][2] < n:
        assert max_rel(outs[0][0], outs[1][0]) <= 1e-5


@pytest.mark.parametrize("phases", [1, 4])
@pytest.mark.parametrize("start,parts", [
    (0.0, [2.0**28, 2.0**-23, 15.0, -2.0**28, -15.0]),
    (-15.0, [2.0**28] * 17 + [2.0**-23, 15.0] + [-2.0**28] * 17),
    (3e38, [3e38, -3e38]),
    (1.0, [3e38, 3e38, -3e38, -3e38]),
    (2e38, [2e38, 1.0]),
    (float("inf"), [1.0, 2.0]),
    (float("inf"), [-3e38] * 17)])
def test_chunk_sums_keep_fp64_range_and_bits(pkg, torch, start, parts, phases):
    """A tile's partial sums are added to the grid with an FP64 sum's range
    and no fewer bits, then rounded once: each chunk's first record brings one
    of `parts`, and the cell is no further from the exact sum than FP64
    additions in chunk order leave it."""
    G, n = 256, 64 * len(parts)
    cube = torch.zeros((1, 2, 2, 2), dtype=torch.float32, device="cuda")
    cube[0, 0, 0, 0] = 1.0
    stack = pkg.KernelStack(1, np.zeros(1, np.int32), 1, 2, cube, "f")
    vis = torch.zeros((n, 2), dtype=torch.float32, device="cuda")
    p = torch.tensor(parts, dtype=torch.float32, device="cuda")
    vis[::64, 0], vis[::64, 1] = p, -p
    at = lambda v: torch.full((n,), float(v), device="cuda")
    plan = pkg.Plan()
    plan.set_tuning({"tile_u": 32, "tile_phases": phases})
    grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
    grid[G // 2 + 5, G // 2 + 3, 0] = start
    grid[G // 2 + 5, G // 2 + 3, 1] = -start
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")
    pkg.grid_wproj_device(plan, stack, at(-3), at(5), at(0), vis, at(1),
                          np.float32(1 / G), np.float32(1.0), G, grid, norm,
                          skip)
    assert plan.stats()["chunk_records"] == 64
    want = np.float64(np.float32(start))
    for x in parts:
        want += np.float64(np.float32(x))
    with np.errstate(over="ignore"):
        want = np.float32(want)
    exact = math.fsum([start] + parts)
    got = grid.cpu().numpy()
    re, im = got[G // 2 + 5, G // 2 + 3]
    assert re == -im
    assert re == want or abs(re - exact) <= abs(want - exact)
    got[G // 2 + 5, G // 2 + 3] = 0
    assert not got.any()


def _auto_groups(pkg, torch, planes, s_min, s_max, plane, seed=1):
    """Plane groups of a default call whose points use the given planes."""
    sup = np.rint(np.linspace(s_min, s_max, planes)).astype(np.int32)
    stack = pkg.KernelStack.generate(planes, sup, 4, 4 * (s_max + 1),
                                     np.full(planes, 3.0))
    G, n = 512, len(plane)
    rng = np.random.default_rng(seed)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    uu, vv = (dev(rng.uniform(-50.0, 50.0, n)) for _ in range(2))
    p = np.asarray(plane, np.float64)
    grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")
    plan = pkg.Plan()
    pkg.grid_wproj_device(plan, stack, uu, vv, dev(p * p),
                          dev(rng.standard_normal((n, 2))),
                          dev(rng.uniform(1, 2, n)), 0.002, np.float32(1.0),
                          G, grid, norm, skip)
    return plan.stats()["num_plane_groups"]


@pytest.mark.parametrize("planes,s_min,s_max,lowest,mb", [
    (200, 4, 72, 170, 41),     # of 118 MB
    (128, 60, 100, 109, 55),   # of 257 MB
    (128, 60, 100, 0, None),   # all
    (300, 40, 72, 0, None)])   # all, more planes than bins
def test_plane_groups_of_few_planes(pkg, torch, planes, s_min, s_max, lowest,
                                    mb):
    """The bytes in use of stacks with fewer planes than the sample has bins,
    whose upper planes the points use, make the groups: three quarters of L2
    each."""
    p = np.random.default_rng(planes).integers(lowest, planes, 20_000)
    if mb is None:   # 7 + 9 * (2 s + 8) rows of 2 s + 2 taps a plane
        sup = np.rint(np.linspace(s_min, s_max, planes))
        mb = float(np.sum(8 * (7 + 9 * (2 * sup + 8)) * (2 * sup + 2))) / 1e6
    budget = torch.cuda.get_device_properties(0).L2_cache_size // 4 * 3
    assert _auto_groups(pkg, torch, planes, s_min, s_max,
                        p) == math.ceil(mb * 1e6 / budget)


@pytest.mark.parametrize("baselines", [1, 8, 64])
def test_plane_groups_of_time_major_points(pkg, torch, baselines):
    """The sample behind the automatic groups meets every baseline where their
    number divides the stride of 8192 samples in time-major points: the first
    baseline has w = 0, the others use the stack's 350 MB evenly."""
    times = 64 * 8192 // baselines
    rng = np.random.default_rng(baselines)
    p = np.rint(600 * np.sqrt(rng.random((times, baselines))))
    p[:, 0] = 0 if baselines > 1 else p[:, 0]
    p = p.reshape(-1)
    got = _auto_groups(pkg, torch, 601, 4, 72, p)
    assert got == _auto_groups(pkg, torch, 601, 4, 72, rng.permutation(p)) == 4


@pytest.mark.parametrize("top,planes_mb,by_plane", [
    (600, 1048576, True),    # 350 MB in one pass
    (600, 300, True),        # 175 MB a pass
    (120, 1048576, False),   # 5.6 MB in use
    (600, 0, True)])         # four groups
def test_record_order_follows_the_cache(pkg, torch, top, planes_mb, by_plane):
    """sort_detail 2 orders a tile's records by plane where there are three
    plane groups or more, or a pass's slices leave the cache: the launches are
    those of sort_detail 1 (more key bits, so more sorting passes), else those
    of sort_detail 0, and so is the grid, bit for bit."""
    G, n = 2048, 20_000
    sup = np.rint(np.linspace(4, 72, 601)).astype(np.int32)
    stack = pkg.KernelStack.generate(601, sup, 4, 4 * 73, np.full(601, 3.0))
    rng = np.random.default_rng(top)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    uu, vv = (dev(rng.uniform(-200.0, 200.0, n)) for _ in range(2))
    p = np.rint(top * np.sqrt(rng.random(n)))
    args = (stack, uu, vv, dev(p * p), dev(rng.standard_normal((n, 2))),
            dev(rng.uniform(1, 2, n)), 0.002, np.float32(1.0), G)
    outs = []
    for detail in (2, 1 if by_plane else 0):
        plan = pkg.Plan()
        plan.set_tuning({"plane_group_mb": planes_mb, "sort_detail": detail})
        grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        skip = torch.zeros(1, dtype=torch.int64, device="cuda")
        pkg.grid_wproj_device(plan, *args, grid, norm, skip)
        outs.append((plan.stats()["num_launches"], grid))
    assert outs[0][0] == outs[1][0]
    assert torch.equal(outs[0][1], outs[1][1])


def test_ctas_per_sm_counts_eight_warps(pkg, torch):
    """ctas_per_sm caps teams of eight warps, the warps of a tile's bands: two
    an SM are sixteen warps where twenty fit, so a call takes at most 20 / 16 of
    the time and 0.1 ms, and one an SM at most 20 / 8."""
    G, n, planes = 2048, 200_000, 64
    sup = np.rint(np.linspace(20, 72, planes)).astype(np.int32)
    stack = pkg.KernelStack.generate(planes, sup, 4, 4 * 73,
                                     np.full(planes, 3.0))
    rng = np.random.default_rng(5)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    uu, vv = (dev(rng.uniform(-200.0, 200.0, n)) for _ in range(2))
    p = rng.integers(0, planes, n).astype(np.float64)
    args = (stack, uu, vv, dev(p * p), dev(rng.standard_normal((n, 2))),
            dev(rng.uniform(1, 2, n)), 0.002, np.float32(1.0), G)
    grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def ms(ctas):
        plan = pkg.Plan()
        plan.set_tuning({"ctas_per_sm": ctas})
        best = float("inf")
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            pkg.grid_wproj_device(plan, *args, grid, norm, skip)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        teams = plan.stats()["num_ctas"]
        assert teams <= (ctas or 32) * sms and teams >= sms
        return best

    free = ms(0)
    assert ms(2) <= 1.25 * free + 0.1
    assert ms(1) <= 2.5 * free + 0.1
