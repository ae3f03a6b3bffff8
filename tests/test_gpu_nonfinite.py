"""GPU tests of visibilities that are infinite or not a number.

The reference adds a visibility to the cells of its footprint and no others
(oskar_grid_wproj.c:190-209), so an infinite one, or one that is not a number,
leaves every other cell as it would be without it.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import max_rel

pytestmark = pytest.mark.gpu

VALUES = [np.inf, -np.inf, np.nan]


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


def _case(synthetic, n, G, s_min, s_max, odd, seed=3):
    """A workload, the same with `odd` of its visibilities not finite, and
    their indices."""
    wl = synthetic.random_uniform_workload("odd", n, G, 16, s_min, s_max,
                                           seed=seed)
    rng = np.random.default_rng(seed)
    which = rng.choice(n, odd, replace=False)
    vis = wl.vis.copy()
    vis[which, rng.integers(0, 2, odd)] = rng.choice(VALUES, odd)
    return wl, vis, which


def _reached(pkg, torch, wl, which, prec="f"):
    """The cells that the points' footprints cover."""
    G = wl.grid_size
    dt = np.float32 if prec == "f" else np.float64
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dt)).cuda()
    place = pkg.place_wproj_device(
        pkg.KernelStack.from_workload(wl, prec), dev(wl.uu[which]),
        dev(wl.vv[which]), dev(wl.ww[which]), dt(wl.cell_size_rad),
        dt(wl.w_scale), G).cpu().numpy()
    mask = np.zeros((G, G), bool)
    for gu, gv, _, _, plane, flags in place:
        if not flags & 1:
            s = int(wl.support[plane])
            mask[gv - s:gv + s + 1, gu - s:gu + s + 1] = True
    assert mask.any()
    return mask


def _check(got, plain, mask):
    """Not finite inside the mask (one of the two components at least, both
    where a tap's own product is not a number), outside it as without the odd
    visibilities."""
    assert (~np.isfinite(got[mask])).any(axis=1).all()
    assert np.isfinite(got[~mask]).all()
    assert max_rel(got[~mask], plain[~mask]) <= 1e-5


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("tuning", [
    {}, {"tile_u": 32, "tile_phases": 1}, {"tile_u": 16, "tile_phases": 4},
    {"tile_u": 8, "tile_phases": 2, "plane_group_mb": 1}])
@pytest.mark.parametrize("n,G,s_min,s_max,odd", [
    (2, 300, 3, 7, 1), (4000, 511, 1, 5, 3), (60_000, 512, 2, 12, 2),
    (300, 256, 2, 4, 300)])
def test_odd_visibilities_stay_in_their_footprints(pkg, synthetic, torch, n,
                                                   G, s_min, s_max, odd,
                                                   tuning, prec):
    wl, vis, which = _case(synthetic, n, G, s_min, s_max, odd)
    dt = np.float32 if prec == "f" else np.float64
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dt)).cuda()
    stack = pkg.KernelStack.from_workload(wl, prec)
    rest = np.setdiff1d(np.arange(n), which)

    def grid(v, keep):
        plan = pkg.Plan()
        plan.set_tuning(tuning)
        g = torch.ones((G, G, 2), dtype=getattr(torch, np.dtype(dt).name),
                       device="cuda")
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        skip = torch.zeros(1, dtype=torch.int64, device="cuda")
        pkg.grid_wproj_device(plan, stack, dev(wl.uu[keep]), dev(wl.vv[keep]),
                              dev(wl.ww[keep]), dev(v[keep]),
                              dev(wl.weight[keep]), dt(wl.cell_size_rad),
                              dt(wl.w_scale), G, g, norm, skip)
        return g.cpu().numpy()

    _check(grid(vis, np.arange(n)), grid(wl.vis, rest),
           _reached(pkg, torch, wl, which, prec))


@pytest.mark.parametrize("mode,pinned,G", [
    ("GRID_ACCESS_COPY", False, 511), ("GRID_ACCESS_COPY", False, 4099),
    ("GRID_ACCESS_PAGEABLE", False, 511), ("GRID_ACCESS_PINNED", True, 511),
    ("GRID_ACCESS_PAGEABLE", False, 4099)])
def test_odd_visibilities_of_host_calls(pkg, synthetic, torch, mode, pinned,
                                        G):
    wl, vis, which = _case(synthetic, 20_000, G, 2, 9, 2)
    rest = np.setdiff1d(np.arange(wl.num_points), which)
    access = pkg.host_grid_access()

    def grid(v, keep):
        g = torch.empty((G, G, 2), dtype=torch.float32,
                        pin_memory=pinned).numpy()
        g[...] = 1
        pkg.oskar_grid_wproj_f(wl.num_w_planes, wl.support, wl.oversample,
                               wl.conv_size_half, wl.conv_func, len(keep),
                               wl.uu[keep], wl.vv[keep], wl.ww[keep], v[keep],
                               wl.weight[keep], wl.cell_size_rad, wl.w_scale,
                               G, g, 0.0)
        return g
    try:
        pkg.set_host_grid_access(getattr(pkg, mode))
        got, plain = grid(vis, np.arange(wl.num_points)), grid(wl.vis, rest)
    finally:
        pkg.set_host_grid_access(access)
    _check(got, plain, _reached(pkg, torch, wl, which))


@pytest.mark.parametrize("limit", [0, 3000])
def test_odd_visibilities_of_batches_and_replays(pkg, synthetic, torch,
                                                 limit):
    """Four grids; a replay with finite values has no trace of the batch's odd
    ones, and a replay brings its own."""
    n, G = 8000, 300
    wl, vis, which = _case(synthetic, n, G, 2, 6, 3)
    offsets = [0, 500, 3000, 5200, n]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    stack = pkg.KernelStack.from_workload(wl, "f")
    plan = pkg.Plan()
    plan.set_batch_limit(limit)
    args = (dev(wl.uu), dev(wl.vv), dev(wl.ww))
    geometry = (np.float32(wl.cell_size_rad), np.float32(wl.w_scale), G)
    out = lambda: (torch.zeros((4, G, G, 2), device="cuda"),
                   torch.zeros(4, dtype=torch.float64, device="cuda"),
                   torch.zeros(4, dtype=torch.int64, device="cuda"))
    without = wl.vis.copy()
    without[which] = 0

    def replay(v):
        g = out()
        pkg.grid_wproj_batched_replay(plan, stack, dev(v), dev(wl.weight), *g)
        return g[0].cpu().numpy()

    g = out()
    pkg.grid_wproj_batched_device(plan, stack, offsets, *args, dev(vis),
                                  dev(wl.weight), *geometry, *g)
    batch = g[0].cpu().numpy()
    plain, again = replay(without), replay(vis)
    assert np.isfinite(plain).all()
    for k in range(4):
        mine = which[(which >= offsets[k]) & (which < offsets[k + 1])]
        mask = (_reached(pkg, torch, wl, mine) if len(mine)
                else np.zeros((G, G), bool))
        for got in (batch[k], again[k]):
            _check(got, plain[k], mask)


def test_odd_visibilities_of_no_alloc_calls(pkg, synthetic, torch):
    from test_zz_no_alloc import _noalloc_fn
    n, G = 5000, 400
    wl, vis, which = _case(synthetic, n, G, 2, 8, 3)
    rest = np.setdiff1d(np.arange(n), which)
    fn = _noalloc_fn(pkg.lib())
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    stack = pkg.KernelStack.from_workload(wl, "f")

    def grid(v, keep):
        g = torch.zeros((G, G, 2), device="cuda")
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        skip = torch.zeros(1, dtype=torch.int64, device="cuda")
        a = [dev(x[keep]) for x in (wl.uu, wl.vv, wl.ww, v, wl.weight)]
        assert fn(stack.handle, len(keep), *(x.data_ptr() for x in a),
                  ctypes.c_float(wl.cell_size_rad), ctypes.c_float(wl.w_scale),
                  G, skip.data_ptr(), norm.data_ptr(), g.data_ptr(),
                  torch.cuda.current_stream().cuda_stream) == 0
        return g.cpu().numpy()

    _check(grid(vis, np.arange(n)), grid(wl.vis, rest),
           _reached(pkg, torch, wl, which))
