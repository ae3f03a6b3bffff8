"""GPU tests of calls that fill the device's memory.

A call needs its points and the sort of its records; prepared records, slots
beside degridding's points and headroom in the buffers only save time.  Where
the device has no room for those the call goes through without them, with the
same norm and skips and the same result but for rounding.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import max_rel

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


class Ballast:
    """Holds all of the device's free memory but `free` bytes."""

    def __init__(self, torch, free):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        left = torch.cuda.mem_get_info()[0] - int(free)
        self.held = torch.empty(max(left, 0), dtype=torch.uint8,
                                device="cuda")
        self.torch = torch

    def __enter__(self):
        return self

    def __exit__(self, *_):
        del self.held
        self.torch.cuda.empty_cache()


def _case(torch, pkg, synthetic, dtype, n, G, s_min, s_max):
    wl = synthetic.random_uniform_workload("memory", n, G, 16, s_min, s_max,
                                           seed=s_max)
    real = np.float64 if dtype == "d" else np.float32
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, real)).cuda()
    stack = pkg.KernelStack.from_workload(wl, dtype)
    arrs = [dev(a) for a in (wl.uu, wl.vv, wl.ww, wl.vis, wl.weight)]
    return stack, arrs, (real(wl.cell_size_rad), real(wl.w_scale), G)


@pytest.mark.parametrize("dtype,tile_u,phases,s_min,s_max", [
    ("f", 32, 1, 20, 40), ("f", 32, 4, 10, 14), ("f", 16, 1, 6, 10),
    ("f", 16, 2, 3, 7), ("f", 8, 1, 2, 4), ("d", 32, 1, 20, 40),
    ("d", 16, 1, 6, 10), ("d", 8, 2, 2, 4)])
def test_gridding_fits_its_points_and_sort(pkg, synthetic, torch, dtype,
                                           tile_u, phases, s_min, s_max):
    """24 bytes a point (FP64 32) and 16.5 a record with a quarter of headroom,
    and 64 MiB for the partial tiles of large items (with phases one for every
    later tile too) hold a gridding call, its repetition, and a smaller one."""
    n, G = 1_000_000, 2048
    stack, arrs, geometry = _case(torch, pkg, synthetic, dtype, n, G, s_min,
                                  s_max)
    tuning = {"tile_u": tile_u, "tile_phases": phases}

    def grid(plan, m):
        g = torch.zeros((G, G, 2), dtype=arrs[0].dtype, device="cuda")
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        skip = torch.zeros(1, dtype=torch.int64, device="cuda")
        pkg.grid_wproj_device(plan, stack, *(a[:m] for a in arrs), *geometry,
                              g, norm, skip)
        return g.cpu().numpy(), norm.item(), int(skip.item())

    plan = pkg.Plan()
    plan.set_tuning(tuning)
    want = {m: grid(plan, m) for m in (n // 8, n)}
    records = plan.stats()["num_records"]
    plan.close()
    plan = pkg.Plan()
    plan.set_tuning(tuning)
    real = 4 if dtype == "f" else 8
    later = (phases - 1) * (G * G + 2048 * G)   # cells of later phases' tiles
    free = 1.25 * ((16 + 2 * real) * n + 16.5 * records + 2 * real * later
                   ) + 64 * MIB
    with Ballast(torch, free + G * G * 2 * real):
        for m in (n, n, n // 8, n):
            got = grid(plan, m)
            assert got[1:] == want[m][1:]
            assert max_rel(got[0], want[m][0]) <= (1e-5 if dtype == "f"
                                                   else 1e-12)
        plan.close()


@pytest.mark.parametrize("dtype,s_min,s_max", [("f", 20, 40), ("d", 2, 8)])
def test_degridding_fits_its_points_and_sort(pkg, synthetic, torch, dtype,
                                             s_min, s_max):
    """16 bytes a point, 24.5 a record (FP64 32.5), with a quarter of headroom
    and 16 MiB: results are equal bit for bit."""
    n, G = 1_000_000, 2048
    stack, arrs, geometry = _case(torch, pkg, synthetic, dtype, n, G, s_min,
                                  s_max)
    y = torch.randn((G, G, 2), dtype=arrs[0].dtype, device="cuda")

    def degrid(plan):
        out = torch.zeros((n, 2), dtype=arrs[0].dtype, device="cuda")
        pkg.degrid_wproj_device(plan, stack, *arrs[:3], *geometry, y, out)
        return out.cpu()

    plan = pkg.Plan()
    want = degrid(plan)
    records = plan.stats()["num_records"]
    plan.close()
    plan = pkg.Plan()
    real = 4 if dtype == "f" else 8
    free = 1.25 * (16 * n + (16.5 + 2 * real) * records) + 16 * MIB
    with Ballast(torch, free + 2 * real * n):
        for _ in range(2):
            assert torch.equal(degrid(plan), want)
        plan.close()


@pytest.mark.parametrize("limit", [0, 600_000])
def test_batched_calls_and_replays_fit(pkg, synthetic, torch, limit):
    """A batched call that is short of memory, whole or in sub-batches (0.6e6
    visibilities each), and its replays: the replay of the call's own values
    gives the call's grids bit for bit."""
    n, G, c = 1_000_000, 1024, 4
    stack, arrs, geometry = _case(torch, pkg, synthetic, "f", n, G, 16, 24)
    offsets = [0, n // 10, n // 2, n // 2 + n // 20, n]

    def outputs():
        return (torch.zeros((c, G, G, 2), dtype=torch.float32, device="cuda"),
                torch.zeros(c, dtype=torch.float64, device="cuda"),
                torch.zeros(c, dtype=torch.int64, device="cuda"))

    def run(plan, f, *args):
        o = outputs()
        f(plan, stack, *args, *o)
        return [x.cpu().numpy() for x in o]

    batched = lambda p: run(p, lambda p, s, *a: pkg.grid_wproj_batched_device(
        p, s, offsets, *arrs, *geometry, *a))
    replay = lambda p: run(p, lambda p, s, g, norm, skip:
                           pkg.grid_wproj_batched_replay(p, s, arrs[3],
                                                         arrs[4], g, norm,
                                                         skip))
    plan = pkg.Plan()
    want = batched(plan)
    records = plan.stats()["num_records"]
    plan.close()
    plan = pkg.Plan()
    plan.set_batch_limit(limit)
    free = 1.25 * (32 * n + 16.5 * records) + (96 + 64 * (limit > 0)) * MIB
    with Ballast(torch, free + 4 * G * G * 8):
        for _ in range(2):
            got = batched(plan)
            again = replay(plan)
            assert np.array_equal(got[0], again[0])
            for x in (got, again):
                assert np.array_equal(x[2], want[2])
                assert np.array_equal(x[1], want[1])
                assert max_rel(x[0], want[0]) <= 1e-5
        plan.close()


@pytest.mark.parametrize("size", [4_000_000])
def test_weighting_fits_its_sort(pkg, torch, size):
    """16.6 bytes a point and a quarter of headroom, 8 MiB."""
    G = 2048
    rng = np.random.default_rng(3)
    dev = lambda a: torch.from_numpy(a.astype(np.float32)).cuda()
    uu, vv = (dev(rng.uniform(-400, 400, size)) for _ in range(2))
    w = dev(rng.uniform(0.5, 1.5, size))
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")

    def density(plan):
        g = torch.zeros((G, G), dtype=torch.float32, device="cuda")
        pkg.grid_weights_write_device(plan, uu, vv, w, 0.001, G, g, skip)
        return g.cpu()

    plan = pkg.Plan()
    want = density(plan)
    plan.close()
    plan = pkg.Plan()
    with Ballast(torch, 1.25 * 16.6 * size + 8 * MIB + 4 * G * G):
        for _ in range(2):
            assert torch.equal(density(plan), want)
        plan.close()


def test_two_calls_in_turn_leave_each_other_room(pkg, synthetic, torch):
    """A plan whose smaller call was prepared gives that memory up for a larger
    call of another kind."""
    n, G = 1_000_000, 2048
    stack, arrs, geometry = _case(torch, pkg, synthetic, "f", n, G, 20, 40)
    y = torch.randn((G, G, 2), dtype=torch.float32, device="cuda")

    def both(plan, m):
        g = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
        norm = torch.zeros(1, dtype=torch.float64, device="cuda")
        skip = torch.zeros(1, dtype=torch.int64, device="cuda")
        pkg.grid_wproj_device(plan, stack, *(a[:m] for a in arrs), *geometry,
                              g, norm, skip)
        out = torch.zeros((n, 2), dtype=torch.float32, device="cuda")
        pkg.degrid_wproj_device(plan, stack, *arrs[:3], *geometry, y, out)
        return g.cpu().numpy(), norm.item(), int(skip.item()), out.cpu()

    plan = pkg.Plan()
    want = {m: both(plan, m) for m in (n // 2, n)}
    records = plan.stats()["num_records"]
    plan.close()
    plan = pkg.Plan()
    # The buffers of the degridding call and the partial tiles of the other.
    free = 1.25 * (24 * n + 24.5 * records) + 64 * MIB
    with Ballast(torch, free + G * G * 8 + 8 * n):
        for m in (n // 2, n, n // 2):
            got = both(plan, m)
            assert got[1:3] == want[m][1:3]
            assert torch.equal(got[3], want[m][3])
            assert max_rel(got[0], want[m][0]) <= 1e-5
        plan.close()


DROP_IN = r"""
import importlib, sys
import numpy as np, torch
sys.path[:0] = [{root!r}, {root!r} + "/oracle", {root!r} + "/tests"]
import oracle
from conftest import max_rel
from test_gpu_memory import Ballast, MIB
pkg = importlib.import_module("gpu-gridding_gb300")
synthetic = importlib.import_module("gpu-gridding_gb300.synthetic")
wl = synthetic.random_uniform_workload("memory", 1_000_000, 2048, 16, 20, 40,
                                       seed=9)
want, skipped, norm = oracle.grid_f_fp64acc(wl)
records = int(sys.argv[1])
pkg.grid_f(wl.subset(1000))   # the device's stack, streams and small buffers
n, G = wl.num_points, wl.grid_size
free = 1.25 * (48 * n + 16.5 * records + 8 * G * G) + 96 * MIB
for k in range(2):
    with Ballast(torch, free) if k == 0 else open("/dev/null"):
        for _ in range(2):
            g, ns, nm = pkg.grid_f(wl)
            assert ns == skipped, (ns, skipped)
            assert abs(nm - norm) <= 1e-12 * abs(norm), (nm, norm)
            assert max_rel(g, want) <= 1e-5
            v = pkg.degrid_f(wl, g)
            if k == 0: first = v
            assert max_rel(v, first) <= 1e-5
print("fits")
"""


def test_drop_in_calls_fit(pkg, synthetic, torch):
    """The host-pointer calls, whose inputs and grid lie on the device too, in
    a process of their own (their buffers stay with it)."""
    import subprocess
    import sys
    from conftest import ROOT
    stack, arrs, geometry = _case(torch, pkg, synthetic, "f", 1_000_000, 2048,
                                  20, 40)
    plan = pkg.Plan()
    plan.set_tuning({"tile_u": 32, "tile_phases": 1})
    G = geometry[2]
    pkg.grid_wproj_device(
        plan, stack, *arrs, *geometry,
        torch.zeros((G, G, 2), dtype=torch.float32, device="cuda"),
        torch.zeros(1, dtype=torch.float64, device="cuda"),
        torch.zeros(1, dtype=torch.int64, device="cuda"))
    records = plan.stats()["num_records"]
    plan.close()
    r = subprocess.run([sys.executable, "-c", DROP_IN.format(root=ROOT),
                        str(records)], capture_output=True, text=True)
    assert r.returncode == 0 and "fits" in r.stdout, r.stdout + r.stderr
