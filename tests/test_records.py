"""Record positions past 2^31: a call has up to 2^32 - 16 (visibility, tile)
records, so the positions that work items hold take all 32 bits."""
from __future__ import annotations

import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CUT = r"""
#include <cstdio>
#include <cstdlib>
#include "gg_common.cuh"
// argv: tile's first record, records, chunk -> chunks, then each item's range
int main(int, char** v) {
  const uint32_t begin = (uint32_t)strtoull(v[1], nullptr, 10);
  const uint32_t count = (uint32_t)strtoull(v[2], nullptr, 10);
  const uint32_t chunk = (uint32_t)strtoull(v[3], nullptr, 10);
  const uint32_t n = gg::num_chunks(count, chunk);
  printf("%u\n", n);
  for (uint32_t j = 0; j < n; ++j) {
    const gg::WorkItem w =
        gg::chunk_item(7, begin, begin + count, chunk, j, (int)j);
    printf("%lld %lld %d %d\n", (long long)w.rec_begin, (long long)w.rec_end,
           w.tile, w.slot);
  }
}
"""


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    """The host build of the work items' arithmetic."""
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not shutil.which("g++") or not os.path.isdir(f"{cuda}/include"):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("cut")
    (d / "cut.cpp").write_text(CUT)
    subprocess.run(["g++", "-std=c++17", "-I", f"{cuda}/include", "-I",
                    os.path.join(ROOT, "gpu-gridding_gb300", "csrc"),
                    str(d / "cut.cpp"), "-o", str(d / "cut")], check=True)

    def run(begin, count, chunk):
        out = subprocess.run([str(d / "cut"), str(begin), str(count),
                              str(chunk)], check=True, capture_output=True,
                             text=True).stdout.split("\n")
        return int(out[0]), [tuple(map(int, x.split())) for x in out[1:] if x]
    return run


@pytest.mark.parametrize("begin,count,chunk", [
    (0, 1, 64), (5, 64, 64), (5, 65, 64), (0, 2**32 - 16, 700_001),
    (2**31 - 40, 100, 64), (2**32 - 16 - 1000, 1000, 999),
    (3, 2**32 - 19, 2**31 - 1), (2**31 + 3, 2**31 - 19, 1 << 26)])
def test_chunks_cover_a_tile(cut, begin, count, chunk):
    """The chunks of a tile's records lie end to end from its first record to
    its last, each `chunk` long but the last, wherever in 32 bits they lie."""
    n, items = cut(begin, count, chunk)
    assert n == len(items) == -(-count // chunk)
    at = begin
    for j, (a, b, tile, slot) in enumerate(items):
        assert a == at and (tile, slot) == (7, j)
        assert b - a == (chunk if j < n - 1 else count - chunk * (n - 1))
        at = b
    assert at == begin + count


@pytest.mark.gpu
def test_more_than_2_31_records(pkg):
    """2.2e9 records: every cell counts the footprints over it.  The taps,
    weights and visibilities are one, so each sum is a whole number below
    2^24, exact in FP32."""
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    G, s, n = 1040, 500, 4_400_000
    if torch.cuda.mem_get_info()[0] < 140e9:
        pytest.skip("needs 140 GB of device memory")
    csh = s + 2
    cube = torch.zeros((1, csh, csh, 2), dtype=torch.float32, device="cuda")
    cube[..., 0] = 1.0
    stack = pkg.KernelStack(1, np.array([s], np.int32), 1, csh, cube, "f")
    plan = pkg.Plan()
    plan.set_tuning({"tile_u": 8, "tile_phases": 1})
    # Cells from the grid's centre, each taken by every fourth point.
    du = torch.tensor([-15.0, -8.0, 0.0, 11.0], device="cuda")
    dv = torch.tensor([9.0, -20.0, 0.0, 3.0], device="cuda")
    k = torch.arange(n, device="cuda") % 4
    one = torch.ones(n, device="cuda")
    vis = torch.zeros((n, 2), device="cuda")
    vis[:, 0] = 1.0
    grid = torch.zeros((G, G, 2), dtype=torch.float32, device="cuda")
    norm = torch.zeros(1, dtype=torch.float64, device="cuda")
    skip = torch.zeros(1, dtype=torch.int64, device="cuda")
    pkg.grid_wproj_device(plan, stack, -du[k], dv[k], torch.zeros(
        n, device="cuda"), vis, one, np.float32(1.0 / G), np.float32(1.0), G,
        grid, norm, skip)
    assert plan.stats()["num_records"] > 2**31
    want = torch.zeros((G, G), dtype=torch.float32, device="cuda")
    for j in range(4):
        u, v = int(du[j]) + G // 2, int(dv[j]) + G // 2
        want[v - s:v + s + 1, u - s:u + s + 1] += float(n // 4)
    assert int(skip.item()) == 0
    assert norm.item() == float(n) * (2 * s + 1) ** 2
    assert torch.equal(grid[..., 0], want)
    assert not grid[..., 1].any()
    plan.close()
    torch.cuda.empty_cache()
