"""The ranges of line vertices that warps take (31 segments of a linestring at a
time, up to 124 vertices a range, fewer in calls of few vertices): linestrings
that end on a range's border or next to it, bit-exact vs the oracle, and long
segments of a small call, which have to be walked side by side."""

import time

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300.device import DeviceTable, rasterize_device

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu

SIDE = 200


@pytest.mark.parametrize("touched", [False, True])
@pytest.mark.parametrize("first", [30, 31, 32, 61, 62, 63, 92, 93, 94, 123, 124, 125, 154, 155, 156, 247, 248, 249])
def test_first_part_ends_at_the_border(first, touched):
    rng = np.random.default_rng(first)
    for rest in (0, 1, 40, 4000):  # 4,000: more ranges than the grid of such a call has warps
        b = G.TableBuilder()
        for k in range(1 + rest):
            nv = first if k == 0 or rest < 100 else int(rng.integers(2, 200))
            xy = np.cumsum(np.vstack([rng.uniform(0, SIDE, (1, 2)), rng.uniform(-5, 5, (nv - 1, 2))]), axis=0)
            G.add_linestring(b, xy)
        t = b.build()
        grid = dict(nrows=SIDE, ncols=SIDE, xmin=0.0, xmax=float(SIDE), ymin=0.0, ymax=float(SIDE), xres=1.0, yres=1.0)
        kw = dict(fn="sum", values=np.arange(1, t.n_geoms + 1).astype(np.int64), background=0, dtype="int64",
                  all_touched=touched)
        got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), f"{rest} behind: " + diff_report(got, ref)


@pytest.mark.parametrize("n", [400, 6000])  # as one launch, and as separate kernels
def test_long_segments_side_by_side(n):
    info = rz.RasterInfo(nrows=1500, ncols=3000, xmin=0.0, xmax=3000.0, ymin=0.0, ymax=1500.0, xres=1.0, yres=1.0)

    def best(k):
        b = G.TableBuilder()
        for i in range(k):
            G.add_linestring(b, [(0.5, 1.5 + 1400 * i / k), (2999.5, 60.5 + 1400 * i / k)])
        dt = DeviceTable.upload(b.build())
        took = []
        for _ in range(12):
            start = time.perf_counter()
            rasterize_device(dt, info, fn="any", background=0, dtype="uint8")
            took.append(time.perf_counter() - start)
        return min(took)

    few, many = best(12), best(n)
    assert many < 1.6 * few + 0.0002  # rounds of walks one after the other: twice and more
