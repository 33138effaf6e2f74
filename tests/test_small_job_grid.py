"""The grid of a small call's one launch, which has to suit all its phases: few
parts of few vertices can have many windows to burn, and the time of such a
call must not be above that of the separate kernels."""

import time

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300.device import DeviceTable, rasterize_device

from _util import diff_report, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


def ellipses(n, nrows, ncols, points_outside=0):
    rng = np.random.default_rng(n)
    a = np.arange(50) * (2 * np.pi / 50)
    b = G.TableBuilder()
    for _ in range(n):
        cx, cy = rng.uniform(0, ncols), rng.uniform(0, nrows)
        G.add_polygon(b, np.stack([cx + 1500 * rng.uniform(0.5, 1) * np.cos(a), cy + 1500 * np.sin(a)], axis=1))
    for _ in range(points_outside):
        G.add_point(b, -5.0, -5.0)
    return b.build()


@pytest.mark.parametrize("n,nrows,ncols", [(3, 1000, 2048), (100, 1000, 2048), (20, 100, 5000), (20, 1024, 8192)])
def test_few_parts_of_many_windows(n, nrows, ncols):
    info = rz.RasterInfo(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0,
                         yres=1.0)
    kw = dict(fn="count", background=0, dtype="int32")

    def best(t):
        dt = DeviceTable.upload(t)
        took = []
        for _ in range(12):
            start = time.perf_counter()
            out = rasterize_device(dt, info, **kw)
            took.append(time.perf_counter() - start)
        return min(took), out.cpu().numpy()

    t = ellipses(n, nrows, ncols)
    one, got = best(t)
    separate, same = best(ellipses(n, nrows, ncols, 5000))  # more parts than a small call has
    grid = dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0, yres=1.0)
    ref = oracle_burn(t, grid, values=None, **kw)
    assert same_bits(got, ref), diff_report(got, ref)
    assert np.array_equal(got, same)
    assert one < 1.25 * separate + 0.00003
