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


@pytest.mark.parametrize("geoms,rings", [(1000, 0), ((1 << 17) - 40, 0), ((1 << 17) - 39, 0), (0, (1 << 17) - 40),
                                         (0, (1 << 17) - 39), (1_000_000, 1_000_000)])
def test_many_empty_geometries_and_rings(geoms, rings):
    # 40 polygons, empty geometries behind them and empty rings in the last one
    rng = np.random.default_rng(geoms + rings)
    b = G.TableBuilder()
    for _ in range(40):
        x, y = rng.uniform(0, 200, 2)
        G.add_polygon(b, np.array([[x, y], [x + 30, y + 3], [x + 20, y + 40]]))
    t = b.build()
    ro, vo = t.ring_offsets.copy(), np.concatenate([t.vertex_offsets, np.full(rings, t.n_vertices, np.uint64)])
    ro[-1] += rings
    t = G.GeometryTable(np.concatenate([t.part_offsets, np.full(geoms, t.n_parts, np.uint64)]), t.part_kind, ro, vo,
                        np.concatenate([t.ring_flags, np.zeros(rings, np.uint8)]), t.xy)
    grid = dict(nrows=240, ncols=240, xmin=0.0, xmax=240.0, ymin=0.0, ymax=240.0, xres=1.0, yres=1.0)
    kw = dict(fn="sum", values=np.arange(1, t.n_geoms + 1).astype(np.int32), background=0, dtype="int32")
    stats = {}
    got = rz.rasterize_table(t, rz.RasterInfo(**grid), stats=stats, **kw)
    ref = oracle_burn(t, grid, **kw)
    assert same_bits(got, ref), diff_report(got, ref)
    small = t.n_geoms <= 1 << 17 and len(t.ring_flags) <= 1 << 17
    assert (stats["kernel_launches"] <= 4) == small  # one launch and the fills, or every kernel by itself
