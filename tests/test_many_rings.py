"""Polygon parts of more than 32 rings: ring starts at every place of a warp's
chunk of 32 vertices, rings of few vertices and runs of empty ones, on every
route of a part (one launch, narrow, wide and column windows, windows walked by
chunk), bit-exact vs the oracle; and the time of parts of very many rings beside
the same vertices as one ring, and of parts of two windows beside parts of one."""

import time

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300.device import DeviceTable, rasterize_device

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


def offsets(sizes):
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)


def polygons(rings, sizes, xy):
    n = len(rings)
    return G.GeometryTable(np.arange(n + 1), np.full(n, G.POLYGON, np.uint8), offsets(rings), offsets(sizes),
                           np.zeros(len(sizes), np.uint8), xy)


def part(rng, nrings, empty, nrows, ncols):
    """Ring sizes and vertices: small rings, mostly closed, with runs of empty ones between them."""
    sizes, xy = [], []
    for _ in range(nrings):
        nv = int(rng.choice([1, 2, 3, 4, 5, 9, 31, 33]))
        c = np.array([rng.uniform(0, ncols), rng.uniform(0, nrows)])
        r = c + rng.uniform(-6, 6, (nv, 2))
        sizes.append(nv + (nv > 1 and rng.random() < 0.9))
        xy.append(r)
        if sizes[-1] > nv:
            xy.append(r[:1])
        if rng.random() < 0.05:
            sizes += [0] * int(rng.integers(0, empty + 1))
    return sizes, np.concatenate(xy)


@pytest.mark.parametrize("nrows,ncols", [(60, 90), (300, 2100), (700, 16), (6, 270000)])
@pytest.mark.parametrize("nrings,empty", [(33, 0), (40, 3), (64, 40), (65, 70), (400, 33), (3000, 100)])
def test_against_oracle(nrings, empty, nrows, ncols):
    rng = np.random.default_rng(nrings + ncols)
    for parts in (1, 3):
        p = [part(rng, nrings, empty, nrows, ncols) for _ in range(parts)]
        # one ring that spans the raster, so that some parts are as wide
        p[0][0].append(5)
        p[0] = (p[0][0], np.concatenate([p[0][1], [[1, 1], [ncols - 1, 2], [ncols - 2, nrows], [0, nrows - 1], [1, 1]]]))
        t = polygons([len(s) for s, _ in p], np.concatenate([s for s, _ in p]), np.concatenate([c for _, c in p]))
        grid = dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0,
                    yres=1.0)
        kw = dict(fn="sum", values=np.arange(1, parts + 1).astype(np.int32), background=0, dtype="int32")
        stats: dict = {}
        got, ref = gpu_burn(t, grid, stats=stats, **kw), oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), diff_report(got, ref)
        assert stats["edges"] == len(t.xy) - sum(int(x > 0) for x in np.diff(t.vertex_offsets.astype(np.int64)))


def test_time_of_many_rings():
    side, parts = 548, 10
    at = np.arange(side * side)
    x, y = at % side * 3.0 + 0.3, at // side * 3.0 + 0.4
    xy = np.stack([np.stack([x + dx, y + dy], 1) for dx, dy in ((0, 0), (2, 0), (2, 2.2), (0, 2.2), (0, 0))], 1)
    n = side * side // parts
    xy = xy[: n * parts].reshape(-1, 2)
    info = rz.RasterInfo(nrows=3 * side, ncols=3 * side, xmin=0.0, xmax=3.0 * side, ymin=0.0, ymax=3.0 * side, xres=1.0,
                         yres=1.0)

    def best(t):
        dt = DeviceTable.upload(t)
        took = []
        for _ in range(8):
            start = time.perf_counter()
            rasterize_device(dt, info, fn="count", background=0, dtype="int32")
            took.append(time.perf_counter() - start)
        return min(took)

    many = best(polygons(np.full(parts, n), np.full(n * parts, 5), xy))
    one = best(polygons(np.full(parts, 1), np.full(parts, 5 * n), xy))
    assert many < one  # 0.6 of it; with a search by every lane whose ring had ended 1.2


def test_time_of_two_windows():
    side = 548
    at = np.arange(side * side)
    x, y = at % side * 3.0 + 0.3, at // side * 3.0 + 0.4
    xy = np.stack([np.stack([x + dx, y + dy], 1) for dx, dy in ((0, 0), (2, 0), (2, 2.2), (0, 2.2), (0, 0))], 1)
    info = rz.RasterInfo(nrows=3 * side, ncols=3 * side, xmin=0.0, xmax=3.0 * side, ymin=0.0, ymax=3.0 * side, xres=1.0,
                         yres=1.0)

    def best(parts):
        n = side * side // parts
        dt = DeviceTable.upload(polygons(np.full(parts, 1), np.full(parts, 5 * n), xy[: n * parts].reshape(-1, 2)))
        took = []
        for _ in range(8):
            start = time.perf_counter()
            rasterize_device(dt, info, fn="count", background=0, dtype="int32")
            took.append(time.perf_counter() - start)
        return min(took)

    one, two = best(20), best(10)  # windows of up to 128 rows: 82 rows a part, and 164
    assert two < 1.45 * one  # 1.1 times; every window walking the whole part 1.8
