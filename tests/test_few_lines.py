"""Line calls on both sides of the vertex count below which a lane takes two
pixels between two looks at the warp, as separate kernels: long segments along
rows and columns, single pixels and repeated ones, parts that deduplicate,
bit-exact vs the oracle."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu

FEW = 1 << 17


def offsets(sizes):
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)


def lines(rng, total, nrows, ncols):
    """Linestrings of `total` vertices: the first eight up to the raster's length, then short walks."""
    sizes, xy, left = [], [], total
    while left > 0:
        k = len(sizes)
        n = min(left, 3 if k < 8 else 1000)
        at = np.array([rng.uniform(0, ncols), rng.uniform(0, nrows)])
        if k < 8:
            d = np.array([[ncols, 3.0], [ncols, 0.0], [0.0, nrows], [2.0, nrows], [ncols, nrows], [0.2, 0.1], [-ncols, 9.0],
                          [0.0, 0.0]])[k]
            p = at + np.outer([0, 1, 0.25], d)
        else:
            p = at + np.cumsum(rng.uniform(-2, 2, (n, 2)), axis=0)
        sizes.append(n)
        xy.append(p[:n])
        left -= n
    n = len(sizes)
    ar = np.arange(n + 1, dtype=np.uint64)
    return G.GeometryTable(ar, np.full(n, G.LINE, np.uint8), ar, offsets(sizes), np.zeros(n, np.uint8),
                           np.concatenate(xy))


@pytest.mark.parametrize("yres", [1.0, 2.0])  # pixels that are not square: a part writes a pixel once
@pytest.mark.parametrize("total", [2, 3, 24, 63, 5000, FEW - 1, FEW, FEW + 1])
def test_against_oracle(total, yres):
    nrows, ncols = 9000, 700  # more buckets than a small call has
    t = lines(np.random.default_rng(total), total, nrows * yres, ncols)
    grid = dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=nrows * yres, xres=1.0, yres=yres)
    v = np.arange(1, t.n_geoms + 1).astype(np.int32)
    for fn in ("sum", "first"):
        kw = dict(fn=fn, values=v, background=0, dtype="int32")
        got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), f"{fn}: " + diff_report(got, ref)
