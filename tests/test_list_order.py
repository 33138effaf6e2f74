"""Lists ordered by rows (calls of at least 4,096 parts and 2^21 vertices) and
the bucket prefix sums around their block limits, vs the oracle: parts of
every kind whose rows fall into, between and outside the bins, all_touched
(a polygon is on two lists), row windows, and bucket counts around one scan
block (4,096 buckets)."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G
from rusterize_gb300 import synth

from _util import diff_report, gpu_burn, grid_of, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


def collection(rng, side, nlines, npolys):
    polys = synth.star_polygons(rng, npolys, (3, 40), rng.uniform(1, 30, npolys), rng.uniform(-40, side + 40, npolys),
                                rng.uniform(-40, side + 40, npolys), n_holes=rng.integers(0, 2, npolys))
    lines = synth.random_walk_lines(rng, nlines, (400, 560), (0.05, 1.5), (-20, -20, side + 20, side + 20))
    pts = synth.random_points(rng, 500, (0, 0, side, side))
    return G.GeometryTable.concat([polys, lines, pts])


@pytest.mark.parametrize("rows,touched", [(37, False), (1023, False), (1025, False), (2500, False), (700, True)])
def test_ordered_lists(rows, touched):
    from rusterize_gb300.engine import RasterInfo, rasterize_table

    rng = np.random.default_rng(rows)
    t = collection(rng, 900.0, 4300, 1500)
    assert t.n_parts >= 4096 and t.n_vertices >= 1 << 21
    v = rng.integers(1, 9, t.n_geoms).astype(np.int32)
    grid = dict(nrows=rows, ncols=600, xmin=0.0, xmax=900.0, ymin=0.0, ymax=900.0, xres=900.0 / 600,
                yres=900.0 / rows)
    for fn in ("sum", "last"):
        kw = dict(fn=fn, values=v, background=0, dtype="int32", all_touched=touched)
        got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), f"{fn}: " + diff_report(got, ref)
    r0, r1 = rows // 3, rows // 3 + max(1, rows // 7)
    part = rasterize_table(t, RasterInfo(**grid_of(grid)), rows=(r0, r1), **kw)
    assert same_bits(part, np.ascontiguousarray(ref[:, r0:r1]))


@pytest.mark.parametrize("nrows,ncols", [(4095, 300), (4096, 512), (4097, 500), (2049, 513), (1, 1)])
def test_bucket_scan_limits(nrows, ncols):
    rng = np.random.default_rng(nrows + ncols)
    n = 300
    t = synth.star_polygons(rng, n, (3, 20), rng.uniform(1, 60, n), rng.uniform(0, ncols, n), rng.uniform(0, nrows, n))
    grid = dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0, yres=1.0)
    kw = dict(fn="sum", values=np.arange(1, n + 1).astype(np.int64), background=0, dtype="int64")
    got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
    assert same_bits(got, ref), diff_report(got, ref)
