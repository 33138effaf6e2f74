"""Large polygon parts (prep by a block, windows that walk only the chunks of
vertices near their rows: k_part_prep_big / k_poly_spans_chunked) vs the
oracle, bit-exact, around the sizes where the rules change: 1,024 vertices a
part, 8,192 a call, 65,536 per batch of chunks; smooth boundaries (chunks are
skipped) and jagged ones (they are not), holes, resolutions, row windows."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, grid_of, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


def ring(rng, n, cx, cy, r, jag):
    a = np.arange(n) * (2 * np.pi / n)
    rad = r * (1.0 + 0.2 * np.sin(3 * a + rng.uniform(0, 6)) + 0.1 * np.sin(11 * a + rng.uniform(0, 6))
               + rng.uniform(-jag, jag, n))
    return np.stack([cx + rad * np.cos(a), cy + rad * np.sin(a)], axis=1)


def table(rng, nv, side, jag):
    b = G.TableBuilder()
    for k in range(max(3, 12000 // nv)):
        cx, cy = rng.uniform(0, side, 2)
        r = float(np.exp(rng.uniform(np.log(40), np.log(side * 0.7))))
        holes = [ring(rng, max(8, nv // 3), cx, cy, r * 0.3, 0.01)] if k % 3 == 0 else []
        G.add_polygon(b, ring(rng, nv - 1, cx, cy, r, jag), holes)
        if k % 4 == 0:  # several rings of one part, far apart
            G.add_multipolygon(b, [(ring(rng, nv // 2, *rng.uniform(0, side, 2), 60.0, jag),) for _ in range(3)])
    G.add_polygon(b, np.array([[5.0, 5.0], [90.0, 5.0], [90.0, 70.0], [5.0, 70.0]]))
    return b.build()


@pytest.mark.parametrize("jag", [0.002, 0.4])
@pytest.mark.parametrize("nv", [1000, 1023, 1024, 1025, 2000, 5000, 66000])
def test_part_sizes(nv, jag):
    rng = np.random.default_rng(nv + int(1000 * jag))
    side = 1500
    t = table(rng, nv, side, jag)
    v = rng.integers(1, 100, t.n_geoms).astype(np.float32)
    for res in (1.0, 30.0):
        s = G.GeometryTable(t.part_offsets, t.part_kind, t.ring_offsets, t.vertex_offsets, t.ring_flags, t.xy * res)
        grid = dict(nrows=side - 13, ncols=side + 77, xmin=0.0, xmax=(side + 77) * res, ymin=0.0,
                    ymax=(side - 13) * res, xres=res, yres=res)
        kw = dict(fn="sum", values=v, background=np.nan, dtype="float32")
        got, ref = gpu_burn(s, grid, **kw), oracle_burn(s, grid, **kw)
        assert same_bits(got, ref), f"res {res}: " + diff_report(got, ref)


def test_wide_parts_rows_and_non_finite():
    from rusterize_gb300.engine import RasterInfo, rasterize_table

    # a part wider than the bitmap (column windows), and one with a far-away spike
    rng = np.random.default_rng(5)
    ncols = 300_000
    b = G.TableBuilder()
    e = ring(rng, 6000, 0.5, 0.5, 0.4, 0.001)
    G.add_polygon(b, e * np.array([ncols, 90.0]))
    e[100] = [3.0e7, 0.5]
    G.add_polygon(b, e * np.array([1000.0, 90.0]))
    e2 = ring(rng, 6000, 500.0, 45.0, 40.0, 0.001)
    G.add_polygon(b, e2)
    t = b.build()
    grid = dict(nrows=90, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=90.0, xres=1.0, yres=1.0)
    kw = dict(fn="count", values=None, background=0, dtype="uint8")
    ref = oracle_burn(t, grid, **kw)
    got = gpu_burn(t, grid, **kw)
    assert same_bits(got, ref), diff_report(got, ref)
    for r0, r1 in ((0, 1), (17, 63), (89, 90)):
        rows = rasterize_table(t, RasterInfo(**grid_of(grid)), rows=(r0, r1), **kw)
        assert same_bits(rows, np.ascontiguousarray(ref[:, r0:r1])), f"rows {r0}:{r1}"
