"""Calls that fail while their polygon windows are burned: a part with an
infinite y has crossings that are NaN and sort to column 0, outside its
bitmap, so the call is refused by whichever kernel burns the part (narrow,
wide, by chunk, or the one launch of small calls) while other blocks of the
same kernel work or have yet to start.  The refusal ends the call with its
error, and the next call of the context burns as if it had not been."""

import concurrent.futures as cf

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300 import synth

from _util import diff_report, oracle_burn, same_bits

pytestmark = pytest.mark.gpu

NROWS, NCOLS = 1200, 3000


def ring(n, cx, cy, rx, ry):
    a = np.arange(n) * (2 * np.pi / n)
    return np.stack([cx + rx * np.cos(a), cy + ry * np.sin(a)], axis=1)


def bad_part(kind):
    if kind == "narrow":
        r = ring(12, 600.0, 500.0, 80.0, 60.0)
    elif kind == "wide":
        r = ring(60, 1700.0, 500.0, 1100.0, 400.0)
    else:
        r = ring(4000, 1700.0, 500.0, 1100.0, 400.0)
    r[len(r) // 4, 1] = np.inf
    b = G.TableBuilder()
    G.add_polygon(b, r)
    return b.build()


def good(n):
    rng = np.random.default_rng(n)
    polys = synth.star_polygons(rng, n, (4, 12), rng.uniform(1, 12, n), rng.uniform(0, NCOLS, n),
                                rng.uniform(0, NROWS, n))
    b = G.TableBuilder()
    for k in range(12):
        G.add_polygon(b, ring(3000, rng.uniform(0, NCOLS), rng.uniform(0, NROWS), 900.0, 400.0))
        G.add_polygon(b, ring(50, rng.uniform(0, NCOLS), rng.uniform(0, NROWS), 900.0, 400.0))
    return G.GeometryTable.concat([polys, b.build()])


@pytest.mark.parametrize("n", [300, 6000])  # as one launch, and as separate kernels
@pytest.mark.parametrize("kind", ["narrow", "wide", "chunked"])
def test_refusal_ends_the_call(kind, n):
    t = good(n)
    mixed = G.GeometryTable.concat([t, bad_part(kind)])
    info = rz.RasterInfo(nrows=NROWS, ncols=NCOLS, xmin=0.0, xmax=float(NCOLS), ymin=0.0, ymax=float(NROWS), xres=1.0,
                         yres=1.0)
    kw = dict(fn="count", background=0, dtype="uint16")
    grid = dict(nrows=NROWS, ncols=NCOLS, xmin=0.0, xmax=float(NCOLS), ymin=0.0, ymax=float(NROWS), xres=1.0, yres=1.0)
    ref = oracle_burn(t, grid, **kw)

    def work(_):
        ctx = rz.Context(0)
        out = []
        for _ in range(5):
            with pytest.raises(RuntimeError, match="non-finite or out-of-range"):
                rz.rasterize_table(mixed, info, context=ctx, **kw)
            out.append(rz.rasterize_table(t, info, context=ctx, **kw))
        ctx.close()
        return out

    with cf.ThreadPoolExecutor(4) as ex:
        for got in (g for gs in ex.map(work, range(4)) for g in gs):
            assert same_bits(got, ref), diff_report(got, ref)
