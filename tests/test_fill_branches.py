"""The fills' branches vs the oracle, bit-exact: records of one pixel, of a few,
of most of a word and of whole words in one tile; tile depths around the
limits (32 and 64 records in registers, 256 sorted in shared memory, 1,024 in
an order-free pass); values that are the background, NaN, -0.0 or infinite;
rows that start off a 16-byte boundary; parts more than 2^22 apart."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


def grid(nrows, ncols):
    return dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0, yres=1.0)


def shapes(rng, n, nrows, ncols):
    """n geometries in random order: rectangles of every width, points and short lines."""
    b = G.TableBuilder()
    for _ in range(n):
        kind = int(rng.integers(0, 4))
        x, y = rng.uniform(-5, ncols), rng.uniform(-1, nrows)
        if kind == 0:
            G.add_point(b, x, y)
        elif kind == 1:
            G.add_linestring(b, [(x, y), (x + rng.uniform(-9, 9), y + rng.uniform(-3, 3))])
        else:
            w = float(np.exp(rng.uniform(0, np.log(ncols + 2.0))))
            h = float(rng.uniform(0.5, nrows))
            G.add_polygon(b, np.array([[x, y], [x + w, y], [x + w, y + h], [x, y + h]]))
    return b.build()


def check(t, g, **kw):
    got, ref = gpu_burn(t, g, **kw), oracle_burn(t, g, **kw)
    assert same_bits(got, ref), f"{kw['fn']} {kw['dtype']}: " + diff_report(got, ref)


@pytest.mark.parametrize("dtype", ["uint8", "int16", "int32", "uint32", "int64", "float32", "float64"])
@pytest.mark.parametrize("n", [20, 31, 33, 63, 65, 250, 262, 900, 1400])
def test_depths_and_masks(n, dtype):
    rng = np.random.default_rng(n * 31 + len(dtype))
    nrows, ncols = 3, 700
    t = shapes(rng, n, nrows, ncols)
    dt = np.dtype(dtype)
    plain = (rng.integers(1, 100, n) - (50 if dt.kind in "if" else 0)).astype(dt)
    plain[plain == 0] = 1
    odd = plain.copy()
    odd[rng.random(n) < 0.02] = 0  # the background
    if dt.kind == "f":
        odd[rng.random(n) < 0.01] = -0.0
        odd[rng.random(n) < 0.01] = np.nan
        odd[rng.random(n) < 0.01] = np.inf
    for fn in ("sum", "first", "last", "min", "max", "count", "any"):
        for values in (plain, odd):
            check(t, grid(nrows, ncols), fn=fn, values=values, background=0, dtype=dtype)
        if dt.kind == "f":
            check(t, grid(nrows, ncols), fn=fn, values=plain, background=np.nan, dtype=dtype)


@pytest.mark.parametrize("ncols", [1, 3, 15, 16, 17, 31, 33, 511, 512, 513, 1029])
def test_row_starts(ncols):
    rng = np.random.default_rng(ncols)
    t = shapes(rng, 30, 9, ncols)
    v = rng.integers(1, 100, t.n_geoms)
    for dtype, bg in (("uint8", 7), ("int16", -3), ("float32", np.nan), ("uint64", 2**40 + 5), ("float64", 0.5)):
        for fn in ("any", "count", "last", "max"):
            check(t, grid(9, ncols), fn=fn, values=v.astype(dtype), background=bg, dtype=dtype)


def test_parts_far_apart():
    # the register sort packs parts relative to the tile's smallest in 22 bits
    rng = np.random.default_rng(3)
    a, c = shapes(rng, 12, 4, 600), shapes(rng, 12, 4, 600)
    n = (1 << 22) + 100
    ar = np.arange(n + 1, dtype=np.uint64)
    far = G.GeometryTable(ar, np.zeros(n, np.uint8), ar, ar, np.zeros(n, np.uint8), np.full((n, 2), -10.0))
    t = G.GeometryTable.concat([a, far, c])
    v = rng.integers(1, 100, t.n_geoms).astype(np.float32)
    check(t, grid(4, 600), fn="sum", values=v, background=np.nan, dtype="float32")
