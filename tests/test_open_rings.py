"""Rows with an odd number of crossings are looked for only in polygons that
can have them: a ring that does not end at the y it starts at, or a crossing
that was dropped (a NaN crossing, an edge below the horizontal filter's
EPSILON).  All window kinds vs the oracle and vs the same polygons with a ring
below the raster that keeps them on the general path, bit-exact."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu

TINY = 2.0 ** -60


def star(rng, n, cx, cy, r):
    a = np.sort(rng.uniform(0, 2 * np.pi, n))
    rad = r * rng.uniform(0.3, 1.0, n)
    return np.stack([cx + rad * np.cos(a), cy + rad * np.sin(a)], axis=1)


def rings_of(kind, rng, n, side, tall):
    """The rings of one polygon part."""
    r = star(rng, n, 0.5 * side, 0.4 * tall, 0.4 * min(side, 4 * tall))
    r[:, 1] = np.clip(r[:, 1], -3.0, tall + 3.0)
    closed = np.concatenate([r, r[:1]])
    small = np.concatenate([(h := star(rng, 9, 0.5 * side, 0.4 * tall, 6.0)), h[:1]])
    if kind == "closed":
        return [closed, small]
    if kind == "open":
        return [r]
    if kind == "open_hole":  # one ring of several
        return [closed, small, small[:-1] + 3.0, small[:0]]
    if kind == "same_y":  # the ends share y alone: the missing edge has no row
        r[-1, 1] = r[0, 1]
        return [r]
    if kind == "zeros":  # +0.0 and -0.0 are the same y
        r[0, 1], r[-1, 1] = 0.0, -0.0
        return [r]
    if kind == "nan":
        closed[n // 2] = [np.nan, 3.0]
        return [closed, small]
    if kind == "nan_y":
        closed[n // 2] = [3.0, np.nan]
        closed[0, 1] = closed[-1, 1] = np.nan
        return [closed]
    if kind == "inf":  # inf - inf: crossings that are NaN
        closed[n // 2] = [np.inf, 3.0]
        closed[n // 3] = [-np.inf, tall - 3.0]
        return [closed, small]
    # steps below EPSILON around a row's centre (tiny only near pixel y 0.5: see the grid)
    closed[1:n:3, 1] = 0.5 + TINY
    closed[2:n:3, 1] = 0.5 - 2.0 ** -54
    return [closed]


def table_of(parts):
    rings = [r for p in parts for r in p]
    return G.GeometryTable(np.arange(len(parts) + 1, dtype=np.uint64), np.full(len(parts), 2, np.uint8),
                           np.cumsum([0] + [len(p) for p in parts]).astype(np.uint64),
                           np.cumsum([0] + [len(r) for r in rings]).astype(np.uint64),
                           np.zeros(len(rings), np.uint8), np.concatenate(rings))


@pytest.mark.parametrize("kind", ["closed", "open", "open_hole", "same_y", "zeros", "nan", "nan_y", "inf", "tiny"])
@pytest.mark.parametrize("n,side,tall", [(12, 70, 50), (40, 700, 50), (200, 1500, 40), (3000, 900, 400),
                                         (300, 300_000, 12)])
def test_open_rings(kind, n, side, tall):
    rng = np.random.default_rng(n + side + len(kind))
    parts = [rings_of(k, rng, n, side, tall) for k in (kind, "closed", kind)]
    # ymax 1 with one-unit rows from there on: pixel y is 1 - y
    ymax = 1.0 if kind == "tiny" else float(tall)
    ymin = ymax - tall
    grid = dict(nrows=tall, ncols=side, xmin=0.0, xmax=float(side), ymin=ymin, ymax=ymax, xres=1.0, yres=1.0)
    kw = dict(fn="sum", values=np.array([1.0, 2.0, 4.0]), background=np.nan, dtype="float64")
    t = table_of(parts)
    got = gpu_burn(t, grid, **kw)
    below = np.array([[0.5 * side, ymin - 10.0], [0.5 * side, ymin - 20.0]])  # open, without a row
    general = gpu_burn(table_of([p + [below] for p in parts]), grid, **kw)
    assert same_bits(got, general), diff_report(got, general)
    if kind != "inf":  # infinities make NaNs whose sign, and so their place in a row, is the machine's
        ref = oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), diff_report(got, ref)
