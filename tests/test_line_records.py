"""Line segments -> coverage records (rusterize_gb300/csrc/rz_line.cuh) vs the
oracle, bit-exact, where the work split can go wrong: linestrings around the
32 vertices a warp sets up at a time and the 128 it takes at once, empty
linestrings between them, parts of many linestrings, segments much longer
than their neighbours, and pixels one part visits several times."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu

SIDE = 300


def walks(rng, sizes, step):
    return [np.cumsum(np.vstack([rng.uniform(-10, SIDE + 10, (1, 2)), rng.uniform(-step, step, (n - 1, 2))]), axis=0)
            if n else np.zeros((0, 2)) for n in sizes]


@pytest.mark.parametrize("touched", [False, True])
@pytest.mark.parametrize("nv", [1, 2, 31, 32, 33, 127, 128, 129, 700])
def test_linestring_lengths(nv, touched):
    rng = np.random.default_rng(1000 * nv + touched)
    b = G.TableBuilder()
    for k in range(max(4, 400 // nv)):
        G.add_linestring(b, walks(rng, [nv], 6.0)[0])
        if k % 3 == 0:
            G.add_linestring(b, np.zeros((0, 2)))                        # empty linestring
        if k % 5 == 0:
            G.add_multilinestring(b, walks(rng, [2, 0, nv, 1, 3], 4.0))  # pooled linestrings
        if k % 7 == 0:
            G.add_linestring(b, rng.uniform(-400, 700, (2, 2)))          # one long segment, partly outside
        if k % 4 == 0:
            G.add_point(b, *rng.uniform(0, SIDE, 2))
    t = b.build()
    v = rng.integers(1, 6, t.n_geoms).astype(np.float64)
    for res in (1.0, 0.75):
        grid = dict(nrows=SIDE, ncols=SIDE, xmin=0.0, xmax=float(SIDE), ymin=0.0, ymax=SIDE * res, xres=1.0, yres=res)
        for fn, bg in (("sum", np.nan), ("count", 0.0), ("last", 0.0)):
            kw = dict(fn=fn, values=v, background=bg, all_touched=touched)
            got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
            assert same_bits(got, ref), f"{fn} res {res}: " + diff_report(got, ref)


@pytest.mark.parametrize("touched", [False, True])
def test_repeated_visits_keep_their_writes(touched):
    # back and forth over the same pixels: without a PixelCache every visit is a write
    b = G.TableBuilder()
    for k in range(70):
        y = 2.3 + 3 * k
        G.add_linestring(b, [(1.5, y), (1.5 + k, y + 0.5), (1.5, y + 0.2), (1.5 + k, y + 0.4)])
    t = b.build()
    grid = dict(nrows=220, ncols=100, xmin=0.0, xmax=100.0, ymin=0.0, ymax=220.0, xres=1.0, yres=1.0)
    for fn, dt in (("count", "uint16"), ("sum", "int32"), ("any", "uint8")):
        kw = dict(fn=fn, values=np.arange(1, t.n_geoms + 1).astype(dt), background=0, dtype=dt, all_touched=touched)
        got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), f"{fn}: " + diff_report(got, ref)


@pytest.mark.parametrize("shift", [0, 1, 15, 30, 31, 32, 33])
def test_runs_of_single_vertex_parts(shift):
    # every vertex of a warp's 32 can belong to a part of its own, and the
    # part that starts with the next 32 must not be missed
    rng = np.random.default_rng(shift)
    b = G.TableBuilder()
    for k in range(shift):
        G.add_linestring(b, rng.uniform(0, SIDE, (1, 2)))
    for k in range(40):
        G.add_linestring(b, rng.uniform(0, SIDE, (2, 2)))
        for _ in range(int(rng.integers(25, 35))):
            G.add_linestring(b, rng.uniform(0, SIDE, (1, 2)))
    for k in range(500):
        G.add_point(b, *rng.uniform(0, SIDE, 2))
        if k % 37 == shift % 37:
            G.add_multipoint(b, rng.uniform(0, SIDE, (shift + 1, 2)))
    t = b.build()
    grid = dict(nrows=SIDE, ncols=SIDE, xmin=0.0, xmax=float(SIDE), ymin=0.0, ymax=float(SIDE), xres=1.0, yres=1.0)
    for touched in (False, True):
        kw = dict(fn="count", values=None, background=0, dtype="int32", all_touched=touched)
        got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
        assert same_bits(got, ref), diff_report(got, ref)
