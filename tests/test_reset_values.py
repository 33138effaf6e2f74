"""min / max over tiles in which a value resets the pixel (the background, NaN,
-0.0), which take the ordered fold: few and many such tiles beside deep and
clean ones, bit-exact vs the oracle, and the time of such a call beside that of
an ordered sum over the same records."""

import time

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300 import synth
from rusterize_gb300.device import DeviceTable, rasterize_device, upload

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


def grid(nrows, ncols):
    return dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0, yres=1.0)


def tiles(rng, nrows, ncols, depth, deep):
    """Points, `depth` per tile on average, and `deep` more on each of three tiles."""
    n = depth * nrows * ((ncols + 511) // 512)
    xy = [np.stack([rng.uniform(0, ncols, n), rng.uniform(0, nrows, n)], axis=1)]
    for row in rng.integers(0, nrows, 3):
        xy.append(np.stack([rng.uniform(0, min(512, ncols), deep), np.full(deep, row + 0.5)], axis=1))
    xy = rng.permutation(np.concatenate(xy))
    ar = np.arange(len(xy) + 1, dtype=np.uint64)
    return G.GeometryTable(ar, np.zeros(len(xy), np.uint8), ar, ar, np.zeros(len(xy), np.uint8), xy)


def values(rng, n, dtype, share):
    v = (rng.integers(1, 90, n) - (40 if np.dtype(dtype).kind in "if" else 0)).astype(dtype)
    v[v == 0] = 1
    at = rng.random(n) < share
    v[at] = rng.choice([0.0, -0.0, np.nan], int(at.sum())) if np.dtype(dtype).kind == "f" else 0
    return v


@pytest.mark.parametrize("dtype", ["uint8", "int16", "int32", "float32", "int64", "float64"])
@pytest.mark.parametrize("nrows,ncols,depth", [(1, 40, 1), (3, 700, 30), (40, 700, 33), (40, 700, 64), (40, 700, 66),
                                               (40, 700, 130), (40, 700, 255), (8300, 1029, 3)])
def test_tiles_with_and_without(nrows, ncols, depth, dtype):
    rng = np.random.default_rng(nrows + depth)
    t = tiles(rng, nrows, ncols, depth, 1100)
    for fn in ("min", "max"):
        for share in (0.01, 0.7):
            kw = dict(fn=fn, values=values(rng, t.n_geoms, dtype, share), background=0, dtype=dtype)
            got, ref = gpu_burn(t, grid(nrows, ncols), **kw), oracle_burn(t, grid(nrows, ncols), **kw)
            assert same_bits(got, ref), f"{fn} {share}: " + diff_report(got, ref)


@pytest.mark.parametrize("dtype", ["uint8", "float32", "float64"])
def test_rasters_of_a_batch(dtype):
    rng = np.random.default_rng(4)
    jobs, refs = [], []
    for nrows, ncols, fn in ((30, 600, "max"), (1, 5, "min"), (200, 1500, "max"), (77, 40, "min"), (90, 513, "max")):
        t = tiles(rng, nrows, ncols, 20, 300)
        v = values(rng, t.n_geoms, dtype, 0.2)
        jobs.append(rz.BatchJob(t, rz.RasterInfo(**grid(nrows, ncols)), v, fn, 0.0))
        refs.append(oracle_burn(t, grid(nrows, ncols), fn=fn, values=v, background=0, dtype=dtype))
    for got, ref in zip(rz.rasterize_batch(jobs, dtype=dtype), refs):
        assert same_bits(got.reshape(ref.shape), ref), diff_report(got.reshape(ref.shape), ref)


@pytest.mark.parametrize("dtype", ["uint8", "int32", "float32", "float64"])
def test_time_beside_an_ordered_sum(dtype):
    rng = np.random.default_rng(5)
    n, side = 100000, 12000
    t = synth.star_polygons_sorted(rng, np.full(n, 64), rng.lognormal(3.0, 0.6, n), rng.uniform(0, side, n),
                                   rng.uniform(0, side, n))
    info, dt = rz.RasterInfo(**grid(side, side)), DeviceTable.upload(t)
    v = upload(rng.integers(0, 3, n).astype(dtype))

    def best(fn):
        took = []
        for _ in range(10):
            start = time.perf_counter()
            rasterize_device(dt, info, fn=fn, background=0, dtype=dtype, values=v)
            took.append(time.perf_counter() - start)
        return min(took)

    assert best("max") < 1.5 * best("sum")  # 1.3 times; with half the warps and a list walked for every tile 1.7 to 2.4
