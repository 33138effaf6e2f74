"""Small calls run as one cooperative launch (k_small_job): results around the
limits of its rule (4,096 parts, 2^19 vertices, 2^14 buckets) vs the oracle,
parts that it leaves to other kernels, record buffers that overflow, tables
and bands that are refused, and calls from several threads at once."""

import concurrent.futures as cf

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


def mixture(rng, n, nrows, ncols, nv=(3, 12)):
    k = [n - n // 3 - n // 3, n // 3, n // 3]
    polys = synth.star_polygons(rng, max(1, k[0]), nv, rng.uniform(0.5, 30, max(1, k[0])),
                                rng.uniform(-5, ncols + 5, max(1, k[0])), rng.uniform(-5, nrows + 5, max(1, k[0])))
    parts = [polys]
    if k[1]:
        parts.append(synth.random_walk_lines(rng, k[1], (1, 9), (0.2, 9.0), (0, 0, ncols, nrows)))
        parts.append(synth.random_points(rng, k[2], (0, 0, ncols, nrows)))
    return G.GeometryTable.concat(parts)


def check(t, g, **kw):
    got, ref = gpu_burn(t, g, **kw), oracle_burn(t, g, **kw)
    assert same_bits(got, ref), f"{kw['fn']}: " + diff_report(got, ref)


@pytest.mark.parametrize("n,nrows,ncols", [(1, 1, 1), (1, 5, 2000), (2, 300, 40), (64, 256, 256), (4095, 500, 700),
                                           (4096, 500, 700), (4097, 500, 700), (50, 16383, 100), (50, 8192, 1024),
                                           (50, 8193, 1024)])
def test_limits(n, nrows, ncols):
    rng = np.random.default_rng(n + nrows)
    t = mixture(rng, n, nrows, ncols)
    v = rng.integers(1, 50, t.n_geoms).astype(np.int32)
    for fn in ("last", "sum", "count"):
        check(t, grid(nrows, ncols), fn=fn, values=v, background=0, dtype="int32")


@pytest.mark.parametrize("nv", [(126, 127), (127, 128)])
def test_vertex_limit(nv):
    rng = np.random.default_rng(nv[0])
    n = 4096
    t = synth.star_polygons(rng, n, nv, rng.uniform(2, 20, n), rng.uniform(0, 600, n), rng.uniform(0, 600, n))
    check(t, grid(600, 600), fn="sum", values=rng.uniform(0, 1, n), background=np.nan, dtype="float64")


@pytest.mark.parametrize("big", [1000, 1024, 1026, 9000, 40000])
def test_large_part_among_small(big):
    rng = np.random.default_rng(big)
    b = G.TableBuilder()
    a = np.arange(big) * (2 * np.pi / big)
    G.add_polygon(b, np.stack([300 + (250 + 3 * np.sin(40 * a)) * np.cos(a), 300 + 280 * np.sin(a)], axis=1))
    t = G.GeometryTable.concat([mixture(rng, 1500, 600, 600, (20, 30)), b.build(), mixture(rng, 30, 600, 600)])
    v = rng.uniform(0, 1, t.n_geoms)
    check(t, grid(600, 600), fn="first", values=v, background=np.nan, dtype="float64")


def test_record_overflow_and_bands():
    # 1.6 M one-pixel records of steep lines outgrow the first record buffer
    rng = np.random.default_rng(9)
    b = G.TableBuilder()
    for _ in range(400):
        x = rng.uniform(0, 1000)
        G.add_linestring(b, [(x, 0.5), (x + rng.uniform(-200, 200), 3999.5)])
    t = b.build()
    ctx = rz.Context(0)
    got = rz.rasterize_table(t, rz.RasterInfo(**grid(4000, 1000)), fn="count", background=0, dtype="uint16", context=ctx)
    ref = oracle_burn(t, grid(4000, 1000), fn="count", background=0, dtype="uint16")
    assert same_bits(got, ref), diff_report(got, ref)
    ctx.close()
    t = mixture(rng, 300, 200, 200)
    bands = rng.integers(0, 5, t.n_geoms).astype(np.uint32)
    check(t, grid(200, 200), fn="any", values=None, background=0, dtype="uint8", bands=bands, n_bands=5)
    bands[17] = 5
    with pytest.raises(ValueError, match="band index out of range at geometry 17"):
        gpu_burn(t, grid(200, 200), fn="any", background=0, dtype="uint8", bands=bands, n_bands=5)


def test_refused_device_table():
    rng = np.random.default_rng(2)
    t = mixture(rng, 90, 100, 100)
    info = rz.RasterInfo(**grid(100, 100))
    dt = DeviceTable.upload(t)
    good = rasterize_device(dt, info, fn="count", background=0, dtype="int32").cpu().numpy()
    bad = t.vertex_offsets.copy()
    bad[5] = bad[4] - 1 if bad[4] else 10**6
    dt.tensors["vertex_offsets"] = upload(bad)
    with pytest.raises(ValueError, match="inconsistent"):
        rasterize_device(dt, info, fn="count", background=0, dtype="int32")
    dt.tensors["vertex_offsets"] = upload(t.vertex_offsets)
    again = rasterize_device(dt, info, fn="count", background=0, dtype="int32").cpu().numpy()
    assert np.array_equal(good, again)


def test_threads_with_their_own_contexts():
    jobs = []
    for k in range(8):
        rng = np.random.default_rng(100 + k)
        t = mixture(rng, 60 + 500 * k, 300, 300)
        jobs.append((t, rng.uniform(0, 1, t.n_geoms)))
    refs = [oracle_burn(t, grid(300, 300), fn="sum", values=v, background=np.nan, dtype="float64") for t, v in jobs]

    def work(k):
        ctx = rz.Context(0)
        t, v = jobs[k]
        ok = True
        for _ in range(20):
            got = rz.rasterize_table(t, rz.RasterInfo(**grid(300, 300)), values=v, fn="sum", background=np.nan,
                                     dtype="float64", context=ctx)
            ok = ok and same_bits(got, refs[k])
        ctx.close()
        return ok

    with cf.ThreadPoolExecutor(8) as ex:
        assert all(ex.map(work, range(8)))
