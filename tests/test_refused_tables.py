"""The table check, which maps parts to geometries as it goes: offsets that go
up and down are refused after about one pass over them, although the ranges of
such a table add up to the parts times the geometries, and geometries of any
number of parts are mapped, at about the speed of a write of the map."""

import time

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300 import synth
from rusterize_gb300.device import DeviceTable, rasterize_device, upload

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4000, 400_000])  # as one launch, and as separate kernels
def test_offsets_up_and_down(n):
    rng = np.random.default_rng(n)
    t = synth.random_points(rng, n, (0, 0, 100, 100))
    info = rz.RasterInfo(nrows=100, ncols=100, xmin=0.0, xmax=100.0, ymin=0.0, ymax=100.0, xres=1.0, yres=1.0)
    dt = DeviceTable.upload(t)
    want = rasterize_device(dt, info, fn="count", background=0, dtype="int32").cpu().numpy()
    assert want.sum() == n
    bad = t.part_offsets.copy()
    bad[1:-1:2], bad[2:-1:2] = n, 0  # 0, n, 0, n, ..., n
    dt.tensors["part_offsets"] = upload(bad)
    start = time.perf_counter()
    with pytest.raises(ValueError, match="geometry table is inconsistent"):
        rasterize_device(dt, info, fn="count", background=0, dtype="int32")
    assert time.perf_counter() - start < 0.5  # 400,000 ranges of 400,000 parts would take many seconds
    dt.tensors["part_offsets"] = upload(t.part_offsets)
    again = rasterize_device(dt, info, fn="count", background=0, dtype="int32").cpu().numpy()
    assert np.array_equal(again, want)


@pytest.mark.parametrize("sizes", [[0, 1, 7, 8, 9, 31, 32, 33, 0, 1023, 1024, 1025, 0, 3, 2049], [1], [9] * 40,
                                   [5000, 1, 20, 0, 0, 3000]])
def test_geometries_of_many_parts(sizes):
    # every part counts under its own geometry's value
    rng = np.random.default_rng(len(sizes))
    n = sum(sizes)
    t = synth.random_points(rng, n, (0, 0, 60, 60))
    t = G.GeometryTable(np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64), t.part_kind, t.ring_offsets,
                        t.vertex_offsets, t.ring_flags, t.xy)
    grid = dict(nrows=60, ncols=60, xmin=0.0, xmax=60.0, ymin=0.0, ymax=60.0, xres=1.0, yres=1.0)
    kw = dict(fn="sum", values=np.arange(1, len(sizes) + 1).astype(np.int64), background=0, dtype="int64")
    got, ref = gpu_burn(t, grid, **kw), oracle_burn(t, grid, **kw)
    assert same_bits(got, ref), diff_report(got, ref)


def test_one_geometry_of_a_million_parts():
    n = 1_000_000
    t = synth.random_points(np.random.default_rng(1), n, (0, 0, 500, 500))
    t = G.GeometryTable(np.array([0, n], np.uint64), t.part_kind, t.ring_offsets, t.vertex_offsets, t.ring_flags, t.xy)
    info = rz.RasterInfo(nrows=500, ncols=500, xmin=0.0, xmax=500.0, ymin=0.0, ymax=500.0, xres=1.0, yres=1.0)
    dt = DeviceTable.upload(t)
    took = []
    for _ in range(4):
        start = time.perf_counter()
        got = rasterize_device(dt, info, fn="count", background=0, dtype="int32")
        took.append(time.perf_counter() - start)
    assert int(got.sum()) == n
    assert min(took) < 0.015  # 0.04 s and more when one thread writes the million entries
