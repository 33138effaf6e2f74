"""Device tables whose part offsets go up and down are refused after about one
pass over them: the ranges of such a table add up to the parts times the
geometries, and the check maps parts to geometries as it goes."""

import time

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import synth
from rusterize_gb300.device import DeviceTable, rasterize_device, upload

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
