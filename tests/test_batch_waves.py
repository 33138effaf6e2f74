"""The device memory a batch's jobs are counted with when they are split into
waves by a byte limit: the row ranges of the vertices' chunks belong to it."""

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300.device import DeviceTable, rasterize_batch_device

from _util import oracle_burn

pytestmark = pytest.mark.gpu


def test_chunk_ranges_count():
    nv, side = 1 << 18, 64
    a = np.arange(nv) * (2 * np.pi / nv)
    xy = np.stack([32 + 30 * np.cos(a), 32 + 30 * np.sin(a) * (0.9 + 0.1 * np.cos(7 * a))], axis=1)
    b = G.TableBuilder()
    G.add_polygon(b, xy)
    t = b.build()
    grid = dict(nrows=side, ncols=side, xmin=0.0, xmax=float(side), ymin=0.0, ymax=float(side), xres=1.0, yres=1.0)
    dt, info = DeviceTable.upload(t), rz.RasterInfo(**grid)
    ref = oracle_burn(t, grid, fn="count", background=0, dtype="int32")
    for limit, waves in ((2 * 16.15, 2), (2 * 16.5, 1)):  # bytes a vertex: 16 and a quarter, and little else
        jobs = [rz.BatchJob(dt, info, None, "count", 0) for _ in range(2)]
        stats: dict = {}
        outs = rasterize_batch_device(jobs, dtype="int32", wave_bytes=int(limit * nv), stats=stats)
        assert stats["waves"] == waves
        for o in outs:
            assert np.array_equal(o.cpu().numpy().view(np.int32).reshape(side, side), ref.reshape(side, side))
