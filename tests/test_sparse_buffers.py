"""Time of sparse burns that get the host buffers of freed results after these
have lain idle, beside burns that get fresh ones."""

import time

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G
from rusterize_gb300.engine import rasterize_table_sparse

pytestmark = pytest.mark.gpu

SIDE = 3500  # 12 M triplets: columns of 98 MB


def burn(k):
    x = k * 3.0
    b = G.TableBuilder()
    G.add_polygon(b, np.array([[x, 0], [SIDE, 0], [SIDE, SIDE], [x, SIDE]]))
    info = rz.RasterInfo(nrows=SIDE, ncols=SIDE, xmin=0.0, xmax=float(SIDE), ymin=0.0, ymax=float(SIDE), xres=1.0,
                         yres=1.0)
    stats = {}
    res = rasterize_table_sparse(b.build(), info, values=np.array([2.5]), fn="sum", dtype="float64", stats=stats)
    return res, stats["ms_d2h"]


def check(res, k):
    n, w = SIDE * (SIDE - 3 * k), SIDE - 3 * k
    _, rows, cols, values = res
    assert len(rows) == n and (values == 2.5).all()
    assert np.array_equal(rows.reshape(SIDE, w)[:, 0], np.arange(SIDE, dtype=np.uint64))
    assert np.array_equal(cols[-w:], np.arange(3 * k, SIDE, dtype=np.uint64))


def test_idle_buffers():
    burn(0)  # device buffers
    kept = [burn(0) for _ in range(4)]  # fresh pages each
    fresh = min(ms for _, ms in kept)
    del kept
    again = []
    for k in range(1, 6):
        time.sleep(0.7)
        res, ms = burn(k)  # not read by the host: that would touch its pages
        again.append(ms)
        if k == 5:
            check(res, k)
        del res
    assert sorted(again)[2] < 2 * fresh + 2.0  # on pages the host had not touched again: four to ten times as long
