"""Large polygon parts at the bottom of rasters of more than 2^24 rows, whose
row numbers have no exact float32: a window that starts at the last row needs
the chunks of vertices that end below it.  Bit-exact vs the oracle."""

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import geometry as G

from _util import diff_report, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrows", [2**24, 2**24 + 1, 2**24 + 3, 2**25 + 5])
def test_last_row(nrows):
    ncols, n = 8, 12000
    a = np.arange(n) * (2 * np.pi / n)
    # rows [nrows - 1 - 1280, nrows): ten windows of 128 rows and one of the last row; the ring goes on below it
    top, low = 1281.0, -14.0
    y = (top + low) / 2 + (top - low) / 2 * np.sin(a)
    b = G.TableBuilder()
    G.add_polygon(b, np.stack([4.0 + 3.5 * np.cos(a), y], axis=1))
    t = b.build()
    grid = dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0, yres=1.0)
    kw = dict(fn="count", values=None, background=0, dtype="uint8")
    ref = np.ascontiguousarray(oracle_burn(t, grid, **kw)[:, nrows - 1400:])
    got = rz.rasterize_table(t, rz.RasterInfo(**grid), rows=(nrows - 1400, nrows), **kw)
    assert same_bits(got, ref), diff_report(got, ref)
    assert got[:, -1].any()
