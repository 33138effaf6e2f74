"""Small calls with a part that the one launch does not take: known beforehand
from a table on the host, and where the raster's bands would be copied to the
host before the call is known to be burned; else found on the device, with the
time it took in the phase times."""

import ctypes

import numpy as np
import pytest

import rusterize_gb300 as rz
from rusterize_gb300 import _lib
from rusterize_gb300 import geometry as G
from rusterize_gb300.device import DeviceTable, rasterize_device

from _util import diff_report, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


def grid(nrows, ncols):
    return dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0, yres=1.0)


def boundary(nv, nrows, ncols, points=0, large=True):
    a = np.arange(nv) * (2 * np.pi / nv)
    r = 0.4 * min(nrows, ncols) * (0.9 + 0.1 * np.sin(9 * a))
    xy = np.stack([ncols / 2 + r * np.cos(a), nrows / 2 + r * np.sin(a)], axis=1)
    b = G.TableBuilder()
    for ring in [xy] if large else np.split(xy, nv // 1000):
        G.add_polygon(b, ring)
    for _ in range(points):
        G.add_point(b, -5.0, -5.0)
    return b.build()


@pytest.mark.parametrize("nrows,ncols", [(300, 400), (2000, 4000)])  # the second one's bands are copied while others fill
def test_host_table(nrows, ncols):
    info, kw = rz.RasterInfo(**grid(nrows, ncols)), dict(fn="last", background=np.nan, dtype="float64")
    launches = []
    for points in (0, 5000):  # 5,000: more parts than a small call has
        t, stats = boundary(20000, nrows, ncols, points), {}
        got = rz.rasterize_table(t, info, values=np.full(t.n_geoms, 3.0), stats=stats, **kw)
        ref = oracle_burn(t, grid(nrows, ncols), values=np.full(t.n_geoms, 3.0), **kw)
        assert same_bits(got, ref), diff_report(got, ref)
        launches.append(stats["kernel_launches"])
    assert launches[0] == launches[1]  # no launch for nothing


def test_device_table_to_host():
    nrows, ncols = 2000, 4000
    t = boundary(20000, nrows, ncols)
    dt, info = DeviceTable.upload(t), rz.RasterInfo(**grid(nrows, ncols))
    lib, ctx = _lib.load(), _lib.default_context()
    out, bg, st, e = np.zeros((1, nrows, ncols)), np.array([np.nan]), _lib.RzStats(), _lib.errbuf()
    g, ri = dt.c_view(), info.c_struct()
    with ctx.lock:
        rc = lib.rz_rasterize(ctx.handle, ctypes.byref(g), None, bg.ctypes.data, None, 1, ctypes.byref(ri),
                              _lib.PIXEL_FNS["last"], _lib.DTYPES["float64"], _lib.FLAG_INPUT_DEVICE, out.ctypes.data,
                              ctypes.byref(st), e, len(e))
    _lib.raise_for(rc, e.value)
    stats = {}
    same = rz.rasterize_table(t, info, fn="last", background=np.nan, dtype="float64", stats=stats)
    assert same_bits(out.reshape(same.shape), same)
    assert st.as_dict()["kernel_launches"] == stats["kernel_launches"]


@pytest.mark.parametrize("large", [True, False])
def test_phase_times(large):
    t = boundary(20000, 300, 400, large=large)
    stats = {}
    rasterize_device(DeviceTable.upload(t), rz.RasterInfo(**grid(300, 400)), fn="count", background=0, dtype="int32",
                     stats=stats)
    one = stats["kernel_launches"] <= 3
    assert one == (not large)
    # as one launch all phases but the fill are in ms_spans; a launch that stopped is in ms_prep
    assert (stats["ms_prep"] > 0) == large and (stats["ms_bucket"] > 0) == large and stats["ms_spans"] > 0
