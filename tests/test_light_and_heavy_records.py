"""first / last over tiles whose words are covered by records of one pixel, of a
few and of most of a word at once: the order-free pass takes the former with
shared-memory atomics of the lane that loaded them and the latter one lane per
pixel, so a pixel is reached both ways within 32 records.  Bit-exact vs the
oracle, at depths below and above 32 records and up to the pass's limit."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["uint8", "float32", "float64"])
@pytest.mark.parametrize("n", [12, 32, 33, 200, 1024])
def test_pixels_reached_both_ways(n, dtype):
    rng = np.random.default_rng(n + len(dtype))
    nrows, ncols = 40, 96
    b = G.TableBuilder()
    for k in range(n):
        word = 32 * int(rng.integers(0, 3))
        if k % 2:  # heavy: 9 to 31 pixels of a word, every row
            w = int(rng.integers(9, 32))
            x = word + int(rng.integers(0, 33 - w))
            G.add_polygon(b, np.array([[x, 0.0], [x + w, 0.0], [x + w, nrows], [x, nrows]], dtype=np.float64))
        elif k % 4:  # light: up to 8 pixels of a word, every row
            w = int(rng.integers(1, 9))
            x = word + int(rng.integers(0, 33 - w))
            G.add_polygon(b, np.array([[x, 0.0], [x + w, 0.0], [x + w, nrows], [x, nrows]], dtype=np.float64))
        else:
            G.add_linestring(b, [(word + rng.uniform(0, 32), 0.2), (word + rng.uniform(0, 32), nrows - 0.3)])
    t = b.build()
    v = rng.integers(1, 200, n).astype(dtype)
    v[rng.random(n) < 0.3] = 0  # the background: not sticky for first
    grid = dict(nrows=nrows, ncols=ncols, xmin=0.0, xmax=float(ncols), ymin=0.0, ymax=float(nrows), xres=1.0, yres=1.0)
    for fn in ("first", "last"):
        kw = dict(fn=fn, values=v, background=0, dtype=dtype)
        ref = oracle_burn(t, grid, **kw)
        for _ in range(3):
            got = gpu_burn(t, grid, **kw)
            assert same_bits(got, ref), f"{fn}: " + diff_report(got, ref)
