"""Ordered folds of words with more records than a warp keeps at a time (512, and
256 for min / max of up to four bytes): record counts around those limits and
around the 128 records that are looked through at a time, parts with more
records in a word than that alone, bit-exact vs the oracle."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu

GRID = dict(nrows=2, ncols=100, xmin=0.0, xmax=100.0, ymin=0.0, ymax=2.0, xres=1.0, yres=1.0)


def table(rng, n, multi):
    """n points on 20 pixels of one word in order, `multi` more of one part in their middle, some elsewhere."""
    counts = np.ones(n + 40, dtype=np.int64)
    x = np.concatenate([rng.integers(33, 53, n), rng.integers(0, 100, 40)]) + 0.5
    parts = [x[i:i + 1] for i in range(n + 40)]
    if multi:
        at = (n + 40) // 2
        parts.insert(at, rng.integers(33, 37, multi) + 0.5)
        counts = np.insert(counts, at, multi)
    x = np.concatenate(parts)
    ar = np.arange(len(counts) + 1, dtype=np.uint64)
    vo = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    return G.GeometryTable(ar, np.zeros(len(counts), np.uint8), ar, vo, np.zeros(len(counts), np.uint8),
                           np.stack([x, np.full(len(x), 0.5)], axis=1))


@pytest.mark.parametrize("multi", [0, 100, 255, 513, 1300])
@pytest.mark.parametrize("n", [257, 383, 384, 385, 511, 512, 513, 1000, 1025, 4097])
def test_against_oracle(n, multi):
    rng = np.random.default_rng(n + multi)
    t = table(rng, n, multi)
    g = t.n_geoms
    size = rng.uniform(1, 2, g) * 10.0 ** rng.integers(-6, 7, g) * rng.choice((-1, 1), g)
    odd = np.where(rng.random(g) < 0.3, 0.0, np.round(size, 3))
    for fn, dtype, v, bg in (("sum", "float32", size, np.nan), ("sum", "float64", size, 0.0), ("max", "float32", odd, 0),
                             ("min", "int16", np.rint(np.clip(odd, -300, 300)), 0), ("max", "float64", odd, 0),
                             ("count", "int32", np.ones(g), 1), ("sum", "uint8", rng.integers(0, 256, g), 7)):
        kw = dict(fn=fn, values=v.astype(dtype), background=bg, dtype=dtype)
        got, ref = gpu_burn(t, GRID, **kw), oracle_burn(t, GRID, **kw)
        assert same_bits(got, ref), f"{fn} {dtype}: " + diff_report(got, ref)
