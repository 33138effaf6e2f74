"""Ordered fills of tiles, and of words of deeper tiles, with 65 to 256
records (sorted in registers, four or eight keys a lane, or in shared memory
where the parts are too far apart for one 32-bit key) and around, vs the
oracle: values of very different size, so that any other order gives other
sums, bit-exact."""

import numpy as np
import pytest

from rusterize_gb300 import geometry as G

from _util import diff_report, gpu_burn, oracle_burn, same_bits

pytestmark = pytest.mark.gpu

GRID = dict(nrows=1, ncols=512, xmin=0.0, xmax=512.0, ymin=0.0, ymax=1.0, xres=1.0, yres=1.0)


def check(xy, dtype, fn="sum"):
    n = len(xy)
    ar = np.arange(n + 1, dtype=np.uint64)
    t = G.GeometryTable(ar, np.zeros(n, np.uint8), ar, ar, np.zeros(n, np.uint8), xy)
    rng = np.random.default_rng(n)
    v = (rng.uniform(1, 2, n) * 10.0 ** rng.integers(-6, 7, n) * rng.choice((-1, 1), n)).astype(dtype)
    kw = dict(fn=fn, values=v, background=np.nan, dtype=dtype)
    got, ref = gpu_burn(t, GRID, **kw), oracle_burn(t, GRID, **kw)
    assert same_bits(got, ref), diff_report(got, ref)


def points(rng, n):
    """n points on 37 pixels of the tile, every word among them."""
    px = np.concatenate([np.arange(16) * 32 + 31, rng.integers(0, 512, 21)])
    return np.stack([rng.choice(px, n) + 0.5, np.full(n, 0.5)], axis=1)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [63, 64, 65, 96, 127, 128, 129, 160, 255, 256, 257])
def test_tile_depths(n, dtype):
    check(points(np.random.default_rng(n), n), dtype)


@pytest.mark.parametrize("n,span", [(100, (1 << 21) - 2), (100, (1 << 21) - 1), (200, (1 << 20) - 2),
                                    (200, (1 << 20) - 1)])
def test_tile_part_ranges(n, span):
    # the tile's last part lies `span` behind its first, across points outside the raster
    xy = points(np.random.default_rng(n), n)
    far = np.full((span + 1 - n, 2), -10.0)
    check(np.concatenate([xy[: n // 2], far, xy[n // 2:]]), "float32")


@pytest.mark.parametrize("n,span", [(64, 0), (127, 0), (128, 0), (129, 0), (255, 0), (256, 0), (257, 0), (600, 0),
                                    (100, (1 << 21) - 2), (100, (1 << 21) - 1)])
def test_word_depths(n, span):
    # one word of a tile too deep for one warp
    rng = np.random.default_rng(n + 1)
    word = np.stack([rng.integers(64, 84, n) + 0.5, np.full(n, 0.5)], axis=1)
    rest = np.stack([rng.integers(96, 128, 300) + 0.5, np.full(300, 0.5)], axis=1)
    far = np.full((max(0, span + 1 - n), 2), -10.0)
    check(np.concatenate([rest[:150], word[: n // 2], far, word[n // 2:], rest[150:]]), "float32")
    if not span:
        check(rng.permutation(np.concatenate([word, rest])), "float64")
