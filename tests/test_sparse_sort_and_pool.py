"""The radix sort under the sparse paths at its limits (tiles of 4,096 elements,
passes of up to 9 bits, 32- and 64-bit keys), the triplets' expansion, and the
host buffers that freed sparse results leave to the next ones."""

import concurrent.futures as cf

import numpy as np
import pytest

import oracle
import rusterize_gb300 as rz
from rusterize_gb300 import synth
from rusterize_gb300.engine import rasterize_table_sparse, sparse_build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrows,ncols", [(1, 1), (1, 2), (16, 32), (16, 33), (512, 512), (513, 512)])
@pytest.mark.parametrize("n", [1, 511, 4095, 4096, 4097, 12289])
def test_replay_sizes(n, nrows, ncols):
    rng = np.random.default_rng(n + ncols)
    rows = rng.integers(0, nrows, n).astype(np.uint64)
    cols = rng.integers(0, ncols, n).astype(np.uint64)
    vals = rng.uniform(-1, 1, n).astype(np.float32)
    counts = np.array([n], dtype=np.uint64)
    got = sparse_build(counts, rows, cols, vals, nrows, ncols, fn="sum", background=np.nan)
    ref = np.full((1, nrows, ncols), np.nan, dtype=np.float32)
    order = np.argsort(rows * np.uint64(ncols) + cols, kind="stable")
    for r, c, v in zip(rows[order].tolist(), cols[order].tolist(), vals[order]):
        x = ref[0, r, c]
        ref[0, r, c] = v if np.isnan(x) else np.float32(x + v)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


def test_replay_keys_beyond_32_bits():
    nrows, ncols, n = 65537, 65540, 50000
    rng = np.random.default_rng(8)
    rows = rng.integers(0, nrows, n).astype(np.uint64)
    cols = rng.integers(0, ncols, n).astype(np.uint64)
    rows[:3], cols[:3] = [0, nrows - 1, nrows - 1], [0, 0, ncols - 1]
    rows[-1000:], cols[-1000:] = rows[:1000], cols[:1000]
    vals = rng.integers(1, 256, n).astype(np.uint8)
    got = sparse_build(np.array([n], np.uint64), rows, cols, vals, nrows, ncols, fn="last", background=0)
    want = {}
    for r, c, v in zip(rows.tolist(), cols.tolist(), vals.tolist()):
        want[r, c] = v
    assert all(got[0, r, c] == v for (r, c), v in want.items())
    assert np.count_nonzero(got) == len(want)


@pytest.mark.parametrize("side,n,dtype", [(40, 3, "uint8"), (300, 60, "int16"), (900, 200, "float64")])
def test_triplets_and_buffers_of_freed_results(side, n, dtype):
    jobs = []
    for k in range(4):
        rng = np.random.default_rng(100 * n + k)
        t = synth.star_polygons(rng, n, (3, 30), rng.uniform(0.3, side * 0.1, n), rng.uniform(0, side, n),
                                rng.uniform(0, side, n))
        v = rng.integers(1, 100, n).astype(dtype)
        info = rz.RasterInfo(nrows=side, ncols=side, xmin=0.0, xmax=float(side), ymin=0.0, ymax=float(side), xres=1.0,
                             yres=1.0)
        bands = rng.integers(0, 3, n).astype(np.uint32)
        o = oracle.rasterize_sparse(t, side, side, 0.0, float(side), 0.0, float(side), 1.0, 1.0, values=v, fn="sum",
                                    dtype=dtype, bands=bands, n_bands=3)
        jobs.append((t, info, v, bands, [np.asarray(a) for a in o]))

    def ordered(counts, rows, cols, vals):
        b = np.repeat(np.arange(len(counts)), counts.astype(np.int64))
        i = np.lexsort((cols, rows, b))  # stable: one pixel's writes keep their order
        return b[i], rows[i], cols[i], vals[i]

    def same(got, o):
        return all(np.array_equal(x, y) for x, y in zip(ordered(*got), ordered(*o)))

    def work(seed):
        ctx = rz.Context(0)
        rng = np.random.default_rng(seed)
        kept = []
        for _ in range(6):  # results live on beside ones whose buffers were freed and taken again
            t, info, v, bands, o = jobs[int(rng.integers(0, 4))]
            got = rasterize_table_sparse(t, info, values=v, fn="sum", dtype=dtype, bands=bands, n_bands=3, context=ctx)
            kept.append((got, o))
            if len(kept) > 3:
                kept.pop(int(rng.integers(0, 3)))
            if not all(same(g, r) for g, r in kept):
                return False
        ctx.close()
        return all(same(g, r) for g, r in kept)

    with cf.ThreadPoolExecutor(3) as ex:
        assert all(ex.map(work, range(3)))
