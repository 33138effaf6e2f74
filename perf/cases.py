"""The work that a user of this package has it do, as cases that can be timed.

Each case is one call of a public entry point (``rusterize``,
``rasterize_device``, ``rasterize_batch_device``, ``SparseArray.to_numpy``) on
seeded synthetic inputs with the laws of ``rusterize_gb300.synth``: star
polygons with lognormal radii, random-walk lines and uniform points, in pixel
units of the raster.  The inputs are generated with torch (sorting, integer
prefix sums and element-wise arithmetic only, so that a seed gives the same
bits every time) and are resident on the GPU where the entry point takes them
there.
"""

from __future__ import annotations

import math
import struct

import numpy as np
import torch

from rusterize_gb300 import BatchJob, GeometryTable, SparseArray, raster_info, rusterize
from rusterize_gb300.device import DeviceTable, rasterize_batch_device, rasterize_device, upload
from rusterize_gb300.geometry import LINE, POINT, POLYGON

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
FNS = ("sum", "first", "last", "min", "max", "count", "any")


def listed() -> list[dict]:
    return [
        # one map tile of a tile server: a few dozen small parcels, 256 x 256 classes; launches and latency count
        {"name": "tile_256_last_u8", "kind": "fill", "n": 64, "nrows": 256, "ncols": 256, "nv_lo": 8, "nv_hi": 64,
         "median": 12.0, "sigma": 0.8, "holes": False, "res": 1.0, "fn": "last", "dtype": "uint8"},
        # the everyday call from Python: WKB blobs in, a numpy raster out (1,000 polygons over 1,000 x 1,000)
        {"name": "host_1k_wkb_last_f64", "kind": "host", "n": 1000, "nrows": 1000, "ncols": 1000, "nv_lo": 8,
         "nv_hi": 64, "median": 22.0, "sigma": 0.6, "holes": False, "res": 1.0, "fn": "last", "dtype": "float64"},
        # administrative boundaries on a 30 m grid: few wide polygons of thousands of vertices, ragged raster
        {"name": "boundaries_first_f32", "kind": "boundaries", "n": 200, "nrows": 7001, "ncols": 9003, "nv_lo": 2000,
         "nv_hi": 20000, "r_lo": 150.0, "r_hi": 2000.0, "res": 30.0, "fn": "first", "dtype": "float32"},
        # the benchmark's large fill, weighted density: 100,000 polygons with holes over 20,000 x 20,000, float64 sum
        {"name": "large_fill_sum_f64", "kind": "fill", "n": 100000, "nrows": 20000, "ncols": 20000, "nv_lo": 16,
         "nv_hi": 512, "median": 20.0, "sigma": 1.0, "holes": True, "res": 1.0, "fn": "sum", "dtype": "float64"},
        # the same geometries counted, the benchmark's second burn (overlap depth, uint32)
        {"name": "large_fill_count_u32", "kind": "fill", "n": 100000, "nrows": 20000, "ncols": 20000, "nv_lo": 16,
         "nv_hi": 512, "median": 20.0, "sigma": 1.0, "holes": True, "res": 1.0, "fn": "count", "dtype": "uint32"},
        # a mixed collection split into one presence band per category (by=): 16 bands of uint8 `any`
        {"name": "mixed_any_16_bands_u8", "kind": "mixed", "polys": 12500, "lines": 50000, "points": 250000,
         "nrows": 20000, "ncols": 20000, "bands": 16, "fn": "any", "dtype": "uint8"},
        # the same kind of collection at the benchmark's full size in one band: largest category of a pixel
        {"name": "mixed_max_i32", "kind": "mixed", "polys": 50000, "lines": 200000, "points": 1000000,
         "nrows": 40000, "ncols": 40000, "bands": 1, "fn": "max", "dtype": "int32"},
        # a point density raster (sightings, addresses): millions of points counted on an odd-sized grid
        {"name": "points_count_u32", "kind": "points", "n": 5000000, "nrows": 9999, "ncols": 10001, "fn": "count",
         "dtype": "uint32"},
        # road networks of several regions burned all_touched in one call (every pixel of a line once per line)
        {"name": "roads_touched_sum_f32", "kind": "batch", "shape": "lines", "jobs": 16, "n": 2000, "side_lo": 1024.0,
         "side_hi": 4096.0, "fn": "sum", "dtype": "float32", "touched": True},
        # many independent rasters of uneven size in one call, the function drawn per raster (the benchmark's batch)
        {"name": "batch_uneven_f32", "kind": "batch", "shape": "polygons", "jobs": 256, "n": 500, "side_lo": 256.0,
         "side_hi": 8192.0, "fn": "each", "dtype": "float32", "touched": False},
        # the sparse encoding: polygons burned to (row, col, value) triplets on the host
        {"name": "sparse_burn_sum_f64", "kind": "sparse", "n": 5000, "nrows": 4472, "ncols": 4472, "nv_lo": 16,
         "nv_hi": 512, "median": 20.0, "sigma": 1.0, "holes": True, "res": 1.0, "fn": "sum", "dtype": "float64"},
        # ... and such a stream materialised as a raster
        {"name": "sparse_to_numpy_sum_f64", "kind": "replay", "n": 5000, "nrows": 4472, "ncols": 4472, "nv_lo": 16,
         "nv_hi": 512, "median": 20.0, "sigma": 1.0, "holes": True, "res": 1.0, "fn": "sum", "dtype": "float64"},
    ]


def _logu(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    kind = rng.choice(("fill", "fill", "fill", "host", "boundaries", "mixed", "points", "batch", "batch", "sparse",
                       "replay"))
    if kind == "fill":  # from one tile to the large fill, with the polygons per pixel of those
        side = _logu(rng, 200, 20000)
        fn = rng.choice(FNS)
        dtype = rng.choice(("uint8", "int16", "int32", "uint32", "float32", "float64"))
        n = max(1, int(side * side * _logu(rng, 1e-4, 2.5e-4)))
        return {"kind": kind, "n": n, "nrows": max(1, int(side * rng.uniform(0.7, 1.0))), "ncols": int(side),
                "nv_lo": rng.randint(4, 16), "nv_hi": rng.randint(32, 512), "median": rng.uniform(8.0, 20.0),
                "sigma": rng.uniform(0.5, 1.0), "holes": rng.random() < 0.5,
                "res": rng.choice((1.0, 0.5, 10.0, 30.0)), "fn": fn, "dtype": dtype}
    if kind in ("host", "sparse", "replay"):
        side = _logu(rng, 300, 3000 if kind == "host" else 4400)
        return {"kind": kind, "n": max(1, int(side * side * _logu(rng, 1e-4, 2.5e-4))),
                "nrows": max(1, int(side * rng.uniform(0.7, 1.0))), "ncols": int(side), "nv_lo": 8,
                "nv_hi": rng.randint(32, 256), "median": rng.uniform(8.0, 20.0), "sigma": rng.uniform(0.5, 1.0),
                "holes": rng.random() < 0.5,
                "res": rng.choice((1.0, 0.5, 2.0) if kind == "sparse" else (1.0, 0.5, 10.0)),
                "fn": rng.choice(("sum", "first", "last", "max")),
                "dtype": rng.choice(("float32", "float64", "int32"))}
    if kind == "boundaries":
        side = _logu(rng, 1000, 9000)
        return {"kind": kind, "n": rng.randint(10, 200), "nrows": int(side * rng.uniform(0.6, 1.0)),
                "ncols": int(side), "nv_lo": 500, "nv_hi": rng.randint(2000, 20000), "r_lo": side * 0.02,
                "r_hi": side * 0.22, "res": rng.choice((1.0, 10.0, 30.0)),
                "fn": rng.choice(("first", "last", "sum", "max")), "dtype": rng.choice(("float32", "uint8", "int32"))}
    if kind == "mixed":
        side = _logu(rng, 2000, 20000)
        k = side * side / 1.6e9
        bands = rng.choice((1, 1, 5, 16))
        return {"kind": kind, "polys": max(1, int(50000 * k)), "lines": max(1, int(200000 * k)),
                "points": max(1, int(1000000 * k)), "nrows": int(side * rng.uniform(0.8, 1.0)), "ncols": int(side),
                "bands": bands, "fn": rng.choice(("any", "max", "last", "count")),
                "dtype": "uint8" if bands == 16 else rng.choice(("uint8", "int32"))}
    if kind == "points":
        side = _logu(rng, 500, 10000)
        return {"kind": kind, "n": int(_logu(rng, 1e4, 5e6)), "nrows": int(side * rng.uniform(0.7, 1.0)),
                "ncols": int(side), "fn": rng.choice(("count", "any", "last")),
                "dtype": rng.choice(("uint8", "uint32"))}
    if rng.random() < 0.3:
        return {"kind": "batch", "shape": "lines", "jobs": rng.randint(2, 16), "n": int(_logu(rng, 100, 2000)),
                "side_lo": 300.0, "side_hi": _logu(rng, 500, 4096), "fn": rng.choice(("sum", "last", "any")),
                "dtype": rng.choice(("float32", "uint8")), "touched": True}
    return {"kind": "batch", "shape": "polygons", "jobs": int(_logu(rng, 4, 256)), "n": int(_logu(rng, 50, 500)),
            "side_lo": 256.0, "side_hi": _logu(rng, 600, 6000), "fn": "each", "dtype": "float32", "touched": False}


# ---- generators (pixel units: x to the right, y down from the raster's top) ----

def _rand(gen, n: int) -> torch.Tensor:
    return torch.rand(n, generator=gen, dtype=torch.float64, device=DEV)


def _dev(a) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _offsets(sizes) -> np.ndarray:
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)


def _closed_rings(x, y, ring, counts):
    """Vertices (ring by ring) with every ring's first vertex repeated at its end."""
    total, nr = len(x), len(counts)
    xy = torch.empty((total + nr, 2), dtype=torch.float64, device=DEV)
    pos = torch.arange(total, device=DEV) + ring
    xy[pos, 0], xy[pos, 1] = x, y
    sizes = counts + 1
    starts = _dev(np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int64))
    xy[starts + _dev(counts)] = xy[starts]
    return xy, sizes


def _star_rings(gen, counts, cx, cy, radius):
    """Star rings: sorted uniform angles, vertex radius R * U[0.4, 1]."""
    ring = torch.repeat_interleave(torch.arange(len(counts), device=DEV), _dev(counts))
    total = len(ring)
    ang = (torch.sort(ring.double() + _rand(gen, total)).values - ring) * (2.0 * math.pi)
    rad = _dev(radius)[ring] * (0.4 + 0.6 * _rand(gen, total))
    return _closed_rings(_dev(cx)[ring] + rad * torch.cos(ang), _dev(cy)[ring] + rad * torch.sin(ang), ring, counts)


def _polygons(rng, gen, n, nrows, ncols, nv, median, sigma, holes, r_max=2000.0):
    """(rings per polygon, ring sizes, hole flags, vertices) of n star polygons with 0-3 holes."""
    radius = np.clip(np.exp(np.log(median) + rng.normal(0.0, sigma, n)), 2.0, r_max)
    cx, cy = rng.uniform(0, ncols, n), rng.uniform(0, nrows, n)
    rings = 1 + (rng.integers(0, 4, n) if holes else np.zeros(n, dtype=np.int64))
    of = np.repeat(np.arange(n), rings)
    first = np.concatenate([[0], np.cumsum(rings)[:-1]])
    hole = np.ones(len(of), dtype=bool)
    hole[first] = False
    counts = np.where(hole, rng.integers(8, 65, len(of)), np.repeat(rng.integers(nv[0], nv[1] + 1, n), rings))
    shrink = np.where(hole, rng.uniform(0.1, 0.3, len(of)), 1.0)
    dx, dy = (np.where(hole, rng.uniform(-0.25, 0.25, len(of)), 0.0) for _ in range(2))
    xy, sizes = _star_rings(gen, counts.astype(np.int64), cx[of] + dx * radius[of], cy[of] + dy * radius[of],
                            radius[of] * shrink)
    return rings, sizes, hole, xy


def _moved_polygons(rng, n, nrows, ncols, nv, median, sigma, holes):
    """Polygons whose shapes depend on the arguments alone, moved by whole pixels to places inside the raster that
    `rng` draws: every draw writes the same number of pixels, at other places (coordinates on a 2^-20 px grid)."""
    shapes, gen = _gens(n * 1000003 + nrows)
    r_max = max(2.0, 0.2 * min(nrows, ncols))
    rings, sizes, hole, xy = _polygons(shapes, gen, n, 1.0, 1.0, nv, median, sigma, holes, r_max)
    xy = torch.round(xy * 2.0**20) / 2.0**20
    m = math.ceil(1.3 * r_max) + 2
    to = np.stack([rng.integers(m, max(m + 1, ncols - m), n), rng.integers(m, max(m + 1, nrows - m), n)], axis=1)
    of = np.repeat(np.repeat(np.arange(n), rings), sizes)
    return rings, sizes, hole, xy + _dev(to.astype(np.float64))[_dev(of)]


def _boundaries(rng, gen, n, nrows, ncols, nv, r):
    """Closed boundaries: a circle bent by a few harmonics with a fine irregular edge."""
    radius = np.exp(rng.uniform(math.log(r[0]), math.log(r[1]), n))
    cx, cy = rng.uniform(0, ncols, n), rng.uniform(0, nrows, n)
    counts = np.exp(rng.uniform(math.log(nv[0]), math.log(nv[1]), n)).astype(np.int64)
    ring = torch.repeat_interleave(torch.arange(n, device=DEV), _dev(counts))
    within = torch.arange(len(ring), device=DEV) - _dev(np.concatenate([[0], np.cumsum(counts)[:-1]]))[ring]
    ang = within.double() * (2.0 * math.pi) / _dev(counts)[ring]
    shape = 0.8 + 0.004 * (_rand(gen, len(ring)) - 0.5)
    for k in (2, 3, 5, 9, 17):
        shape = shape + (0.25 / k) * torch.sin(k * ang + _dev(rng.uniform(0, 2 * math.pi, n))[ring])
    rad = _dev(radius)[ring] * shape
    xy, sizes = _closed_rings(_dev(cx)[ring] + rad * torch.cos(ang), _dev(cy)[ring] + rad * torch.sin(ang), ring,
                              counts)
    return np.ones(n, dtype=np.int64), sizes, np.zeros(n, dtype=bool), xy


def _lines(rng, gen, n, nrows, ncols):
    """Random walks of 2-200 vertices with steps of U[1, 20] pixels."""
    counts = rng.integers(2, 201, n).astype(np.int64)
    line = torch.repeat_interleave(torch.arange(n, device=DEV), _dev(counts))
    total = len(line)
    step, head = 1.0 + 19.0 * _rand(gen, total), 2.0 * math.pi * _rand(gen, total)
    first = _dev(np.concatenate([[0], np.cumsum(counts)[:-1]]))
    cols = []
    for f, size in ((torch.cos, ncols), (torch.sin, nrows)):
        # the walk in fixed point (2^-24 px): integer prefix sums do not depend on their order
        walk = torch.cumsum(torch.round(step * f(head) * 2.0**24).to(torch.int64), 0)
        cols.append((walk - walk[first][line]).double() / 2.0**24 + _dev(rng.uniform(0, size, n))[line])
    return counts, torch.stack(cols, dim=1)


def _world(xy, nrows, res):
    """Pixel units -> world coordinates (y up) of a raster with its lower left corner at the origin."""
    return torch.stack([xy[:, 0] * res, (nrows - xy[:, 1]) * res], dim=1).contiguous()


def _info(nrows, ncols, res):
    return raster_info(None, shape=(nrows, ncols), extent=(0.0, 0.0, ncols * res, nrows * res))


def _poly_table(rings, sizes, hole, xy) -> GeometryTable:
    n = len(rings)
    return GeometryTable(np.arange(n + 1), np.full(n, POLYGON, np.uint8), _offsets(rings), _offsets(sizes),
                         hole.astype(np.uint8), xy.cpu().numpy())


def _simple_table(kind, counts, xy) -> GeometryTable:
    n = len(counts)
    ar = np.arange(n + 1, dtype=np.uint64)
    return GeometryTable(ar, np.full(n, kind, np.uint8), ar, _offsets(counts), np.zeros(n, np.uint8), xy.cpu().numpy())


def _values(rng, n, dtype):
    if np.dtype(dtype).kind == "f":
        return rng.uniform(0, 1, n).astype(dtype)
    return rng.integers(1, 100, n).astype(dtype)


def _background(dtype):
    return float("nan") if np.dtype(dtype).kind == "f" else 0


def _gens(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return np.random.default_rng(seed), gen


def _polygon_table(case, rng, gen) -> GeometryTable:
    nr, nc = case["nrows"], case["ncols"]
    nv = (case["nv_lo"], max(case["nv_lo"], case["nv_hi"]))
    if case["kind"] == "boundaries":
        r, s, h, xy = _boundaries(rng, gen, case["n"], nr, nc, nv, (case["r_lo"], case["r_hi"]))
    elif case["kind"] == "sparse":  # the number of triplets does not depend on the seed
        r, s, h, xy = _moved_polygons(rng, case["n"], nr, nc, nv, case["median"], case["sigma"], case["holes"])
    else:
        r, s, h, xy = _polygons(rng, gen, case["n"], nr, nc, nv, case["median"], case["sigma"], case["holes"])
    return _poly_table(r, s, h, _world(xy, nr, case["res"]))


def _wkb(t: GeometryTable) -> list[bytes]:
    """Each geometry of a polygon table as an ISO WKB Polygon."""
    out = []
    ro, vo, xy = t.ring_offsets.tolist(), t.vertex_offsets.tolist(), t.xy
    for g in range(t.n_geoms):
        rings = range(ro[g], ro[g + 1])
        body = [struct.pack("<I", vo[r + 1] - vo[r]) + xy[vo[r]:vo[r + 1]].tobytes() for r in rings]
        out.append(struct.pack("<BII", 1, 3, len(body)) + b"".join(body))
    return out


def _batch(case, rng, gen):
    lo, hi = math.log(case["side_lo"]), math.log(case["side_hi"])
    # log-uniform sides, the same for every seed, in mixed order
    at = (np.random.default_rng(case["jobs"]).permutation(case["jobs"]) + 0.5) / case["jobs"]
    sides = np.round(np.exp(lo + (hi - lo) * at)).astype(np.int64)
    size = np.dtype(case["dtype"]).itemsize
    step = (sides * sides * size + 255) // 256 * 256
    at = np.concatenate([[0], np.cumsum(step)])
    buf = torch.zeros(int(at[-1]), dtype=torch.uint8, device=DEV)  # every job's raster, 256-byte aligned
    jobs, outs = [], []
    for j, side in enumerate(sides.tolist()):
        # the median job has n geometries
        n = int(np.clip(round(case["n"] * math.exp(rng.normal(0.0, 1.0))), 10, 50000))
        if case["shape"] == "lines":
            counts, xy = _lines(rng, gen, n, side, side)
            t = _simple_table(LINE, counts, _world(xy, side, 1.0))
        else:
            r, s, h, xy = _polygons(rng, gen, n, side, side, (8, 256), 0.02 * side, 1.0, False, 0.25 * side)
            t = _poly_table(r, s, h, _world(xy, side, 1.0))
        fn = FNS[int(rng.integers(0, 6))] if case["fn"] == "each" else case["fn"]
        jobs.append(BatchJob(DeviceTable.upload(t), _info(side, side, 1.0), upload(_values(rng, n, case["dtype"])),
                             fn, _background(case["dtype"])))
        outs.append(buf[int(at[j]):int(at[j]) + side * side * size])
    return {"jobs": jobs, "outs": outs, "buf": buf.view(getattr(torch, case["dtype"]))}


def prepare(case, seed):
    kind = case["kind"]
    rng, gen = _gens(seed)
    st = {"case": case}
    if kind == "batch":
        return st | _batch(case, rng, gen)
    nr, nc, dtype = case["nrows"], case["ncols"], case["dtype"]
    st["background"] = _background(dtype)
    if kind == "mixed":
        r, s, h, pxy = _polygons(rng, gen, case["polys"], nr, nc, (16, 512), 20.0, 1.0, True)
        counts, lxy = _lines(rng, gen, case["lines"], nr, nc)
        qxy = torch.stack([_rand(gen, case["points"]) * nc, _rand(gen, case["points"]) * nr], dim=1)
        ones = np.ones(case["points"], dtype=np.int64)
        table = GeometryTable.concat([_poly_table(r, s, h, _world(pxy, nr, 1.0)),
                                      _simple_table(LINE, counts, _world(lxy, nr, 1.0)),
                                      _simple_table(POINT, ones, _world(qxy, nr, 1.0))])
        category = rng.integers(0, 16, table.n_geoms)
        st["values"] = upload((1 + category).astype(dtype))
        st["bands"] = upload((category % case["bands"]).astype(np.uint32)) if case["bands"] > 1 else None
        st["n_bands"] = case["bands"]
        st["info"] = _info(nr, nc, 1.0)
    elif kind == "points":
        xy = torch.stack([_rand(gen, case["n"]) * nc, _rand(gen, case["n"]) * nr], dim=1)
        table = _simple_table(POINT, np.ones(case["n"], dtype=np.int64), _world(xy, nr, 1.0))
        st["values"] = None if case["fn"] == "count" else upload(_values(rng, case["n"], dtype))
        st["info"] = _info(nr, nc, 1.0)
    else:
        table = _polygon_table(case, rng, gen)
        values = _values(rng, case["n"], dtype)
        res = case["res"]
        st["info"] = _info(nr, nc, res)
        if kind in ("host", "sparse", "replay"):
            args = {"out_shape": (nr, nc), "extent": (0.0, 0.0, nc * res, nr * res), "burn": values,
                    "fun": case["fn"], "background": st["background"], "dtype": dtype}
            if kind == "replay":  # the stream of an earlier burn
                st["sparse"] = rusterize(table, encoding="sparse", **args)
            else:
                st["args"] = args
                st["data"] = _wkb(table) if kind == "host" else table
            return st
        st["values"] = None if case["fn"] in ("count", "any") else upload(values)
    st["table"] = DeviceTable.upload(table)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "batch":
        rasterize_batch_device(st["jobs"], dtype=case["dtype"], outs=st["outs"], all_touched=case["touched"])
        return st["buf"]
    if kind == "host":
        return rusterize(st["data"], encoding="numpy", **st["args"])
    if kind == "sparse":
        sp: SparseArray = rusterize(st["data"], encoding="sparse", **st["args"])
        return {"row": sp.rows.view(np.int64), "col": sp.cols.view(np.int64), "values": sp.values}
    if kind == "replay":
        return st["sparse"].to_numpy()
    return rasterize_device(st["table"], st["info"], fn=case["fn"], background=st["background"], dtype=case["dtype"],
                            values=st["values"], bands=st.get("bands"), n_bands=st.get("n_bands", 1))


# ---- what the path cannot do without -------------------------------------------

def _star_pixels(n, median, sigma, holes):
    # expected area of a star ring of radius R is 0.49 pi R^2; three half holes of 0.2 R cut out about 6%
    return n * 0.49 * math.pi * (median * median * math.exp(2 * sigma * sigma)) * (0.94 if holes else 1.0)


def work(case):
    kind, size = case["kind"], np.dtype(case["dtype"]).itemsize
    if kind == "batch":
        span = math.log(case["side_hi"] / case["side_lo"])
        px = (case["side_hi"] ** 2 - case["side_lo"] ** 2) / (2 * span)  # mean of a log-uniform side, squared
        n = case["n"] * math.exp(0.5)
        verts = n * (101 if case["shape"] == "lines" else 133)
        return {"bytes": case["jobs"] * (px * size + verts * 16 + n * (size + 24)), "flops": 0.0}
    px = case["nrows"] * case["ncols"]
    if kind == "mixed":
        geoms = case["polys"] + case["lines"] + case["points"]
        verts = case["polys"] * (265 + 1.5 * 37) + case["lines"] * 101 + case["points"]
        rings = case["polys"] * 2.5 + case["lines"] + case["points"]
        return {"bytes": px * case["bands"] * size + verts * 16 + rings * 8 + geoms * (size + 4 + 17), "flops": 0.0}
    if kind == "points":
        return {"bytes": px * size + case["n"] * (16 + 25), "flops": 0.0}
    n = case["n"]
    if kind == "boundaries":
        mean = (case["nv_hi"] - case["nv_lo"]) / math.log(case["nv_hi"] / case["nv_lo"])
        return {"bytes": px * size + n * (mean * 16 + size + 25), "flops": 0.0}
    verts = n * ((case["nv_lo"] + case["nv_hi"]) / 2 + 1 + (1.5 * 37 if case["holes"] else 0))
    inputs = verts * 16 + n * (size + 17 + 8 * (2.5 if case["holes"] else 1))
    triplets = _star_pixels(n, case["median"], case["sigma"], case["holes"])
    if kind == "sparse":
        return {"bytes": inputs + triplets * (16 + size), "flops": 0.0}
    if kind == "replay":
        return {"bytes": triplets * (16 + size) + px * size, "flops": 0.0}
    return {"bytes": inputs + px * size, "flops": 0.0}


# ---- the result in 64 bits, by numpy ---------------------------------------------

def exact(case, seed):
    """Polygons burned scanline by scanline in float64, one geometry after another."""
    if case["kind"] not in ("fill", "host", "boundaries", "replay") or np.dtype(case["dtype"]).kind != "f":
        return None
    if case["kind"] == "boundaries":
        rows = case["n"] * 2 * case["r_hi"]
    else:
        rows = case["n"] * 4 * case["median"] * math.exp(case["sigma"] ** 2 / 2) * 3
    if rows > 3e6 or case["nrows"] * case["ncols"] > 1e8:
        return None
    rng, gen = _gens(seed)
    table = _polygon_table(case, rng, gen)
    values = _values(rng, case["n"], case["dtype"]).astype(np.float64)
    nr, nc, res, fn = case["nrows"], case["ncols"], case["res"], case["fn"]
    ro, vo = table.ring_offsets.astype(np.int64), table.vertex_offsets.astype(np.int64)
    px, py = table.xy[:, 0] / res, (nr * res - table.xy[:, 1]) / res
    edge = np.ones(len(px) - 1, dtype=bool)
    edge[vo[1:-1] - 1] = False  # no edge from one ring's end to the next ring's start
    a = np.flatnonzero(edge)
    geom = np.searchsorted(vo[ro], a, side="right") - 1
    top = np.where(py[a] <= py[a + 1], a, a + 1)
    bot = 2 * a + 1 - top
    r0 = np.clip(np.ceil(py[top] - 0.5), 0, nr).astype(np.int64)
    r1 = np.clip(np.ceil(py[bot] - 0.5), 0, nr).astype(np.int64)
    keep = r1 > r0
    top, bot, geom, r0, r1 = top[keep], bot[keep], geom[keep], r0[keep], r1[keep]
    cnt = r1 - r0
    e = np.repeat(np.arange(len(cnt)), cnt)
    row = np.arange(len(e)) - np.repeat(np.cumsum(cnt) - cnt, cnt) + r0[e]
    slope = (px[bot] - px[top]) / (py[bot] - py[top])
    x = px[top][e] + ((row + 0.5) - py[top][e]) * slope[e]
    col = np.clip(np.floor(x + 0.5), 0, nc).astype(np.int64)
    order = np.lexsort((col, row, geom[e]))
    col, row, g = col[order], row[order], geom[e][order]
    out = np.full((nr, nc), np.nan)
    vals = values[g[0::2]].tolist()
    for y, xa, xb, v in zip(row[0::2].tolist(), col[0::2].tolist(), col[1::2].tolist(), vals):
        s = out[y, xa:xb]
        if fn == "last":
            s[:] = v
        elif fn == "any":
            s[:] = 1.0
        else:
            new = np.isnan(s)
            if fn == "sum":
                s[:] = np.where(new, v, s + v)
            elif fn == "count":
                s[:] = np.where(new, 1.0, s + 1.0)
            elif fn == "first":
                s[new] = v
            else:
                s[:] = np.where(new, v, np.minimum(s, v) if fn == "min" else np.maximum(s, v))
    return out[None]
