// rz_kernels.cuh -- validation, per-part planning, span generation
// (polygon scanlines, Bresenham lines, points) and the bucket scatter.
//
// Reference semantics restated here (ttrotto/rusterize, rust/src/):
//   geo/edges.rs:79-134              world->pixel, extract_point/ring/line filters
//   rasterization/burners.rs:40-91   Standard::burn_line (Bresenham)
//   rasterization/burners.rs:250-258 burn_point
//   rasterization/burners.rs:261-320 burn_polygon (active-edge scanline, even-odd)
//   rasterization/burn_geometry.rs   part semantics (pooled rings / edges)
#pragma once

#include <type_traits>

#include "rz_device.cuh"
#include "rz_line.cuh"
#include "rz_poly.cuh"

namespace rzd {

// ---------------------------------------------------------------- tables ----
// Reject tables that would make any later kernel read out of bounds, and map
// every part to its geometry.  (A range is written only when its end passes;
// the kernels after this one do nothing once an error is set.)  A lane writes
// its geometry's parts itself if they are few; the warp writes longer ranges
// together (one geometry of 1 M parts written by its lane took 77 ms).  In a
// table whose offsets go up and down the ranges can add up to the parts times
// the geometries, so the long ones stop once the error is known; the lane that
// sees the offsets fall sets it before it writes.
constexpr unsigned PART_RUN = 8;

__device__ __forceinline__ void tables_body(const Geo& geo, unsigned* part_geom, Ctrl* ctrl) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned long long tid = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i0 = tid - lane; i0 <= geo.n_geoms; i0 += stride) {
    const unsigned long long i = i0 + lane;
    unsigned long long a = 0, b = 0;  // the geometry's parts
    if (i <= geo.n_geoms) {
      a = geo.part_offsets[i];
      if ((i == 0 && a != 0) || (i == geo.n_geoms && a != geo.n_parts) ||
          (i > 0 && a < geo.part_offsets[i - 1]) || a > geo.n_parts)
        set_error(ctrl, ERR_BAD_TABLE, i);
      if (i < geo.n_geoms) b = geo.part_offsets[i + 1];
      if (b > geo.n_parts) b = 0;
    }
    const bool run = b > a && b - a > PART_RUN;
    if (!run)
      for (unsigned long long p = a; p < b; ++p) part_geom[p] = (unsigned)i;
    unsigned runs = __ballot_sync(0xFFFFFFFFu, run);
    while (runs) {
      const int j = __ffs(runs) - 1;
      runs &= runs - 1u;
      const unsigned long long ja = __shfl_sync(0xFFFFFFFFu, a, j), jb = __shfl_sync(0xFFFFFFFFu, b, j);
      for (unsigned long long p0 = ja; p0 < jb; p0 += 1024) {
        if (p0 > ja && __any_sync(0xFFFFFFFFu, *reinterpret_cast<volatile unsigned*>(&ctrl->err) != 0u)) break;
        const unsigned long long pe = min(p0 + 1024, jb);
        for (unsigned long long p = p0 + lane; p < pe; p += 32) part_geom[p] = (unsigned)(i0 + (unsigned)j);
      }
    }
  }
  for (unsigned long long i = tid; i <= geo.n_parts; i += stride) {
    const unsigned long long a = geo.ring_offsets[i];
    if ((i == 0 && a != 0) || (i == geo.n_parts && a != geo.n_rings) ||
        (i > 0 && a < geo.ring_offsets[i - 1]) || a > geo.n_rings)
      set_error(ctrl, ERR_BAD_TABLE, (1ull << 62) | i);
    if (i < geo.n_parts && geo.part_kind[i] > 2) set_error(ctrl, ERR_BAD_KIND, i);
  }
  for (unsigned long long i = tid; i <= geo.n_rings; i += stride) {
    const unsigned long long a = geo.vertex_offsets[i];
    if ((i == 0 && a != 0) || (i == geo.n_rings && a != geo.n_vertices) ||
        (i > 0 && a < geo.vertex_offsets[i - 1]) || a > geo.n_vertices)
      set_error(ctrl, ERR_BAD_TABLE, (2ull << 62) | i);
  }
}

__global__ void k_tables(Geo geo, unsigned* part_geom, Ctrl* ctrl) { tables_body(geo, part_geom, ctrl); }

__device__ __forceinline__ void bands_body(const Geo& geo, unsigned n_bands, Ctrl* ctrl) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < geo.n_geoms;
       i += stride)
    if (geo.bands[i] >= n_bands) set_error(ctrl, ERR_BAD_BAND, i);
}

__global__ void k_check_bands(Geo geo, unsigned n_bands, Ctrl* ctrl) {
  if (ctrl->err) return;
  bands_body(geo, n_bands, ctrl);
}

// ------------------------------------------------------------ part plans ----
// Smallest and largest world coordinates of a polygon part, on the integer
// pipe: monotone keys of the bit patterns, NaN excluded (edges with NaN never
// burn).
struct Extent {
  long long ylo = 0x7FFFFFFFFFFFFFFFll, yhi = (long long)0x8000000000000000ull;
  long long xlo = 0x7FFFFFFFFFFFFFFFll, xhi = (long long)0x8000000000000000ull;
  int nan_x = 0;

  __device__ __forceinline__ void fold(double2 w) {
    const unsigned long long by = f64_bits(w.y), bx = f64_bits(w.x);
    if (!nan_bits(by)) {
      const long long k = (long long)(by ^ ((unsigned long long)((long long)by >> 63) >> 1));
      ylo = min(ylo, k);
      yhi = max(yhi, k);
    }
    if (!nan_bits(bx)) {
      const long long k = (long long)(bx ^ ((unsigned long long)((long long)bx >> 63) >> 1));
      xlo = min(xlo, k);
      xhi = max(xhi, k);
    } else {
      nan_x = 1;
    }
  }
  // vertices first, first + 32 k, ... below ve, with four loads in flight per
  // lane and step; min / max are idempotent, so a missing vertex folds
  // another one again
  __device__ __forceinline__ void fold_range(const double2* xy, unsigned long long first, unsigned long long ve,
                                             unsigned long long step) {
    for (unsigned long long v = first; v < ve; v += step) {
      const double2 w = xy[v];
      const double2 w2 = v + 32 < ve ? xy[v + 32] : w;
      const double2 w3 = v + 64 < ve ? xy[v + 64] : w;
      const double2 w4 = v + 96 < ve ? xy[v + 96] : w;
      fold(w);
      fold(w2);
      fold(w3);
      fold(w4);
    }
  }
  __device__ __forceinline__ void merge(const Extent& o) {
    ylo = min(ylo, o.ylo);
    yhi = max(yhi, o.yhi);
    xlo = min(xlo, o.xlo);
    xhi = max(xhi, o.xhi);
    nan_x |= o.nan_x;
  }
  // smallest of the lanes' keys: by their high words, then by the low words
  // of the lanes that have the smallest high word
  static __device__ __forceinline__ long long warp_min(long long k) {
    const int hi = (int)(k >> 32), m = __reduce_min_sync(0xFFFFFFFFu, hi);
    const unsigned lo = __reduce_min_sync(0xFFFFFFFFu, hi == m ? (unsigned)k : 0xFFFFFFFFu);
    return ((long long)m << 32) | lo;
  }
  __device__ __forceinline__ void warp_merge() {
    ylo = warp_min(ylo);
    yhi = ~warp_min(~yhi);
    xlo = warp_min(xlo);
    xhi = ~warp_min(~xhi);
    nan_x = __any_sync(0xFFFFFFFFu, nan_x);
  }
};

// The window heights of a planned polygon part, with the small bitmap of one
// warp (narrow) or the bitmap of a block; returns its number of windows.
__device__ __forceinline__ unsigned long long set_windows(const Tune& tn, bool narrow, PartPlan& pl) {
  const int rows = pl.row1 - pl.row0;
  if (pl.bw > BITMAP_WORDS) {  // wider than one bitmap: windows of columns too
    pl.wr = min(COLWIN_ROWS, tn.rows_per_window);
    const unsigned ncw = (unsigned)((pl.bw + COLWIN_WORDS - 1) / COLWIN_WORDS);
    pl.ncw = ncw | (pl.ncw & RINGS_CLOSED);
    return (unsigned long long)((rows + pl.wr - 1) / pl.wr) * ncw;
  }
  pl.wr = min((narrow ? SMALL_BITMAP_WORDS : BITMAP_WORDS) / pl.bw, tn.rows_per_window);
  return (unsigned long long)((rows + pl.wr - 1) / pl.wr);
}

// The row range and bitmap window geometry of a polygon part from its extent
// (the world->pixel map is monotone, so transforming the extremes gives the
// pixel extremes).  Returns its number of windows, and whether one warp's
// bitmap holds their rows (narrow).
__device__ __forceinline__ unsigned long long plan_polygon(const Grid& g, const JobDims& jd, const Extent& ex,
                                                           const Tune& tn, PartPlan& pl, bool& narrow) {
  narrow = false;
  auto unkey = [](long long k) {
    const unsigned long long b = (unsigned long long)k ^ ((unsigned long long)(k >> 63) >> 1);
    return __longlong_as_double((long long)b);
  };
  if (ex.ylo > ex.yhi) return 0;
  // pixel y decreases with world y
  const int row0 = max(row_ceil(to_py(g, unkey(ex.yhi)), jd.nrows), jd.row_lo);
  const int row1 = min(row_ceil(to_py(g, unkey(ex.ylo)), jd.nrows), jd.row_hi);
  if (row1 <= row0) return 0;
  double c_lo = 0.0, c_hi = (double)jd.ncols;
  if (ex.xlo <= ex.xhi && !ex.nan_x) {
    const double pxl = to_px(g, unkey(ex.xlo)), pxh = to_px(g, unkey(ex.xhi));
    // crossings are interpolations between edge end points; allow a
    // rounding margin that grows with the coordinate magnitude
    const double mag = fmax(fabs(pxl), fabs(pxh));
    const double margin = 2.0 + ldexp(mag, -40);
    c_lo = floor(pxl - margin);
    c_hi = ceil(pxh + margin);
  }
  // the bitmap starts on a 32-pixel word so that its words are raster words
  const int col0 = (c_lo <= 0.0 ? 0 : (c_lo >= jd.ncols ? jd.ncols : (int)c_lo)) & ~31;
  const int colmax = c_hi <= 0.0 ? 0 : (c_hi >= jd.ncols ? jd.ncols : (int)c_hi);
  const int bw = (colmax - col0 + 1 + 31) >> 5;
  pl.row0 = row0;
  pl.row1 = row1;
  pl.col0 = col0;
  pl.bw = bw;
  narrow = bw <= tn.narrow_max_words;
  return set_windows(tn, narrow, pl);
}

// chunk_rows of chunks [c0, c1) of a part with nv vertices from vs on, by
// one warp: a range of rows that holds the first scanlines of the chunk's
// vertices and of the one before them.  An edge ending in the chunk crosses
// rows [a, b) of the first scanlines of its ends, so a window [r0, r1) needs
// the chunk only if its smallest is < r1 and its largest > r0.  The rows are
// estimated in FP32 with a margin for its rounding (an FP64 division per
// vertex would take most of the kernel).  Returns how many (chunk, window)
// pairs that makes with windows of pl.wr rows, to within one per chunk.
__device__ __forceinline__ float chunk_ranges(const Geo& geo, const Grid& g, const PartPlan& pl, unsigned long long vs,
                                              unsigned nv, unsigned c0, unsigned c1, int2* out) {
  const int lane = threadIdx.x & 31;
  const double2* xy = geo.xy + vs;
  const float inv = 1.0f / (float)g.yres, inv_wr = 1.0f / (float)pl.wr;
  const bool usable = inv > 0.0f && inv < 1e30f;
  auto world = [&](unsigned c) { return xy[min(32u * c + (unsigned)lane, nv - 1u)].y; };
  auto rows = [&](double wy, int& lo, int& hi) {  // holds clamp(ceil(y - 0.5), 0, nrows); NaN: row 0
    const float f = (float)__dsub_rn(g.ymax, wy) * inv;
    const float m = 0.51f + fabsf(f) * 9.5367431640625e-07f;  // 2^-20
    // clamped as integers: a raster's row count need not have an exact float
    lo = min(max(__float2int_rd(f - m), 0), pl.nrows);        // saturates; NaN: 0
    hi = min(max(__float2int_ru(f + m), 0), pl.nrows);
    if (!usable) {
      lo = 0;
      hi = pl.nrows;
    }
    hi = max(hi, lo);
  };
  int plo = 0x7FFFFFFF, phi = -1;  // rows of the vertex before the chunk
  if (c0 > 0) rows(xy[32ull * c0 - 1].y, plo, phi);
  float pairs = 0.0f;
  double y0 = c0 < c1 ? world(c0) : 0.0, y1 = c0 + 1 < c1 ? world(c0 + 1) : 0.0;  // two chunks of loads in flight
  for (unsigned c = c0; c < c1; ++c) {
    const double y2 = c + 2 < c1 ? world(c + 2) : 0.0;
    int lo, hi;
    rows(y0, lo, hi);
    const int wlo = min(plo, __reduce_min_sync(0xFFFFFFFFu, lo)), whi = max(phi, __reduce_max_sync(0xFFFFFFFFu, hi));
    if (lane == 0) out[c] = make_int2(wlo, whi);
    const int a = max(wlo, pl.row0), b = min(whi, pl.row1);
    if (b > a) pairs += 1.0f + (float)(b - a) * inv_wr;
    plo = __shfl_sync(0xFFFFFFFFu, lo, 31);
    phi = __shfl_sync(0xFFFFFFFFu, hi, 31);
    y0 = y1;
    y1 = y2;
  }
  return pairs;
}

// Add the parts p of the lanes with n > 0 elements to a work list.
__device__ __forceinline__ void list_add(const WorkList& l, unsigned long long* counter, unsigned long long n,
                                         unsigned p, Ctrl* ctrl) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xFFFFFFFFu, n > 0);
  if (m == 0u) return;
  unsigned long long incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += t;
  }
  unsigned long long base = 0;
  if (lane == 31) {
    base = atomicAdd(counter, ((unsigned long long)__popc(m) << WL_BITS) + incl);
    // no table has 2^37 vertices; more windows are refused before they could carry into the length
    if (incl >> WL_BITS || (wl_total(base) + incl) >> WL_BITS) set_error(ctrl, ERR_WINDOWS, p);
  }
  base = __shfl_sync(0xFFFFFFFFu, base, 31);
  if (n > 0) {
    const unsigned e = (unsigned)wl_length(base) + __popc(m & ((1u << lane) - 1u));
    if (e < l.cap) {
      l.part[e] = p;
      l.first[e] = wl_total(base) + incl - n;
    }
  }
}

// Whether a part of `band` can write inside the call's window.
__device__ __forceinline__ bool plan_window(const JobDims& jd, unsigned band) {
  return band >= jd.band_lo && band < jd.band_hi && jd.row_lo < jd.row_hi;
}

// The part's raster and window, shared by every kind of part.
__device__ __forceinline__ void plan_base(const JobDims& jd, unsigned kind, unsigned band, PartPlan& pl) {
  pl.row0 = pl.row1 = pl.col0 = pl.bw = pl.wr = 0;
  pl.band = band;
  pl.nrows = jd.nrows;
  pl.ncols = jd.ncols;
  pl.wpr = jd.ntx * WPT;
  // unsigned arithmetic wraps: row r of the window lands on wid0 + r * wpr
  pl.wid0 = jd.wid_base + (band - jd.band_lo) * (unsigned)(jd.row_hi - jd.row_lo) * pl.wpr -
            (unsigned)jd.row_lo * pl.wpr;
  pl.flags = kind == 1 ? jd.line_flag : (kind == 2 ? jd.poly_flag : 0u);
  pl.rlo = jd.row_lo;
  pl.rhi = jd.row_hi;
  pl.ncw = 0;
}

// Count the parts p of the lanes with n > 0 elements into their bins of an
// ordered list, and keep an entry of each.
__device__ __forceinline__ void order_add(const ListOrder& o, int list, unsigned long long n, int row,
                                          const JobDims& jd, unsigned p, Ctrl* ctrl) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xFFFFFFFFu, n > 0);
  if (m == 0u) return;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&ctrl->ordered, (unsigned long long)__popc(m));
  base = __shfl_sync(0xFFFFFFFFu, base, 0) + __popc(m & ((1u << lane) - 1u));
  if (n == 0) return;
  const unsigned rows = (unsigned)(jd.row_hi - jd.row_lo);
  const unsigned r = (unsigned)(min(max(row, jd.row_lo), jd.row_hi - 1) - jd.row_lo);
  const unsigned tag = (unsigned)list * ORDER_BINS + (unsigned)((unsigned long long)r * ORDER_BINS / rows);
  const unsigned long long old = atomicAdd(&o.bins[tag], (1ull << WL_BITS) + n);
  if (n >> WL_BITS || (wl_total(old) + n) >> WL_BITS) set_error(ctrl, ERR_WINDOWS, p);
  o.part[base] = p;
  o.tag[base] = tag;
  o.got[base] = old;
}

// Bases of the bins of every ordered list (a block per list), and the lists'
// counters.
__global__ void __launch_bounds__(ORDER_BINS) k_order_bases(ListOrder o, Ctrl* ctrl) {
  __shared__ unsigned long long s_sum[32];
  if (block_skips(ctrl->err != 0u)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = blockIdx.x;
  const unsigned long long v = o.bins[k * ORDER_BINS + threadIdx.x];
  unsigned long long incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) s_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long w = s_sum[lane];
    unsigned long long wi = w, elems = wl_total(w);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, wi, d);
      const unsigned long long u = __shfl_up_sync(0xFFFFFFFFu, elems, d);
      if (lane >= d) {
        wi += t;
        elems += u;
      }
    }
    s_sum[lane] = wi - w;
    if (lane == 31) {
      ctrl->list[k == OL_NARROW ? WL_NARROW : k == OL_WIDE ? WL_WIDE : WL_LINE] = wi;
      if (elems >> WL_BITS) set_error(ctrl, ERR_WINDOWS, 0);
    }
  }
  __syncthreads();
  o.bins[k * ORDER_BINS + threadIdx.x] = s_sum[warp] + incl - v;
}

// Write the parts of the ordered lists to their places.
__global__ void k_order_place(Lists ls, const Ctrl* ctrl) {
  if (ctrl->err) return;
  const unsigned long long n = ctrl->ordered;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    const unsigned tag = ls.order.tag[i], k = tag / ORDER_BINS;
    const unsigned long long at = ls.order.bins[tag] + ls.order.got[i];
    const WorkList& l = ls.l[k == OL_NARROW ? WL_NARROW : k == OL_WIDE ? WL_WIDE : WL_LINE];
    if (wl_length(at) < l.cap) {
      l.part[wl_length(at)] = ls.order.part[i];
      l.first[wl_length(at)] = wl_total(at);
    }
  }
}

// What the prep gathers for later kernels beside the plans.
struct PrepOut {
  const void* values;   // per-geometry burn values, or nullptr
  void* pvals;          // [P] the part's burn value (values[part_geom[p]])
  int vbytes;           // bytes of a value
  int point_plans;      // write the plans of point parts too (the sparse stream and batches read them)
  unsigned long long* last_kept;  // [P] cleared for line parts
};

__device__ __forceinline__ void copy_value(const PrepOut& o, unsigned long long p, unsigned gi) {
  switch (o.vbytes) {
    case 1: static_cast<unsigned char*>(o.pvals)[p] = static_cast<const unsigned char*>(o.values)[gi]; break;
    case 2: static_cast<unsigned short*>(o.pvals)[p] = static_cast<const unsigned short*>(o.values)[gi]; break;
    case 4: static_cast<unsigned*>(o.pvals)[p] = static_cast<const unsigned*>(o.values)[gi]; break;
    default:
      static_cast<unsigned long long*>(o.pvals)[p] = static_cast<const unsigned long long*>(o.values)[gi];
  }
}

// Of the rings first, first + step, ... below re: how many are not empty, and (ENDS)
// whether one does not end at the y it starts at.  Four rings' loads are in
// flight at a time: one linestring part of 300,000 lines, one ring at a time and
// with the ends looked at too, 2.46 ms a call, 1.42 so.
template <bool ENDS>
__device__ __forceinline__ void scan_rings(const Geo& geo, unsigned long long first, unsigned long long re,
                                           unsigned step, unsigned& nonempty, bool& open) {
  for (unsigned long long r = first; r < re; r += 4ull * step) {
    unsigned long long a[4], e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned long long rk = r + (unsigned)k * step;
      a[k] = rk < re ? geo.vertex_offsets[rk] : 0ull;
      e[k] = rk < re ? geo.vertex_offsets[rk + 1] : 0ull;
    }
    double y0[4], y1[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      nonempty += e[k] > a[k];
      y0[k] = ENDS && e[k] > a[k] ? geo.xy[a[k]].y : 0.0;
      y1[k] = ENDS && e[k] > a[k] ? geo.xy[e[k] - 1].y : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) open = open || f64_bits(y0[k]) != f64_bits(y1[k]);
  }
}

// A warp takes `group` neighbouring parts, a lane each for their offsets,
// plans and list entries; the vertices of a polygon part are read by the
// whole warp for its extent.  Calls of many parts take 32 at a time (5 M
// points, a warp each: 1.36 ms), calls of few one, so that their polygons
// spread over the chip.  Polygon parts of more than PREP_BIG_VERTS vertices
// go to k_part_prep_big.
__device__ __forceinline__ void prep_body(const Geo& geo, const Grid& g, const JobDims& one,
                                          const JobDims* __restrict__ jobs, unsigned n_jobs,
                                          const unsigned* __restrict__ part_geom, PartPlan* plan, const Lists& ls,
                                          const PrepOut& out, const Tune& tn, int group, Ctrl* ctrl) {
  const int lane = threadIdx.x & 31;
  const unsigned long long warp0 = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  unsigned long long edges = 0;
  for (unsigned long long b0 = warp0 * group; b0 < geo.n_parts; b0 += nwarps * group) {
    const unsigned long long p = b0 + lane;
    const bool on = lane < group && p < geo.n_parts;
    unsigned kind = 0, band = 0, gi = 0;
    unsigned long long rb = 0, re = 0, vs = 0, ve = 0;
    bool in = false;  // the part's band and rows meet the call's window
    JobDims jd = one;
    if (on) {
      kind = geo.part_kind[p];
      rb = geo.ring_offsets[p];
      re = geo.ring_offsets[p + 1];
      gi = part_geom[p];
      vs = geo.vertex_offsets[rb];
      ve = geo.vertex_offsets[re];
      if (geo.bands) band = geo.bands[gi];
      if (jobs) jd = jobs[job_of(jobs, n_jobs, gi)];
      in = plan_window(jd, band);
      if (out.values) copy_value(out, p, gi);
      if (kind == 1) out.last_kept[p] = 0;
    }
    const bool poly = in && kind == 2, big = poly && ls.big_parts && ve - vs > PREP_BIG_VERTS;
    if (big) ls.big_parts[atomicAdd(&ctrl->big_parts, 1ull)] = (unsigned)p;
    // segments = vertices - non-empty rings
    if (in && kind == 1 && re - rb == 1) edges += ve - vs - (ve > vs ? 1 : 0);
    Extent ex;
    bool closed = false;
    unsigned todo = __ballot_sync(0xFFFFFFFFu, (poly && !big) || (in && kind == 1 && re - rb > 1));
    while (todo) {
      const int j = __ffs(todo) - 1;
      todo &= todo - 1u;
      const unsigned long long jrb = __shfl_sync(0xFFFFFFFFu, rb, j), jre = __shfl_sync(0xFFFFFFFFu, re, j);
      const unsigned long long jvs = __shfl_sync(0xFFFFFFFFu, vs, j), jve = __shfl_sync(0xFFFFFFFFu, ve, j);
      const bool fold = __shfl_sync(0xFFFFFFFFu, (int)poly, j);
      unsigned nonempty = 0;
      bool open = false;  // some ring of the lane's does not end at the y it starts at
      if (fold) scan_rings<true>(geo, jrb + lane, jre, 32, nonempty, open);
      else scan_rings<false>(geo, jrb + lane, jre, 32, nonempty, open);
      if (todo) {  // the next part's vertices on their way into L2 (one line per lane and
        // instruction; 100,000 polygons of 264 vertices: 175 -> 158 us)
        const int jn = __ffs(todo) - 1;
        const unsigned long long nvs = __shfl_sync(0xFFFFFFFFu, vs, jn), nve = __shfl_sync(0xFFFFFFFFu, ve, jn);
        for (unsigned long long v = nvs + 8ull * lane; v < nve && v < nvs + PREP_BIG_VERTS; v += 256)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(geo.xy + v));
      }
      Extent t;
      if (fold) t.fold_range(geo.xy, jvs + lane, jve, 128);
      nonempty = __reduce_add_sync(0xFFFFFFFFu, nonempty);
      open = __any_sync(0xFFFFFFFFu, open);
      if (fold) t.warp_merge();
      if (lane == j) {
        edges += ve - vs - nonempty;
        ex = t;
        closed = !open;
      }
    }
    unsigned long long nwin = 0;
    bool narrow = false;
    int row = 0;
    if (on) {
      PartPlan pl;
      plan_base(jd, kind, band, pl);
      if (poly && !big) nwin = plan_polygon(g, jd, ex, tn, pl, narrow);
      if (poly && closed) pl.ncw |= RINGS_CLOSED;
      if (kind != 0 || out.point_plans) plan[p] = pl;
      row = pl.row0;
    }
    // all_touched also walks polygon rings
    const unsigned long long nline = in && (kind == 1 || (kind == 2 && g.touched)) ? ve - vs : 0;
    if (ls.order.bins) {
      if (nline > 0 && (kind == 1 || big)) row = row_ceil(to_py(g, geo.xy[vs].y), jd.nrows);
      order_add(ls.order, narrow ? OL_NARROW : OL_WIDE, nwin, row, jd, (unsigned)p, ctrl);
      order_add(ls.order, OL_LINE, nline, row, jd, (unsigned)p, ctrl);
    } else {
      list_add(ls.l[WL_NARROW], &ctrl->list[WL_NARROW], narrow ? nwin : 0, (unsigned)p, ctrl);
      list_add(ls.l[WL_WIDE], &ctrl->list[WL_WIDE], narrow ? 0 : nwin, (unsigned)p, ctrl);
      list_add(ls.l[WL_LINE], &ctrl->list[WL_LINE], nline, (unsigned)p, ctrl);
    }
    list_add(ls.l[WL_POINT], &ctrl->list[WL_POINT], in && kind == 0 ? ve - vs : 0, (unsigned)p, ctrl);
  }
  for (int o = 16; o > 0; o >>= 1) edges += __shfl_xor_sync(0xFFFFFFFFu, edges, o);
  if (lane == 0 && edges) atomicAdd(&ctrl->edges, edges);
}

__global__ void __launch_bounds__(256, 4) k_part_prep(Geo geo, Grid g, JobDims one, const JobDims* __restrict__ jobs,
                                                     unsigned n_jobs, const unsigned* __restrict__ part_geom,
                                                     PartPlan* plan, Lists ls, PrepOut out, Tune tn, int group,
                                                     Ctrl* ctrl) {
  if (ctrl->err) return;
  prep_body(geo, g, one, jobs, n_jobs, part_geom, plan, ls, out, tn, group, ctrl);
}

// One block per large polygon part: k_part_prep wrote the part's base plan,
// the block adds its windows.
__global__ void __launch_bounds__(256) k_part_prep_big(Geo geo, Grid g, JobDims one, const JobDims* __restrict__ jobs,
                                                       unsigned n_jobs, const unsigned* __restrict__ part_geom,
                                                       PartPlan* plan, Lists ls, Tune tn, Ctrl* ctrl) {
  constexpr int W = 8;
  __shared__ Extent s_ex[W];
  __shared__ unsigned s_rings[W];
  __shared__ bool s_open[W];
  __shared__ float s_pairs[W];
  __shared__ PartPlan s_pl;
  __shared__ unsigned long long s_nwin;
  if (block_skips(ctrl->err != 0u)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long n = ctrl->big_parts;
  for (unsigned long long i = blockIdx.x; i < n; i += gridDim.x) {
    const unsigned p = ls.big_parts[i];
    const unsigned long long rb = geo.ring_offsets[p], re = geo.ring_offsets[p + 1];
    const unsigned long long vs = geo.vertex_offsets[rb], ve = geo.vertex_offsets[re];
    unsigned nonempty = 0;
    bool open = false;
    scan_rings<true>(geo, rb + threadIdx.x, re, 32 * W, nonempty, open);
    nonempty = __reduce_add_sync(0xFFFFFFFFu, nonempty);
    open = __any_sync(0xFFFFFFFFu, open);
    Extent ex;
    ex.fold_range(geo.xy, vs + 128ull * warp + lane, ve, 128 * W);
    ex.warp_merge();
    if (lane == 0) {
      s_ex[warp] = ex;
      s_rings[warp] = nonempty;
      s_open[warp] = open;
    }
    __syncthreads();
    bool narrow = false;
    if (threadIdx.x == 0) {
      const unsigned gi = part_geom[p];
      const JobDims jd = jobs ? jobs[job_of(jobs, n_jobs, gi)] : one;
      for (int k = 1; k < W; ++k) {
        ex.merge(s_ex[k]);
        nonempty += s_rings[k];
        open = open || s_open[k];
      }
      atomicAdd(&ctrl->edges, ve - vs - nonempty);
      s_pl = plan[p];
      if (!open) s_pl.ncw |= RINGS_CLOSED;
      s_nwin = plan_polygon(g, jd, ex, tn, s_pl, narrow);
    }
    __syncthreads();
    // a part whose windows skip at least half of its chunks is walked by chunk,
    // and a wide one in any case: 10 boundaries of 150,000 vertices with two
    // windows each, most chunks in one of them, 3.0 ms a call as wide parts
    // (four blocks per SM cost k_poly_spans registers, which a few blocks miss),
    // 1.9 by chunk; 1,000 of 2,000, every chunk in both, 0.82 and 0.76
    const bool chunks = s_nwin > 1 && ls.chunk_rows && ve - vs <= 0xFFFFFFFFull - 64;
    const unsigned nv = (unsigned)(ve - vs), nc = (nv + 31) / 32;
    if (chunks) {
      const float pairs = chunk_ranges(geo, g, s_pl, vs, nv, (unsigned)((unsigned long long)nc * warp / W),
                                       (unsigned)((unsigned long long)nc * (warp + 1) / W),
                                       ls.chunk_rows + chunk_slot(p, vs));
      if (lane == 0) s_pairs[warp] = pairs;
    }
    __syncthreads();
    if (warp == 0) {
      float sum = 0.0f;
      for (int k = 0; chunks && k < W; ++k) sum += s_pairs[k];
      const bool nar = __shfl_sync(0xFFFFFFFFu, (int)narrow, 0) != 0;
      const bool by_chunk = chunks && (!nar || sum < 0.5f * (float)nc * (float)s_nwin);
      unsigned long long nwin = 0;
      if (lane == 0) {
        nwin = by_chunk ? set_windows(tn, false, s_pl) : s_nwin;
        plan[p] = s_pl;
      }
      const int which = by_chunk ? WL_CHUNK : (nar ? WL_NARROW : WL_WIDE);
      list_add(ls.l[which], &ctrl->list[which], nwin, p, ctrl);
    }
    __syncthreads();  // the shared values are reused
  }
}

// burners.rs:87-89: after the last kept segment of the part, its end pixel
// is written unless that segment's linestring is closed.  One slot
// reservation per 32 parts: a reservation each, all on one address, took the
// 200,000 lines of a mixed collection 187 us, so it takes 53.
__device__ __forceinline__ void endpix_body(const Geo& geo, const Grid& g, const PartPlan* __restrict__ plan,
                                            const WorkList& wl,
                                            const unsigned long long* __restrict__ last_kept, const RecBuf& sb,
                                            unsigned* bucket_count, Ctrl* ctrl) {
  const int lane = threadIdx.x & 31;
  const unsigned long long nlist = wl_length(ctrl->list[WL_LINE]);
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned npix = 0;
  for (unsigned long long q0 = blockIdx.x * (unsigned long long)blockDim.x + (threadIdx.x & ~31u); q0 < nlist;
       q0 += stride) {
    const unsigned p = q0 + lane < nlist ? wl.part[q0 + lane] : 0u;
    const unsigned long long kept = q0 + lane < nlist ? last_kept[p] : 0ull;
    bool emit = false;
    unsigned wid = 0, mask = 0, flags = 0;
    if (kept != 0) {
      const unsigned long long v = kept - 1;
      const unsigned long long rb = geo.ring_offsets[p], re = geo.ring_offsets[p + 1];
      const unsigned long long r = re - rb > 1 ? ring_of(geo, rb, re, v) : rb;
      bool closed;
      if (geo.ring_closed) {
        closed = geo.ring_closed[r] != 0;
      } else {
        const double2 first = geo.xy[geo.vertex_offsets[r]];
        const double2 last = geo.xy[geo.vertex_offsets[r + 1] - 1];
        closed = first.x == last.x && first.y == last.y;  // LineString::is_closed
      }
      if (!closed) {
        const double2 w1 = geo.xy[v + 1];
        const long long ix = as_isize(floor(to_px(g, w1.x))), iy = as_isize(floor(to_py(g, w1.y)));
        const PartPlan& pl = plan[p];
        if (ix >= 0 && ix < pl.ncols && iy >= pl.rlo && iy < pl.rhi) {
          emit = true;
          wid = pl.wid0 + (unsigned)iy * pl.wpr + ((unsigned)ix >> 5);
          mask = 1u << ((unsigned)ix & 31u);
          flags = p | pl.flags;
          ++npix;
        }
      }
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, emit);
    if (m == 0u) continue;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&ctrl->span_count, (unsigned long long)__popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (emit) {
      const unsigned long long slot = base + __popc(m & ((1u << lane) - 1u));
      if (slot < sb.cap) {
        sb.wid[slot] = wid;
        sb.part[slot] = flags;
        sb.mask[slot] = mask;
      }
      if (wid / WPT < sb.nbuckets) atomicAdd(&bucket_count[wid / WPT], 1u);
      else set_error(ctrl, ERR_RANGE, wid);  // never taken: the pixel is in its raster
    }
  }
  npix = __reduce_add_sync(0xFFFFFFFFu, npix);
  if (lane == 0 && npix) atomicAdd(&ctrl->pixel_writes, (unsigned long long)npix);
}

__global__ void k_line_endpix(Geo geo, Grid g, const PartPlan* __restrict__ plan, WorkList wl,
                              const unsigned long long* __restrict__ last_kept, RecBuf sb,
                              unsigned* bucket_count, Ctrl* ctrl) {
  if (ctrl->err) return;
  endpix_body(geo, g, plan, wl, last_kept, sb, bucket_count, ctrl);
}

// ------------------------------------------------------------- points ------
// extract_point (edges.rs:79-88) + burn_point (burners.rs:250-258).  A warp
// takes 32 neighbouring points of the list at a time, POINT_RANGE in a row,
// and stages their records as the line kernel does.  A call of one raster
// derives the point's place from the raster itself (`one`) instead of
// reading the part's plan, which is then not written either.
constexpr int POINT_RANGE = 128;

__device__ __forceinline__ void point_body(const Geo& geo, const Grid& g, const JobDims& one, int from_plan,
                                           const PartPlan* __restrict__ plan, const unsigned* __restrict__ part_geom,
                                           const WorkList& wl, const RecBuf& sb, unsigned* bucket_count, Ctrl* ctrl) {
  __shared__ unsigned s_stage[LINE_WARPS][3 * LINE_STAGE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  RecStage st;
  st.wid = s_stage[warp];
  st.part = st.wid + LINE_STAGE;
  st.mask = st.part + LINE_STAGE;
  st.n = 0;
  const unsigned nlist = (unsigned)wl_length(ctrl->list[WL_POINT]);
  const unsigned long long total = wl_total(ctrl->list[WL_POINT]);
  unsigned npix = 0;
  for (unsigned long long r0 = ((unsigned long long)blockIdx.x * LINE_WARPS + warp) * POINT_RANGE; r0 < total;
       r0 += (unsigned long long)gridDim.x * LINE_WARPS * POINT_RANGE) {
    unsigned e0 = list_slot(wl.first, nlist, r0);
    for (unsigned long long t0 = r0; t0 < r0 + POINT_RANGE && t0 < total; t0 += 32) {
      unsigned p;
      unsigned long long c;
      list_parts<32>(wl, nlist, t0, e0, p, c);
      bool emit = false;
      unsigned wid = 0, mask = 0;
      if (t0 + lane < total) {
        const double2 w = geo.xy[geo.vertex_offsets[geo.ring_offsets[p]] + (t0 + lane - c)];
        PartPlan pl;
        if (from_plan) pl = plan[p];
        else plan_base(one, 0, geo.bands ? geo.bands[part_geom[p]] : 0u, pl);
        const double x = to_px(g, w.x), y = to_py(g, w.y);
        // extract_point keeps 0 <= y < nrows; the window keeps rows [rlo, rhi) of those
        if (x >= 0.0 && x < (double)pl.ncols && y >= (double)pl.rlo && y < (double)pl.rhi) {
          const unsigned px = (unsigned)(int)x;
          emit = true;
          wid = pl.wid0 + (unsigned)(int)y * pl.wpr + (px >> 5);
          mask = 1u << (px & 31u);
          ++npix;
        }
      }
      line_push(st, emit, wid, p, mask, [&]() { line_flush(st, sb, bucket_count, ctrl); });
    }
  }
  line_flush(st, sb, bucket_count, ctrl);
  npix = __reduce_add_sync(0xFFFFFFFFu, npix);
  if (lane == 0 && npix) atomicAdd(&ctrl->pixel_writes, (unsigned long long)npix);
}

__global__ void __launch_bounds__(LINE_WARPS * 32) k_point_spans(Geo geo, Grid g, JobDims one, int from_plan,
                                                                 const PartPlan* __restrict__ plan,
                                                                 const unsigned* __restrict__ part_geom, WorkList wl,
                                                                 RecBuf sb, unsigned* bucket_count, Ctrl* ctrl) {
  if (ctrl->err) return;
  point_body(geo, g, one, from_plan, plan, part_geom, wl, sb, bucket_count, ctrl);
}

// ------------------------------------------------------------- scatter -----
// Move each coverage record into its bucket's range as {part | word-in-tile
// << REC_W_SHIFT | DEDUP_BIT, mask}.  Order inside a bucket is arbitrary
// here; the fill kernels restore part order (and look up each part's burn
// value).  Records of one bucket that sit in one warp (neighbouring words of
// a row) take their places with one atomic on the bucket's cursor, which
// starts at the bucket's offset: per record one scattered atomic and one
// scattered write, which is what bounds it (150 M records of lines: 59
// records per ns with an offset lookup and a count).
__device__ __forceinline__ void scatter_body(const RecBuf& sb, unsigned long long n, unsigned* cursor, uint2* sorted) {
  const int lane = threadIdx.x & 31;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i0 = blockIdx.x * (unsigned long long)blockDim.x + (threadIdx.x & ~31u); i0 < n;
       i0 += stride) {
    const unsigned long long i = i0 + lane;
    const bool valid = i < n;
    const unsigned wid = valid ? sb.wid[i] : 0xFFFFFFFFu;
    const unsigned b = valid ? wid / WPT : 0xFFFFFFFFu;
    const unsigned same = __match_any_sync(0xFFFFFFFFu, b);
    const int leader = __ffs(same) - 1;
    unsigned pos = 0;
    if (valid && lane == leader) pos = atomicAdd(&cursor[b], (unsigned)__popc(same));
    pos = __shfl_sync(0xFFFFFFFFu, pos, leader) + (unsigned)__popc(same & ((1u << lane) - 1u));  // arrival order
    if (valid) sorted[pos] = make_uint2(sb.part[i] | ((wid % WPT) << REC_W_SHIFT), sb.mask[i]);
  }
}

__global__ void k_scatter(RecBuf sb, unsigned* cursor, uint2* sorted, Ctrl* ctrl) {
  if (ctrl->err || ctrl->span_count > sb.cap) return;
  scatter_body(sb, ctrl->span_count, cursor, sorted);
}

}  // namespace rzd
