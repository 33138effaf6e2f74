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
// Reject tables that would make any later kernel read out of bounds.
__global__ void k_validate(Geo geo, Ctrl* ctrl) {
  const unsigned long long tid = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = tid; i <= geo.n_geoms; i += stride) {
    unsigned long long a = geo.part_offsets[i];
    if ((i == 0 && a != 0) || (i == geo.n_geoms && a != geo.n_parts) ||
        (i > 0 && a < geo.part_offsets[i - 1]) || a > geo.n_parts)
      set_error(ctrl, ERR_BAD_TABLE, i);
  }
  for (unsigned long long i = tid; i <= geo.n_parts; i += stride) {
    unsigned long long a = geo.ring_offsets[i];
    if ((i == 0 && a != 0) || (i == geo.n_parts && a != geo.n_rings) ||
        (i > 0 && a < geo.ring_offsets[i - 1]) || a > geo.n_rings)
      set_error(ctrl, ERR_BAD_TABLE, (1ull << 62) | i);
    if (i < geo.n_parts && geo.part_kind[i] > 2) set_error(ctrl, ERR_BAD_KIND, i);
  }
  for (unsigned long long i = tid; i <= geo.n_rings; i += stride) {
    unsigned long long a = geo.vertex_offsets[i];
    if ((i == 0 && a != 0) || (i == geo.n_rings && a != geo.n_vertices) ||
        (i > 0 && a < geo.vertex_offsets[i - 1]) || a > geo.n_vertices)
      set_error(ctrl, ERR_BAD_TABLE, (2ull << 62) | i);
  }
}

__global__ void k_check_bands(Geo geo, unsigned n_bands, Ctrl* ctrl) {
  if (ctrl->err) return;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < geo.n_geoms;
       i += stride)
    if (geo.bands[i] >= n_bands) set_error(ctrl, ERR_BAD_BAND, i);
}

// part -> owning geometry index
__global__ void k_part_geom(Geo geo, unsigned* part_geom, Ctrl* ctrl) {
  if (ctrl->err) return;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long gi = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; gi < geo.n_geoms;
       gi += stride) {
    for (unsigned long long p = geo.part_offsets[gi]; p < geo.part_offsets[gi + 1]; ++p)
      part_geom[p] = (unsigned)gi;
  }
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
  __device__ __forceinline__ void warp_merge() {
    for (int o = 16; o > 0; o >>= 1) {
      ylo = min(ylo, (long long)__shfl_xor_sync(0xFFFFFFFFu, (unsigned long long)ylo, o));
      yhi = max(yhi, (long long)__shfl_xor_sync(0xFFFFFFFFu, (unsigned long long)yhi, o));
      xlo = min(xlo, (long long)__shfl_xor_sync(0xFFFFFFFFu, (unsigned long long)xlo, o));
      xhi = max(xhi, (long long)__shfl_xor_sync(0xFFFFFFFFu, (unsigned long long)xhi, o));
    }
    nan_x = __any_sync(0xFFFFFFFFu, nan_x);
  }
};

// The window heights and number of windows of a planned polygon part: with the
// small bitmap of one warp (narrow) or the bitmap of a block.
__device__ __forceinline__ unsigned long long set_windows(const Tune& tn, bool narrow, PartPlan& pl,
                                                          unsigned long long* c) {
  const int rows = pl.row1 - pl.row0;
  if (pl.bw > BITMAP_WORDS) {  // wider than one bitmap: windows of columns too
    pl.wr = min(COLWIN_ROWS, tn.rows_per_window);
    pl.ncw = (unsigned)((pl.bw + COLWIN_WORDS - 1) / COLWIN_WORDS);
    return c[PC_WINDOWS] = (unsigned long long)((rows + pl.wr - 1) / pl.wr) * pl.ncw;
  }
  pl.wr = min((narrow ? SMALL_BITMAP_WORDS : BITMAP_WORDS) / pl.bw, tn.rows_per_window);
  return c[narrow ? PC_WIN_SMALL : PC_WINDOWS] = (unsigned long long)((rows + pl.wr - 1) / pl.wr);
}

// The row range and bitmap window geometry of a polygon part from its extent
// (the world->pixel map is monotone, so transforming the extremes gives the
// pixel extremes).  Returns its number of windows.
__device__ __forceinline__ unsigned long long plan_polygon(const Grid& g, const JobDims& jd, const Extent& ex,
                                                           const Tune& tn, PartPlan& pl, unsigned long long* c) {
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
  return set_windows(tn, bw <= tn.narrow_max_words, pl, c);
}

// ChunkList::rows of chunks [c0, c1) of a part with nv vertices from vs on, by
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
  const float inv = 1.0f / (float)g.yres, inv_wr = 1.0f / (float)pl.wr, hi_row = (float)pl.nrows;
  const bool usable = inv > 0.0f && inv < 1e30f;
  auto world = [&](unsigned c) { return xy[min(32u * c + (unsigned)lane, nv - 1u)].y; };
  auto rows = [&](double wy, int& lo, int& hi) {  // holds clamp(ceil(y - 0.5), 0, nrows); NaN: row 0
    const float f = (float)__dsub_rn(g.ymax, wy) * inv;
    const float m = 0.51f + fabsf(f) * 9.5367431640625e-07f;  // 2^-20
    lo = (int)fminf(fmaxf(floorf(f - m), 0.0f), hi_row);      // fmaxf(NaN, 0) = 0
    hi = (int)fminf(fmaxf(ceilf(f + m), 0.0f), hi_row);
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

// Put a planned part on the chunk list when its windows skip at least half of
// its chunks (one lane): its windows move to the list's kernel, which takes a
// block per window.
__device__ __forceinline__ void chunk_list_add(const Geo& geo, const Tune& tn, unsigned long long p, unsigned nv,
                                               unsigned long long nwin, float pairs, PartPlan& pl,
                                               unsigned long long* c, Ctrl* ctrl) {
  if (pairs >= 0.5f * (float)((nv + 31) / 32) * (float)nwin) return;
  c[PC_WINDOWS] = c[PC_WIN_SMALL] = 0;
  const unsigned long long n = set_windows(tn, false, pl, c);
  c[PC_WINDOWS] = c[PC_WIN_SMALL] = 0;
  const unsigned long long old = atomicAdd(&ctrl->chunked, (1ull << CHUNK_WIN_BITS) | n);
  geo.chunks.part[old >> CHUNK_WIN_BITS] = (unsigned)p;
  geo.chunks.win0[old >> CHUNK_WIN_BITS] = old & ((1ull << CHUNK_WIN_BITS) - 1ull);
}

// The part's raster and window, shared by every kind of part; false when its
// band or rows lie outside the call's window (it burns nothing then).
__device__ __forceinline__ bool plan_base(const JobDims& jd, unsigned kind, unsigned band, PartPlan& pl) {
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
  return band >= jd.band_lo && band < jd.band_hi && jd.row_lo < jd.row_hi;
}

// One warp per part.  Polygon parts get their plan from the extent of their
// vertices; line and point parts just report their vertex counts.  The
// kernel waits on dependent loads, so it is held to six blocks per SM (at
// most 42 registers) for more loads in flight.  Polygon parts of more than
// PREP_BIG_VERTS vertices go to k_part_prep_big when there is a list for them.
__global__ void __launch_bounds__(256, 6) k_part_prep(Geo geo, Grid g, JobDims one, const JobDims* __restrict__ jobs,
                                                     unsigned n_jobs, const unsigned* part_geom, PartPlan* plan,
                                                     unsigned long long* counts /*[P][PC_N]*/, Tune tn,
                                                     unsigned* big_list, Ctrl* ctrl) {
  if (ctrl->err) return;
  const int lane = threadIdx.x & 31;
  const unsigned long long warp0 = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  unsigned long long edges = 0;
  for (unsigned long long p = warp0; p < geo.n_parts; p += nwarps) {
    const unsigned kind = geo.part_kind[p];
    const unsigned long long rb = geo.ring_offsets[p], re = geo.ring_offsets[p + 1];
    const unsigned long long vs = geo.vertex_offsets[rb], ve = geo.vertex_offsets[re];
    const unsigned gi = part_geom[p];
    const unsigned band = geo.bands ? geo.bands[gi] : 0u;
    const JobDims jd = jobs ? jobs[job_of(jobs, n_jobs, gi)] : one;
    unsigned long long c[PC_N] = {0, 0, 0, 0, 0, 0};
    PartPlan pl;
    if (!plan_base(jd, kind, band, pl)) {
      if (lane == 0) {
        plan[p] = pl;
#pragma unroll
        for (int k = 0; k < PC_N; ++k) counts[p * PC_N + k] = 0;
      }
      continue;
    }
    if (kind != 0) {
      // segments = vertices - non-empty rings
      unsigned long long nonempty = 0;
      for (unsigned long long r = rb + lane; r < re; r += 32)
        nonempty += geo.vertex_offsets[r + 1] > geo.vertex_offsets[r];
      for (int o = 16; o > 0; o >>= 1) nonempty += __shfl_xor_sync(0xFFFFFFFFu, nonempty, o);
      edges += (lane == 0) ? (ve - vs) - nonempty : 0;
    }
    if ((kind == 1 || (kind == 2 && g.touched)) && ve > vs) {  // all_touched also walks polygon rings
      c[PC_LINE_V] = ve - vs;
      c[PC_LINE_P] = 1;  // the list holds no empty part: its vertex offsets are strictly increasing
    }
    if (kind == 1) {
    } else if (kind == 0) {
      c[PC_POINT_V] = ve - vs;
      c[PC_POINT_P] = 1;
    } else if (big_list && ve - vs > PREP_BIG_VERTS) {
      if (lane == 0) big_list[atomicAdd(&ctrl->big_parts, 1ull)] = (unsigned)p;
    } else {
      Extent ex;
      ex.fold_range(geo.xy, vs + lane, ve, 128);
      ex.warp_merge();
      plan_polygon(g, jd, ex, tn, pl, c);
    }
    if (lane == 0) {
      plan[p] = pl;
#pragma unroll
      for (int k = 0; k < PC_N; ++k) counts[p * PC_N + k] = c[k];
    }
  }
  for (int o = 16; o > 0; o >>= 1) edges += __shfl_xor_sync(0xFFFFFFFFu, edges, o);
  if (lane == 0 && edges) atomicAdd(&ctrl->edges, edges);
}

// One block per large polygon part: k_part_prep wrote the part's base plan
// and its line counts, the block adds the polygon's window plan.
__global__ void __launch_bounds__(256) k_part_prep_big(Geo geo, Grid g, JobDims one, const JobDims* __restrict__ jobs,
                                                       unsigned n_jobs, const unsigned* part_geom, PartPlan* plan,
                                                       unsigned long long* counts, Tune tn,
                                                       const unsigned* __restrict__ big_list, Ctrl* ctrl) {
  constexpr int W = 8;
  __shared__ Extent s_ex[W];
  __shared__ float s_pairs[W];
  __shared__ PartPlan s_pl;
  __shared__ unsigned long long s_nwin, s_c[PC_N];
  if (ctrl->err) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long n = ctrl->big_parts;
  for (unsigned long long i = blockIdx.x; i < n; i += gridDim.x) {
    const unsigned p = big_list[i];
    const unsigned long long vs = geo.vertex_offsets[geo.ring_offsets[p]];
    const unsigned long long ve = geo.vertex_offsets[geo.ring_offsets[p + 1]];
    Extent ex;
    ex.fold_range(geo.xy, vs + 128ull * warp + lane, ve, 128 * W);
    ex.warp_merge();
    if (lane == 0) s_ex[warp] = ex;
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned gi = part_geom[p];
      const JobDims jd = jobs ? jobs[job_of(jobs, n_jobs, gi)] : one;
      for (int k = 1; k < W; ++k) ex.merge(s_ex[k]);
      s_pl = plan[p];
      for (int k = 0; k < PC_N; ++k) s_c[k] = counts[(unsigned long long)p * PC_N + k];
      s_nwin = plan_polygon(g, jd, ex, tn, s_pl, s_c);
    }
    __syncthreads();
    const bool chunks = s_nwin > 1 && geo.chunks.rows && ve - vs <= 0xFFFFFFFFull - 64;
    const unsigned nv = (unsigned)(ve - vs), nc = (nv + 31) / 32;
    if (chunks) {
      const float pairs = chunk_ranges(geo, g, s_pl, vs, nv, (unsigned)((unsigned long long)nc * warp / W),
                                       (unsigned)((unsigned long long)nc * (warp + 1) / W),
                                       geo.chunks.rows + chunk_slot(p, vs));
      if (lane == 0) s_pairs[warp] = pairs;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (chunks) {
        float sum = 0.0f;
        for (int k = 0; k < W; ++k) sum += s_pairs[k];
        chunk_list_add(geo, tn, p, nv, s_nwin, sum, s_pl, s_c, ctrl);
      }
      plan[p] = s_pl;
      for (int k = 0; k < PC_N; ++k) counts[(unsigned long long)p * PC_N + k] = s_c[k];
    }
    __syncthreads();  // the shared values are reused
  }
}

// compact lists of line and point parts
__global__ void k_part_lists(Geo geo, const unsigned long long* off /*[P+1][PC_N]*/, unsigned* line_parts,
                             unsigned* point_parts, Ctrl* ctrl) {
  if (ctrl->err) return;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < geo.n_parts;
       p += stride) {
    // a part is listed when it was counted (parts outside the call's window are not)
    if (off[(p + 1) * PC_N + PC_LINE_P] > off[p * PC_N + PC_LINE_P])
      line_parts[off[p * PC_N + PC_LINE_P]] = (unsigned)p;
    else if (off[(p + 1) * PC_N + PC_POINT_P] > off[p * PC_N + PC_POINT_P])
      point_parts[off[p * PC_N + PC_POINT_P]] = (unsigned)p;
  }
}

// ------------------------------------------------------------- lines -------
// Locate, for compacted index t, the list slot q with cum(q) <= t < cum(q+1)
// where cum(q) = off[list[q]*PC_N + col].  Lane 0 binary-searches the warp's
// first index, the others walk forward from it.
__device__ __forceinline__ unsigned long long locate(const unsigned* list, unsigned long long nlist,
                                                     const unsigned long long* off, int col,
                                                     unsigned long long t, unsigned long long t_first) {
  unsigned long long q0 = 0;
  if ((threadIdx.x & 31) == 0) {
    unsigned long long lo = 0, hi = nlist;  // cum(lo) <= t_first < cum(hi) (cum(nlist) = total)
    while (hi - lo > 1) {
      const unsigned long long mid = (lo + hi) >> 1;
      if (off[(unsigned long long)list[mid] * PC_N + col] <= t_first) lo = mid; else hi = mid;
    }
    q0 = lo;
  }
  q0 = __shfl_sync(0xFFFFFFFFu, q0, 0);
  unsigned long long q = q0;
  while (q + 1 < nlist && off[(unsigned long long)list[q + 1] * PC_N + col] <= t) ++q;
  return q;
}

// burners.rs:87-89: after the last kept segment of the part, its end pixel
// is written unless that segment's linestring is closed.
__global__ void k_line_endpix(Geo geo, Grid g, const PartPlan* __restrict__ plan,
                              const unsigned long long* __restrict__ poff, const unsigned* __restrict__ line_parts,
                              const unsigned long long* __restrict__ last_kept, RecBuf sb,
                              unsigned* bucket_count, Ctrl* ctrl) {
  if (ctrl->err) return;
  const unsigned long long nlist = poff[geo.n_parts * PC_N + PC_LINE_P];
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long npix = 0;
  for (unsigned long long q = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; q < nlist; q += stride) {
    const unsigned p = line_parts[q];
    if (last_kept[p] == 0) continue;
    const unsigned long long v = last_kept[p] - 1;
    const unsigned long long rb = geo.ring_offsets[p], re = geo.ring_offsets[p + 1];
    const unsigned long long r = ring_of(geo, rb, re, v);
    if (geo.ring_closed) {
      if (geo.ring_closed[r]) continue;
    } else {
      const double2 first = geo.xy[geo.vertex_offsets[r]];
      const double2 last = geo.xy[geo.vertex_offsets[r + 1] - 1];
      if (first.x == last.x && first.y == last.y) continue;  // LineString::is_closed
    }
    const double2 w1 = geo.xy[v + 1];
    const long long ix = as_isize(floor(to_px(g, w1.x))), iy = as_isize(floor(to_py(g, w1.y)));
    const PartPlan pl = plan[p];
    if (ix >= 0 && ix < pl.ncols && iy >= pl.rlo && iy < pl.rhi) {
      ++npix;
      emit_run(sb, bucket_count, ctrl, pl, (int)iy, (int)ix, (int)ix + 1, p | pl.flags);
    }
  }
  if (npix) atomicAdd(&ctrl->pixel_writes, npix);
}

// ------------------------------------------------------------- points ------
// extract_point (edges.rs:79-88) + burn_point (burners.rs:250-258)
__global__ void k_point_spans(Geo geo, Grid g, const PartPlan* __restrict__ plan,
                              const unsigned long long* __restrict__ poff, const unsigned* __restrict__ point_parts,
                              RecBuf sb, unsigned* bucket_count, Ctrl* ctrl) {
  if (ctrl->err) return;
  const unsigned long long nlist = poff[geo.n_parts * PC_N + PC_POINT_P];
  const unsigned long long total = poff[geo.n_parts * PC_N + PC_POINT_V];
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long npix = 0;
  for (unsigned long long t0 = blockIdx.x * (unsigned long long)blockDim.x + (threadIdx.x & ~31u); t0 < total;
       t0 += stride) {
    const unsigned long long t = t0 + (threadIdx.x & 31);
    const unsigned long long q = locate(point_parts, nlist, poff, PC_POINT_V, t < total ? t : total - 1, t0);
    if (t >= total) continue;
    const unsigned p = point_parts[q];
    const unsigned long long v =
        geo.vertex_offsets[geo.ring_offsets[p]] + (t - poff[(unsigned long long)p * PC_N + PC_POINT_V]);
    const double2 w = geo.xy[v];
    const double x = to_px(g, w.x), y = to_py(g, w.y);
    const PartPlan pl = plan[p];
    // extract_point keeps 0 <= y < nrows; the window keeps rows [rlo, rhi) of those
    if (x >= 0.0 && x < (double)pl.ncols && y >= (double)pl.rlo && y < (double)pl.rhi) {
      ++npix;
      emit_run(sb, bucket_count, ctrl, pl, (int)y, (int)x, (int)x + 1, p);
    }
  }
  for (int o = 16; o > 0; o >>= 1) npix += __shfl_xor_sync(0xFFFFFFFFu, npix, o);
  if ((threadIdx.x & 31) == 0 && npix) atomicAdd(&ctrl->pixel_writes, npix);
}

// ------------------------------------------------------------- scatter -----
// Move each coverage record into its bucket's range as {part | word-in-tile
// << REC_W_SHIFT | DEDUP_BIT, mask}.  Order inside a bucket is arbitrary
// here; the fill kernels restore part order (and look up each part's burn
// value).  Records of one bucket that sit in one warp (neighbouring words of
// a row) take their slots with one atomic.
__global__ void k_scatter(RecBuf sb, const unsigned* __restrict__ offsets, unsigned* counts, uint2* sorted,
                          Ctrl* ctrl) {
  if (ctrl->err || ctrl->span_count > sb.cap) return;
  const unsigned long long n = ctrl->span_count;
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
    unsigned left = 0;  // records of the bucket not placed yet, before this group
    if (valid && lane == leader) left = atomicSub(&counts[b], (unsigned)__popc(same));
    left = __shfl_sync(0xFFFFFFFFu, left, leader);
    if (valid) {
      const unsigned rank = (unsigned)__popc(same & ((1u << lane) - 1u));
      const unsigned pos = offsets[b + 1] - left + rank;  // arrival order
      sorted[pos] = make_uint2(sb.part[i] | ((wid % WPT) << REC_W_SHIFT), sb.mask[i]);
    }
  }
}

// The burn value of every part (VB bytes): values[part_geom[p]].
template <int VB>
__global__ void k_part_values(const unsigned* __restrict__ part_geom, const void* __restrict__ values,
                              unsigned long long n_parts, void* pvals, Ctrl* ctrl) {
  using V = typename std::conditional<VB == 1, unsigned char,
            typename std::conditional<VB == 2, unsigned short,
            typename std::conditional<VB == 4, unsigned, unsigned long long>::type>::type>::type;
  if (ctrl->err) return;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < n_parts; p += stride)
    static_cast<V*>(pvals)[p] = static_cast<const V*>(values)[part_geom[p]];
}

}  // namespace rzd
