// rz_line.cuh -- line segments -> coverage records: Standard::burn_line
// (Bresenham, rust/src/rasterization/burners.rs:40-91) and
// AllTouched::burn_line (burners.rs:94-247), after extract_line's bbox filter
// (rust/src/geo/edges.rs:112-134).
//
// Work item: one segment (v, v + 1) of a linestring.  A warp sets up 32
// neighbouring vertices at a time and queues the segments that burn
// something in shared memory; its lanes walk the queued segments one pixel
// per step, and a lane whose segment has ended takes the next one from the
// queue.  Every lane collects the pixels of one 32-pixel word in a mask;
// finished words are staged, and a full stage goes into the warp's hash table
// of (part, word) masks with all lanes at work, where the words that
// neighbouring segments share are merged.  The table is written out in
// coalesced runs with one slot reservation per flush.
//
// What bounds it, on 200,000 random-walk lines (20 M segments): with one
// thread per segment and no staging, each divergent group of lanes took its
// record slots with its own atomic, and all of them go to one address: 12.1
// ms (4 M all_touched segments: 14.6 ms).  Staged but not merged: 2.1 ms for
// 150 M records, and the scatter behind it, which pays one atomic per
// record, 2.7 ms.  The queue keeps the lanes of a warp busy although their
// segments have different lengths.  What is left is the latency of the walk's
// chain of steps, so warps in flight count: queue and stage are cut to what
// lets 6 blocks live on an SM (all_touched, 96 registers: 5), and the ranges
// are taken from a counter, so that no warp ends late: 20 M segments 3.33 ->
// 2.30 ms, 4 M all_touched ones 1.49 -> 1.29 (larger queues, 5 and 4 blocks,
// a fixed stride; 7 blocks with a queue of 36: 2.43 ms).
#pragma once

#include "rz_device.cuh"

namespace rzd {

constexpr int LINE_WARPS = 4;
constexpr int LINE_QCAP = 48;    // queued segments per warp (31 are set up at a time)
constexpr int LINE_STAGE = 80;   // staged records per warp
constexpr int LINE_TABLE_LOG = 9;
constexpr int LINE_TABLE = 1 << LINE_TABLE_LOG;  // hash table entries per warp
constexpr int LINE_TABLE_FULL = LINE_TABLE / 2;  // entries that make a warp flush its table
// Consecutive line vertices a warp takes at a time, at most (a multiple of 31;
// 62: 3% slower on 20 M segments, 248: 2% slower on road networks).  Calls with
// fewer vertices than warps for such ranges take as few as 31, one segment a
// lane: 400 segments of up to 3,000 pixels are walked side by side then, not
// in rounds by seven warps.
constexpr int LINE_RANGE = 124;
// Calls of fewer vertices than this take two pixels per lane between two looks
// at the warp: their warps are too few to hide a step's latency (3,000 lines of
// 6,000 pixels along the rows 1.33 -> 1.15 ms a call, 60,000 2.95 -> 2.64, 2,000
// of 10,000 pixels in any direction 8.9 -> 8.4; short segments the same).  With
// 20 M segments that is no faster, and small calls as one launch lose 2%.
constexpr unsigned long long LINE_FEW = 1ull << 17;
constexpr int LINE_REFILL = 8;   // idle lanes that make a warp refill

// 16-byte fields of a queued segment.  Bresenham: end points, part, window.
// all_touched: the walk's four numbers, part, window and two counters, vertex
// and mode.
template <bool TOUCHED>
constexpr int line_fields() { return TOUCHED ? 5 : 3; }
template <bool TOUCHED>
constexpr int line_warp_bytes() { return line_fields<TOUCHED>() * 16 * LINE_QCAP + 12 * LINE_TABLE + 12 * LINE_STAGE; }

// A warp's staged records.
struct RecStage {
  unsigned *wid, *part, *mask;
  int n;
};

// Write a warp's staged records as they are (points; lines merge theirs first):
// one slot reservation, coalesced stores, one bucket count per record.
__device__ __forceinline__ void line_flush(RecStage& st, const RecBuf& rb, unsigned* bucket_count, Ctrl* ctrl) {
  const int lane = threadIdx.x & 31;
  if (st.n == 0) return;
  __syncwarp();
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&ctrl->span_count, (unsigned long long)st.n);
  base = __shfl_sync(0xFFFFFFFFu, base, 0);
  for (int j = lane; j < st.n; j += 32) {
    const unsigned wid = st.wid[j];
    const unsigned long long slot = base + (unsigned)j;
    if (slot < rb.cap) {
      rb.wid[slot] = wid;
      rb.part[slot] = st.part[j];
      rb.mask[slot] = st.mask[j];
    }
    if (wid / WPT < rb.nbuckets) atomicAdd(&bucket_count[wid / WPT], 1u);
    else set_error(ctrl, ERR_RANGE, wid);  // never taken: pixels are clipped to their raster
  }
  st.n = 0;
  __syncwarp();
}

// Add the record (wid, part, mask) of every lane with `emit` to the stage;
// `full` empties it.
template <typename Full>
__device__ __forceinline__ void line_push(RecStage& st, bool emit, unsigned wid, unsigned part, unsigned mask,
                                          Full&& full) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xFFFFFFFFu, emit);
  if (m == 0u) return;
  if (emit) {
    const int k = st.n + __popc(m & ((1u << lane) - 1u));
    st.wid[k] = wid;
    st.part[k] = part;
    st.mask[k] = mask;
  }
  st.n += __popc(m);
  if (st.n > LINE_STAGE - 32) full();
}

// A warp's table of coverage masks keyed by (part, word).
struct RecTable {
  unsigned long long* key;  // part | flags above the word id; LINE_EMPTY: free
  unsigned* mask;
  int n;  // entries in use
};
constexpr unsigned long long LINE_EMPTY = ~0ull;  // no part has all flag and part bits set

__device__ __forceinline__ void table_clear(RecTable& t) {
  for (int i = threadIdx.x & 31; i < LINE_TABLE; i += 32) {
    t.key[i] = LINE_EMPTY;
    t.mask[i] = 0u;
  }
  t.n = 0;
  __syncwarp();
}

// Merge a word into the table (one lane; the table has free entries).
// Returns the pixels it already held (0 without `repeats`); `fresh` says that
// it took an entry.
__device__ __forceinline__ unsigned table_add(const RecTable& t, unsigned wid, unsigned part, unsigned mask,
                                              int repeats, bool& fresh) {
  unsigned h = ((wid ^ (part << 10)) * 0x9E3779B1u) >> (32 - LINE_TABLE_LOG);
  const unsigned long long k = ((unsigned long long)part << 32) | wid;
  while (true) {
    const unsigned long long old = atomicCAS(&t.key[h], LINE_EMPTY, k);
    fresh = old == LINE_EMPTY;
    if (fresh || old == k) break;
    h = (h + 1) & (LINE_TABLE - 1);
  }
  if (repeats) return atomicOr(&t.mask[h], mask) & mask;
  atomicOr(&t.mask[h], mask);
  return 0u;
}

// Write the table's records and clear it.
__device__ __forceinline__ void table_flush(RecTable& t, const RecBuf& rb, unsigned* bucket_count, Ctrl* ctrl) {
  const int lane = threadIdx.x & 31;
  if (t.n == 0) return;
  __syncwarp();
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&ctrl->span_count, (unsigned long long)t.n);
  base = __shfl_sync(0xFFFFFFFFu, base, 0);
  for (int i = lane; i < LINE_TABLE; i += 32) {
    const unsigned long long k = t.key[i];
    const unsigned mask = t.mask[i];
    const bool used = k != LINE_EMPTY;
    const unsigned m = __ballot_sync(0xFFFFFFFFu, used);
    if (m == 0u) continue;
    if (used) {
      t.key[i] = LINE_EMPTY;
      t.mask[i] = 0u;
      const unsigned wid = (unsigned)k;
      const unsigned long long slot = base + __popc(m & ((1u << lane) - 1u));
      if (slot < rb.cap) {
        rb.wid[slot] = wid;
        rb.part[slot] = (unsigned)(k >> 32);
        rb.mask[slot] = mask;
      }
      if (wid / WPT < rb.nbuckets) atomicAdd(&bucket_count[wid / WPT], 1u);
      else set_error(ctrl, ERR_RANGE, wid);  // never taken: pixels are clipped to their raster
    }
    base += __popc(m);
  }
  t.n = 0;
  __syncwarp();
}

// The parts of elements t0 + lane of a list, given the entry e0 whose part
// contains t0: lane j looks up entry e0 + j (every entry has at least one
// element, so the entries start at increasing elements), and every lane
// counts the starts at or before its element.  On return p is the part and c
// its first element; e0 becomes the entry whose part contains t0 + NEXT, the
// first element of the next group.
template <int NEXT>
__device__ __forceinline__ void list_parts(const WorkList& l, unsigned len, unsigned long long t0, unsigned& e0,
                                           unsigned& p, unsigned long long& c) {
  const int lane = threadIdx.x & 31;
  unsigned pj = 0;
  unsigned long long cj = ~0ull;
  if (e0 + lane < len) {
    pj = l.part[e0 + lane];
    cj = l.first[e0 + lane];
  }
  const bool in = cj >= t0 && cj - t0 < 32;
  const unsigned starts = __reduce_or_sync(0xFFFFFFFFu, in ? 1u << (unsigned)(cj - t0) : 0u);
  const int before = __popc(__ballot_sync(0xFFFFFFFFu, cj < t0));
  const int s = before + __popc(starts & ((2u << lane) - 1u)) - 1;
  p = __shfl_sync(0xFFFFFFFFu, pj, s);
  c = __shfl_sync(0xFFFFFFFFu, cj, s);
  e0 += (unsigned)(before + __popc(starts) - 1);
  if (NEXT > 31 && e0 + 1 < len && l.first[e0 + 1] <= t0 + NEXT) ++e0;
}

// ring of vertex v among the rings [rb, re)
__device__ __forceinline__ unsigned long long ring_of(const Geo& geo, unsigned long long rb,
                                                      unsigned long long re, unsigned long long v) {
  unsigned long long lo = rb, hi = re;  // vo[lo] <= v < vo[hi]
  while (hi - lo > 1) {
    const unsigned long long mid = (lo + hi) >> 1;
    if (geo.vertex_offsets[mid] <= v) lo = mid; else hi = mid;
  }
  return lo;
}

// One lane's walk of a segment.
template <bool TOUCHED>
struct LineWalk;

// Standard::burn_line (burners.rs:40-91).  Pixel coordinates are kept modulo
// 2^32: a kept segment overlaps the raster (below 2^31 rows and columns) and
// takes at most 2^26 steps, so the wrapped values are distinct and unsigned
// comparisons with the raster's size are exact.
template <>
struct LineWalk<false> {
  unsigned x, y, x1, y1;
  int dx, dy, sx, sy, err;

  // The segment's end points in the queue; false when it burns nothing.
  static __device__ __forceinline__ bool setup(long long ix0, long long iy0, long long ix1, long long iy1,
                                               unsigned long long v, uint4* f, Ctrl* ctrl) {
    const long long ex = ix1 - ix0, ey = iy1 - iy0;
    if (ex > LINE_MAX_STEPS || ex < -LINE_MAX_STEPS || ey > LINE_MAX_STEPS || ey < -LINE_MAX_STEPS) {
      set_error(ctrl, ERR_LINE_LONG, v);
      return false;
    }
    f[0] = make_uint4((unsigned)ix0, (unsigned)iy0, (unsigned)ix1, (unsigned)iy1);
    return (ex | ey) != 0;
  }
  __device__ __forceinline__ void load(const uint4* q, int k) {
    const uint4 a = q[k];
    x = a.x;
    y = a.y;
    x1 = a.z;
    y1 = a.w;
    const int ddx = (int)(x1 - x), ddy = (int)(y1 - y);
    dx = ddx < 0 ? -ddx : ddx;
    dy = ddy < 0 ? ddy : -ddy;
    sx = ddx > 0 ? 1 : -1;
    sy = ddy > 0 ? 1 : -1;
    err = dx + dy;
  }
  // The current pixel, then one step; returns whether the walk goes on.
  __device__ __forceinline__ bool step(unsigned& px, unsigned& py, bool, bool&, const Geo&, const Grid&,
                                       const PartPlan*, unsigned, Ctrl*) {
    px = x;
    py = y;
    const int e2 = 2 * err;
    if (e2 >= dy) {
      err += dy;
      x += (unsigned)sx;
    }
    if (e2 <= dx) {
      err += dx;
      y += (unsigned)sy;
    }
    return x != x1 || y != y1;
  }
};

// AllTouched::burn_line (burners.rs:94-247, adapted there from GDAL's
// llrasterize.cpp): every pixel the segment touches, left to right.  Sloped
// segments are walked in fixed point (touch_dda, rz_bits.h); those it does not
// take, and from the step on that it does not decide, in FP64 with the
// reference's operations, without FMA.  An FP64 step costs some 18
// instructions of a pipe that retires two lanes per clock and SM, which is
// what the walk was bound by (72% busy): 83 M pixels of road networks took
// 3.3 ms, and took 1.5 ms so.
struct TouchLine {
  double x, y, x_end, slope, inv_slope;
};

template <>
struct LineWalk<true> {
  enum : unsigned { SLOPED = 0, VERTICAL = 1, HORIZONTAL = 2, FIXED = 3, UP = 4, ON_EDGE = 8 };
  // FIXED: g, a, b, a_last.  SLOPED: x, y, x_end, slope.
  unsigned long long r0, r1, r2, r3;
  // FIXED: column, first column not entered, row; margin and direction in
  // `mode`.  SLOPED: steps to go at most (two words), steps not to write.
  // VERTICAL / HORIZONTAL: next and last pixel, the other coordinate.
  int a, b, c;
  unsigned mode;  // | UP | ON_EDGE | margin << 4
  unsigned long long v;

  static __device__ __forceinline__ unsigned long long bits(double d) {
    return (unsigned long long)__double_as_longlong(d);
  }
  static __device__ __forceinline__ uint4 pack(unsigned long long u, unsigned long long w) {
    return make_uint4((unsigned)u, (unsigned)(u >> 32), (unsigned)w, (unsigned)(w >> 32));
  }
  static __device__ __forceinline__ double f64(unsigned long long u) { return __longlong_as_double((long long)u); }
  static __device__ __forceinline__ void put(uint4* f, uint4 f0, uint4 f1, int a, int b, int c, unsigned mode,
                                             unsigned long long v) {
    f[0] = f0;
    f[1] = f1;
    f[3].z = (unsigned)a;
    f[3].w = (unsigned)b;
    f[4] = make_uint4((unsigned)v, (unsigned)(v >> 32), (unsigned)c, mode);
  }
  // Every step crosses a pixel boundary in x or y (or nudges y by TOLERANCE
  // across one) and the clipped walk stays within the raster, so it needs
  // fewer steps than this.
  static __device__ __forceinline__ long long step_limit(const PartPlan& pl) {
    return 4 * ((long long)pl.ncols + pl.nrows + 4) + 1024;
  }

  // The walk of a sloped segment, left to right, clipped to the raster; false
  // when it burns nothing.
  static __device__ __forceinline__ bool clip(double df_x, double df_y, double df_x_end, double df_y_end,
                                              const PartPlan& pl, TouchLine& t) {
    const double nrows_f = (double)pl.nrows, ncols_f = (double)pl.ncols;
    const double slope = __ddiv_rn(__dsub_rn(df_y_end, df_y), __dsub_rn(df_x_end, df_x));
    const double inv_slope = __ddiv_rn(1.0, slope);
    if (df_x < 0.0) { df_y = __dadd_rn(df_y, __dmul_rn(__dsub_rn(0.0, df_x), slope)); df_x = 0.0; }
    if (df_x_end > ncols_f) {
      df_y_end = __dadd_rn(df_y_end, __dmul_rn(__dsub_rn(ncols_f, df_x_end), slope));
      df_x_end = ncols_f;
    }
    if (df_y < 0.0) { df_x = __dadd_rn(df_x, __dmul_rn(__dsub_rn(0.0, df_y), inv_slope)); df_y = 0.0; }
    else if (df_y > nrows_f) { df_x = __dadd_rn(df_x, __dmul_rn(__dsub_rn(nrows_f, df_y), inv_slope)); df_y = nrows_f; }
    if (df_y_end < 0.0) df_x_end = __dadd_rn(df_x_end, __dmul_rn(__dsub_rn(0.0, df_y_end), inv_slope));
    else if (df_y_end > nrows_f) df_x_end = __dadd_rn(df_x_end, __dmul_rn(__dsub_rn(nrows_f, df_y_end), inv_slope));
    // clamp to the raster (f64::clamp)
    t.x = df_x < 0.0 ? 0.0 : (df_x > ncols_f ? ncols_f : df_x);
    t.x_end = df_x_end < 0.0 ? 0.0 : (df_x_end > ncols_f ? ncols_f : df_x_end);
    t.y = df_y;
    t.slope = slope;
    t.inv_slope = inv_slope;
    return t.x >= 0.0 && t.x < t.x_end;
  }

  static __device__ __forceinline__ bool setup(double df_x, double df_y, double df_x_end, double df_y_end,
                                               unsigned long long v, const PartPlan& pl, uint4* f, Ctrl* ctrl) {
    const double EPSILON_INTERSECT = 1e-4;
    const long long nrows = pl.nrows, ncols = pl.ncols;
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    if (df_x > df_x_end) {  // proceed left to right
      double t = df_x; df_x = df_x_end; df_x_end = t;
      t = df_y; df_y = df_y_end; df_y_end = t;
    }
    if (fabs(__dsub_rn(df_x, df_x_end)) < 0.01) {  // vertical
      if (df_y_end < df_y) { const double t = df_y; df_y = df_y_end; df_y_end = t; }
      const long long ix = as_isize(floor(df_x_end));
      long long iy = as_isize(floor(df_y));
      long long iy_end = as_isize(floor(__dsub_rn(df_y_end, EPSILON_INTERSECT)));
      if (ix < 0 || ix >= ncols) return false;
      iy = iy > 0 ? iy : 0;
      iy_end = iy_end < nrows - 1 ? iy_end : nrows - 1;
      if (iy > iy_end) return false;
      if (iy_end - iy > LINE_MAX_STEPS) {
        set_error(ctrl, ERR_LINE_LONG, v);
        return false;
      }
      put(f, none, none, (int)iy, (int)iy_end, (int)ix, VERTICAL, v);
      return true;
    }
    if (fabs(__dsub_rn(df_y, df_y_end)) < 0.01) {  // horizontal
      if (df_x_end < df_x) { const double t = df_x; df_x = df_x_end; df_x_end = t; }
      long long ix = as_isize(floor(df_x));
      const long long iy = as_isize(floor(df_y));
      long long ix_end = as_isize(floor(__dsub_rn(df_x_end, EPSILON_INTERSECT)));
      if (iy < 0 || iy >= nrows) return false;
      ix = ix > 0 ? ix : 0;
      ix_end = ix_end < ncols - 1 ? ix_end : ncols - 1;
      if (ix > ix_end) return false;
      if (ix_end - ix > LINE_MAX_STEPS) {
        set_error(ctrl, ERR_LINE_LONG, v);
        return false;
      }
      put(f, none, none, (int)ix, (int)ix_end, (int)iy, HORIZONTAL, v);
      return true;
    }
    TouchLine t;
    if (!clip(df_x, df_y, df_x_end, df_y_end, pl, t)) return false;
    rzb::TouchDda w;
    if (rzb::touch_dda(t.x, t.y, t.x_end, t.slope, t.inv_slope, pl.ncols, pl.nrows, w)) {
      put(f, pack((unsigned long long)w.g, (unsigned long long)w.a),
          pack((unsigned long long)w.b, (unsigned long long)w.a_last), w.ix, w.end, w.iy,
          FIXED | (w.up ? UP : 0u) | (w.margin << 4), v);
    } else {
      const long long limit = step_limit(pl);
      put(f, pack(bits(t.x), bits(t.y)), pack(bits(t.x_end), bits(t.slope)), (int)(unsigned)limit,
          (int)(limit >> 32), 0, SLOPED, v);
    }
    return true;
  }
  __device__ __forceinline__ void load(const uint4* q, int k) {
    const uint4 f0 = q[k], f1 = q[LINE_QCAP + k], f3 = q[3 * LINE_QCAP + k], f4 = q[4 * LINE_QCAP + k];
    r0 = ((unsigned long long)f0.y << 32) | f0.x;
    r1 = ((unsigned long long)f0.w << 32) | f0.z;
    r2 = ((unsigned long long)f1.y << 32) | f1.x;
    r3 = ((unsigned long long)f1.w << 32) | f1.z;
    a = (int)f3.z;
    b = (int)f3.w;
    v = ((unsigned long long)f4.y << 32) | f4.x;
    c = (int)f4.z;
    mode = f4.w;
  }
  // From FIXED at (a, c), whose pixel has been written, to the FP64 walk: it
  // starts again and does not write the pixels that have been.
  __device__ __noinline__ static TouchLine restart_line(const Geo& geo, const Grid& g, const PartPlan& pl,
                                                        unsigned long long v) {
    const double2 w0 = geo.xy[v], w1 = geo.xy[v + 1];
    double x0 = to_px(g, w0.x), y0 = to_py(g, w0.y), x1 = to_px(g, w1.x), y1 = to_py(g, w1.y);
    if (x0 > x1) {
      double t = x0; x0 = x1; x1 = t;
      t = y0; y0 = y1; y1 = t;
    }
    TouchLine t;
    clip(x0, y0, x1, y1, pl, t);
    return t;
  }
  __device__ __forceinline__ void restart(const Geo& geo, const Grid& g, const PartPlan& pl) {
    const TouchLine t = restart_line(geo, g, pl, v);
    const int cols = a - rzb::floor_clamp(t.x, 0x7FFFFFFF), rows = (int)rzb::floor_i64(t.y) - c;
    c = 1 + cols + ((mode & UP) ? 2 * rows : -rows);
    r0 = bits(t.x);
    r1 = bits(t.y);
    r2 = bits(t.x_end);
    r3 = bits(t.slope);
    const long long limit = step_limit(pl);
    a = (int)(unsigned)limit;
    b = (int)(limit >> 32);
    mode = SLOPED;
  }
  // The current pixel (outside the raster: not written by the caller), then
  // one step; returns whether the walk goes on.  At an edge crossed upwards
  // the FP64 walk stops on the edge first and so writes the pixel twice:
  // reported by `twice` where the part needs a pixel once, else a step of its
  // own.
  __device__ __forceinline__ bool step(unsigned& px, unsigned& py, bool once, bool& twice, const Geo& geo,
                                       const Grid& g, const PartPlan* plan, unsigned part, Ctrl* ctrl) {
    const unsigned kind = mode & 3u;
    if (kind == FIXED) {
      px = (unsigned)a;
      py = (unsigned)c;
      if (mode & ON_EDGE) {
        mode &= ~ON_EDGE;
        --c;
        return true;
      }
      int64_t gg = (int64_t)r0;
      bool row;
      const bool up = (mode & UP) != 0u;
      const int r = rzb::touch_step(gg, (int64_t)r1, (int64_t)r2, (int64_t)r3, a, b, c, mode >> 4, up, row);
      r0 = (unsigned long long)gg;
      if (r == rzb::TOUCH_UNSURE) {
        restart(geo, g, plan[part]);
        return true;
      }
      if (row && up) {
        twice = once;
        if (!once) {
          mode |= ON_EDGE;
          ++c;
        }
      }
      return r == rzb::TOUCH_NEXT;
    }
    if (kind != SLOPED) {
      px = (unsigned)(kind == VERTICAL ? c : a);
      py = (unsigned)(kind == VERTICAL ? a : c);
      return a++ < b;
    }
    const double TOLERANCE = 1e-9;
    const long long budget = (long long)(((unsigned long long)(unsigned)b << 32) | (unsigned)a) - 1;
    a = (int)(unsigned)budget;
    b = (int)(budget >> 32);
    if (budget < 0) {  // more steps than a segment of its extent can need (pathological input)
      set_error(ctrl, ERR_LINE_LONG, v);
      px = py = 0xFFFFFFFFu;
      return false;
    }
    double df_x = f64(r0), df_y = f64(r1);
    const double slope = f64(r3);
    // floors, conversions and comparisons on the integer pipe
    const int ix = rzb::floor_clamp(df_x, 0x7FFFFFFF);  // 0 <= df_x < df_x_end
    const long long iy = rzb::floor_i64(df_y);
    px = (unsigned)ix;
    py = iy >= 0 && iy < 0x7FFFFFFF ? (unsigned)iy : 0xFFFFFFFFu;
    if (c > 0) {
      --c;
      px = py = 0xFFFFFFFFu;
    }
    double sx = __dsub_rn(rzb::int_f64(rzb::floor_clamp(__dadd_rn(df_x, 1.0), 0x7FFFFFFF)), df_x);
    double sy = __dmul_rn(sx, slope);
    const double ny = __dadd_rn(df_y, sy);
    if (rzb::floor_i64(ny) == iy) {
      df_x = __dadd_rn(df_x, sx);
      df_y = ny;
    } else {
      const bool up = f64_bits(slope) >> 63;  // slope < 0: it is neither 0 nor NaN here
      const long long edge = up ? iy : iy + 1;
      sy = __dsub_rn(edge > -(1ll << 53) && edge < (1ll << 53) ? rzb::int_f64(edge) : (double)edge, df_y);
      const double tol = up ? -TOLERANCE : TOLERANCE;
      if (up ? rzb::gt_f64(f64_bits(sy), f64_bits(tol)) : rzb::gt_f64(f64_bits(tol), f64_bits(sy))) sy = tol;
      sx = __ddiv_rn(sy, slope);
      df_x = __dadd_rn(df_x, sx);
      df_y = __dadd_rn(df_y, sy);
    }
    r0 = bits(df_x);
    r1 = bits(df_y);
    const unsigned long long xb = f64_bits(df_x);
    return (!(xb >> 63) || !(xb << 1)) && rzb::gt_f64(r2, xb);
  }
};

// The end pixel of a part's last kept Bresenham segment is written by
// k_line_endpix.
// `repeats`: a pixel that a part writes several times must be in as many
// records (sum, count and the sparse stream, unless the part deduplicates);
// for the other functions a part's repeated writes change nothing.
// STEPS: pixels per lane between two looks at the warp.
template <bool TOUCHED, int STEPS>
__device__ __forceinline__ void line_body(const Geo& geo, const Grid& g, const PartPlan* __restrict__ plan,
                                          const WorkList& wl, unsigned long long* last_kept, int repeats,
                                          const RecBuf& sb, unsigned* bucket_count, Ctrl* ctrl, unsigned char* smem) {
  constexpr int NF = line_fields<TOUCHED>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* q = reinterpret_cast<uint4*>(smem + warp * line_warp_bytes<TOUCHED>());
  RecTable tab;
  tab.key = reinterpret_cast<unsigned long long*>(q + NF * LINE_QCAP);
  tab.mask = reinterpret_cast<unsigned*>(tab.key + LINE_TABLE);
  RecStage st;
  st.wid = tab.mask + LINE_TABLE;
  st.part = st.wid + LINE_STAGE;
  st.mask = st.part + LINE_STAGE;
  st.n = 0;
  const unsigned nlist = (unsigned)wl_length(ctrl->list[WL_LINE]);
  const unsigned long long total = wl_total(ctrl->list[WL_LINE]);
  if (total == 0) return;
  const unsigned range =
      31u * (unsigned)min((unsigned long long)(LINE_RANGE / 31), max(1ull, total / (31ull * LINE_WARPS * gridDim.x)));
  auto next_range = [&]() {
    unsigned long long r = 0;
    if (lane == 0) r = atomicAdd(&ctrl->line_work, (unsigned long long)range);
    return __shfl_sync(0xFFFFFFFFu, r, 0);
  };
  unsigned long long rt = next_range();  // the warp's range
  unsigned long long t0 = rt;            // next vertices to set up, and their list entry
  if (rt >= total) return;
  table_clear(tab);
  // merge the staged words into the table
  auto merge = [&]() {
    __syncwarp();
    for (int j0 = 0; j0 < st.n; j0 += 32) {
      bool todo = j0 + lane < st.n;
      const unsigned wid = todo ? st.wid[j0 + lane] : 0u, part = todo ? st.part[j0 + lane] : 0u;
      unsigned mask = todo ? st.mask[j0 + lane] : 0u;
      while (true) {
        if (tab.n > LINE_TABLE_FULL) table_flush(tab, sb, bucket_count, ctrl);
        bool fresh = false;
        unsigned again = 0u;
        if (todo) again = table_add(tab, wid, part, mask, repeats, fresh);
        tab.n += __popc(__ballot_sync(0xFFFFFFFFu, fresh));
        // pixels written again go into the next table, as records of their own
        todo = again != 0u && !(part & DEDUP_BIT);
        mask = again;
        if (!__any_sync(0xFFFFFFFFu, todo)) break;
        table_flush(tab, sb, bucket_count, ctrl);
      }
    }
    st.n = 0;
    __syncwarp();
  };
  unsigned e0 = 0;
  bool located = false;
  int qn = 0;
  unsigned long long npix = 0;
  LineWalk<TOUCHED> walk;
  bool active = false;
  unsigned flags = 0, wid0 = 0, wpr = 0, ncols = 0, rlo = 0, nr = 0;  // the walked segment's part
  unsigned cwid = 0, cflags = 0, cmask = 0;                           // the word being collected
  while (true) {
    const unsigned idle = __ballot_sync(0xFFFFFFFFu, !active);
    if ((__popc(idle) >= LINE_REFILL) && (qn > 0 || rt < total)) {
      while (qn < min(__popc(idle), LINE_QCAP - 30) && rt < total) {
        // ---- set up 32 vertices: the 31 segments between them ----
        if (!located) {
          e0 = list_slot(wl.first, nlist, t0);
          located = true;
        }
        const unsigned long long t = t0 + lane;
        unsigned p;
        unsigned long long c;
        list_parts<31>(wl, nlist, t0, e0, p, c);
        bool joined = false;  // the next vertex continues the linestring
        unsigned long long v = 0;
        double x0 = 0.0, y0 = 0.0;
        if (t < total) {
          const unsigned long long rb = geo.ring_offsets[p], re = geo.ring_offsets[p + 1];
          v = geo.vertex_offsets[rb] + (t - c);
          const unsigned long long r = re - rb > 1 ? ring_of(geo, rb, re, v) : rb;
          joined = lane < 31 && v + 1 < geo.vertex_offsets[r + 1];
          const double2 w = geo.xy[v];
          x0 = to_px(g, w.x);
          y0 = to_py(g, w.y);
        }
        const long long ix0 = rzb::floor_i64(x0), iy0 = rzb::floor_i64(y0);
        const unsigned nan0 = (nan_bits(f64_bits(x0)) ? 1u : 0u) | (nan_bits(f64_bits(y0)) ? 2u : 0u);
        const long long ix1 = __shfl_down_sync(0xFFFFFFFFu, ix0, 1), iy1 = __shfl_down_sync(0xFFFFFFFFu, iy0, 1);
        const unsigned nan1 = __shfl_down_sync(0xFFFFFFFFu, nan0, 1);
        bool kept = false, push = false;
        uint4 f[NF];
        f[NF == 3 ? 2 : 3] = make_uint4(0u, 0u, 0u, 0u);
        const PartPlan& pl = plan[p];
        if (joined) {
          // extract_line's filter (edges.rs:112-134) on the floors: the raster's
          // bounds are integers; its minima and maxima ignore NaN
          auto meets = [](long long a, long long b, bool na, bool nb, long long size) {
            return ((!na && a < size) || (!nb && b < size)) && ((!na && a >= 0) || (!nb && b >= 0));
          };
          kept = meets(ix0, ix1, nan0 & 1u, nan1 & 1u, pl.ncols) && meets(iy0, iy1, nan0 & 2u, nan1 & 2u, pl.nrows);
        }
        if constexpr (TOUCHED) {
          const double x1 = __shfl_down_sync(0xFFFFFFFFu, x0, 1), y1 = __shfl_down_sync(0xFFFFFFFFu, y0, 1);
          if (kept) push = LineWalk<true>::setup(x0, y0, x1, y1, v, pl, f, ctrl);
        } else {
          if (kept) push = LineWalk<false>::setup(ix0, iy0, ix1, iy1, v, f, ctrl);
        }
        if (push) {
          // a polygon's ring walk carries the polygon's flags: it shares the
          // polygon's PixelCache (sum / count only), not the non-square-pixel
          // cache of LineString::burn
          f[NF == 3 ? 1 : 2] = make_uint4(p | pl.flags, pl.wid0, pl.wpr, (unsigned)pl.ncols);
          f[NF == 3 ? 2 : 3].x = (unsigned)pl.rlo;
          f[NF == 3 ? 2 : 3].y = (unsigned)(pl.rhi - pl.rlo);
        }
        if (!TOUCHED) {
          // the part's last kept segment so far: one atomic per part of the
          // group (parts are contiguous runs of lanes); 0 = no kept segment
          const unsigned km = __ballot_sync(0xFFFFFFFFu, kept);
          const unsigned later = lane == 31 ? 0u : km & ~((2u << lane) - 1u);
          const unsigned pn = __shfl_sync(0xFFFFFFFFu, p, later ? __ffs(later) - 1 : lane);
          if (kept && (!later || pn != p)) atomicMax(&last_kept[p], v + 1);
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, push);
        if (push) {
          const int k = qn + __popc(m & ((1u << lane) - 1u));
#pragma unroll
          for (int i = 0; i < NF; ++i) q[i * LINE_QCAP + k] = f[i];
        }
        qn += __popc(m);
        t0 += 31;
        if (t0 >= rt + range || t0 >= total) {
          rt = next_range();
          t0 = rt;
          located = false;
        }
      }
      __syncwarp();
      // ---- hand queued segments to the idle lanes ----
      const int take = min(qn, __popc(idle));
      const int k = __popc(idle & ((1u << lane) - 1u));
      if (!active && k < take) {
        const int e = qn - 1 - k;
        walk.load(q, e);
        const uint4 fb = q[(NF == 3 ? 1 : 2) * LINE_QCAP + e], fc = q[(NF == 3 ? 2 : 3) * LINE_QCAP + e];
        flags = fb.x;
        wid0 = fb.y;
        wpr = fb.z;
        ncols = fb.w;
        rlo = fc.x;
        nr = fc.y;
        active = true;
      }
      qn -= take;
      __syncwarp();
    }
    if (!__any_sync(0xFFFFFFFFu, active)) break;  // nothing queued and nothing left to set up
    // ---- one pixel per lane, STEPS times ----
#pragma unroll
    for (int k = 0; k < STEPS; ++k) {
      bool emit = false;
      unsigned ewid = 0, eflags = 0, emask = 0;
      if (active) {
        unsigned px, py;
        bool twice = false;
        const bool once = !repeats || (flags & DEDUP_BIT);
        active = walk.step(px, py, once, twice, geo, g, plan, flags & ~DEDUP_BIT, ctrl);
        if (px < ncols && py - rlo < nr) {
          const unsigned wid = wid0 + py * wpr + (px >> 5), bit = 1u << (px & 31u);
          // a pixel visited again is another write of it, which starts a new
          // record unless the part writes a pixel once or repeats change nothing
          const bool same = wid == cwid && flags == cflags, again = same && (cmask & bit);
          if (once) npix += (twice ? 1u : 0u) + (again ? 1u : 0u);
          if (!same || (again && !once)) {
            emit = cmask != 0u;
            ewid = cwid;
            eflags = cflags;
            emask = cmask;
            cwid = wid;
            cflags = flags;
            cmask = 0u;
          }
          cmask |= bit;
        }
      }
      if (emit) npix += (unsigned long long)__popc(emask);
      line_push(st, emit, ewid, eflags, emask, merge);
    }
  }
  npix += (unsigned long long)__popc(cmask);
  line_push(st, cmask != 0u, cwid, cflags, cmask, merge);
  merge();
  table_flush(tab, sb, bucket_count, ctrl);
  for (int o = 16; o > 0; o >>= 1) npix += __shfl_xor_sync(0xFFFFFFFFu, npix, o);
  if (lane == 0 && npix) atomicAdd(&ctrl->pixel_writes, npix);
}

template <bool TOUCHED, int STEPS = 1>
__global__ void __launch_bounds__(LINE_WARPS * 32, TOUCHED ? 5 : 6)
    k_line_spans(Geo geo, Grid g, const PartPlan* __restrict__ plan, WorkList wl, unsigned long long* last_kept,
                 int repeats, RecBuf sb, unsigned* bucket_count, Ctrl* ctrl) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (ctrl->err) return;
  line_body<TOUCHED, STEPS>(geo, g, plan, wl, last_kept, repeats, sb, bucket_count, ctrl, smem);
}

}  // namespace rzd
