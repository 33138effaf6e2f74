// rz_fill.cuh -- bucket fill: every (band, row, column-tile) bucket is staged
// as `background`, its coverage records are applied in part order (= the
// reference's per-geometry write order, rasterize.rs:162-196) with the pixel
// function, and the tile is written to the raster once.
//
// Pixel functions restate rust/src/rasterization/pixel_functions.rs:56-122
// (integer `+=` wraps, as in a release build of the crate).
#pragma once

#include <atomic>
#include <cstdint>
#include <type_traits>

#include "rz_device.cuh"

namespace rzd {

// One job of a batch call, as the fill sees it: where its buckets start and
// where its raster goes.
struct FillJob {
  unsigned long long bucket0;  // first bucket of the job (in the call's numbering)
  void* out;                   // (nrows, ncols) raster of the job
  int nrows, ncols;
  unsigned ntx, pad;
};

struct FillArgs {
  const unsigned* offsets;  // [nbuckets + 1]
  const uint2* recs;        // {part | word << REC_W_SHIFT | DEDUP_BIT, mask} grouped by bucket
  uint2* brecs;             // scratch of the records' size: the deep buckets' records grouped by word, at
                            // the records' own positions
  const void* pvals;        // burn value of each part (T), or nullptr: every record burns `scalar`
  unsigned long long nbuckets;
  unsigned long long scalar;  // raw bits of the single value when pvals == nullptr
  void* out;                // (bands, nrows, ncols)
  unsigned long long bg;    // raw bits of the background
  uint4 bg16;               // background replicated over 16 bytes
  int nrows, ncols;
  unsigned ntx;
  unsigned* big;            // buckets left to k_fill_big: the deep ones, and from its end on the shallow ones
  Ctrl* ctrl;
  unsigned long long rec_cap;
  int sort_max;              // tiles of up to this many records are sorted by one warp (<= FILL_WARP_SORT)
  int sort_cap;              // k_fill_warp: sort entries per warp (a power of two >= sort_max)
  int warp_bytes;            // k_fill_warp: shared memory per warp
  int chunk;                 // persistent fills: buckets per work grab (1..32)
  unsigned long long* work;  // chunk counter of this fill (zero before the launch)
  unsigned* nbig;            // entries of `big` (zero before the launch)
  unsigned* nshallow;        // entries of `big` from its end on (zero before the launch)
  // bucket b of this fill is bucket bucket0 + b of the call (a fill may run
  // over a sub-range of the buckets); batch calls: its raster is that of the
  // job owning it; jobs == nullptr: out / ncols / ntx
  const FillJob* jobs;
  unsigned n_jobs;
  unsigned long long bucket0;
};

__device__ __forceinline__ unsigned long long gb_of(const FillArgs& a, unsigned long long b) {
  return a.bucket0 + b;
}

// The raster tile of bucket b: its first pixel and its width (the last tile
// of a row is cut at ncols).
template <typename T>
__device__ __forceinline__ T* bucket_tile(const FillArgs& a, unsigned long long b, int& len) {
  T* out;
  int nrows, ncols;
  unsigned ntx, lb;
  if (a.jobs) {
    const unsigned long long gb = a.bucket0 + b;
    unsigned lo = 0, hi = a.n_jobs;  // jobs[lo].bucket0 <= gb < jobs[hi].bucket0
    while (hi - lo > 1) {
      const unsigned mid = (lo + hi) >> 1;
      if (a.jobs[mid].bucket0 <= gb) lo = mid; else hi = mid;
    }
    const FillJob j = a.jobs[lo];
    out = static_cast<T*>(j.out);
    nrows = j.nrows;
    ncols = j.ncols;
    ntx = j.ntx;
    lb = (unsigned)(gb - j.bucket0);
  } else {
    out = static_cast<T*>(a.out);
    nrows = a.nrows;  // all bands: rows of the (bands * nrows) stack
    ncols = a.ncols;
    ntx = a.ntx;
    lb = (unsigned)(a.bucket0 + b);  // a fill of a sub-range starts at bucket bucket0
  }
  const unsigned rowid = lb / ntx;  // 32-bit: a 64-bit divide runs on the FP64 pipe
  const int c0 = (int)(lb - rowid * ntx) << TW_SHIFT;
  len = min(TW, ncols - c0);
  if (rowid >= (unsigned)nrows) {  // never taken: the buckets of a fill are its rasters' tiles
    if ((threadIdx.x & 31) == 0) set_error(a.ctrl, ERR_RANGE, gb_of(a, b));
    len = 0;
    return out;
  }
  return out + (unsigned long long)rowid * (unsigned long long)ncols + c0;
}

// The raster tiles of consecutive buckets, without a division (and, in a
// batch, a search for the owning job) per bucket.
template <typename T>
struct TileIter {
  T* out;
  unsigned row, tx, ntx;
  int nrows, ncols;
  unsigned long long gb, end;  // current bucket, first bucket of the next job

  __device__ __forceinline__ void init(const FillArgs& a, unsigned long long b) {
    gb = b;
    unsigned long long lb = b;
    end = ~0ull;
    if (a.jobs) {
      unsigned lo = 0, hi = a.n_jobs;  // jobs[lo].bucket0 <= gb < jobs[hi].bucket0
      while (hi - lo > 1) {
        const unsigned mid = (lo + hi) >> 1;
        if (a.jobs[mid].bucket0 <= gb) lo = mid; else hi = mid;
      }
      const FillJob j = a.jobs[lo];
      out = static_cast<T*>(j.out);
      nrows = j.nrows;
      ncols = j.ncols;
      ntx = j.ntx;
      lb -= j.bucket0;
      if (lo + 1 < a.n_jobs) end = a.jobs[lo + 1].bucket0;
    } else {
      out = static_cast<T*>(a.out);
      nrows = a.nrows;  // all bands: rows of the (bands * nrows) stack
      ncols = a.ncols;
      ntx = a.ntx;
    }
    row = (unsigned)lb / ntx;  // 32-bit: a 64-bit divide runs on the FP64 pipe
    tx = (unsigned)lb - row * ntx;
  }
  __device__ __forceinline__ void next(const FillArgs& a) {
    if (++gb == end) init(a, gb);
    else if (++tx == ntx) {
      tx = 0;
      ++row;
    }
  }
  // the tile's first pixel and its width (the last tile of a row is cut at ncols)
  __device__ __forceinline__ T* tile(const FillArgs& a, int& len) const {
    const int c0 = (int)(tx << TW_SHIFT);
    len = min(TW, ncols - c0);
    if (row >= (unsigned)nrows) {  // never taken: the buckets of a fill are its rasters' tiles
      if ((threadIdx.x & 31) == 0) set_error(a.ctrl, ERR_RANGE, gb);
      len = 0;
      return out;
    }
    return out + (unsigned long long)row * (unsigned long long)ncols + c0;
  }
};

template <typename T> __device__ __forceinline__ bool is_nan_v(T v) { return false; }
template <> __device__ __forceinline__ bool is_nan_v<float>(float v) { return isnan(v); }
template <> __device__ __forceinline__ bool is_nan_v<double>(double v) { return isnan(v); }

template <typename T> __device__ __forceinline__ T add_wrap(T a, T b) {
  if constexpr (std::is_integral<T>::value) {
    using U = typename std::make_unsigned<T>::type;
    return (T)(U)((U)a + (U)b);
  } else {
    return a + b;
  }
}

template <typename T> __device__ __forceinline__ T from_bits(unsigned long long b) {
  T v;
  memcpy(&v, &b, sizeof(T));
  return v;
}

template <typename T> inline T from_bits_host(unsigned long long b) {
  T v;
  memcpy(&v, &b, sizeof(T));
  return v;
}

enum { F_SUM = 0, F_FIRST = 1, F_LAST = 2, F_MIN = 3, F_MAX = 4, F_COUNT = 5, F_ANY = 6 };

template <typename T, int FN>
__device__ __forceinline__ void apply_px(T& cur, T v, T bg) {
  if constexpr (FN == F_SUM) {
    if (cur == bg || is_nan_v(cur) || is_nan_v(v)) cur = v; else cur = add_wrap(cur, v);
  } else if constexpr (FN == F_FIRST) {
    if (cur == bg || is_nan_v(cur)) cur = v;
  } else if constexpr (FN == F_LAST) {
    cur = v;
  } else if constexpr (FN == F_MIN) {
    if (cur == bg || is_nan_v(cur) || cur > v) cur = v;
  } else if constexpr (FN == F_MAX) {
    if (cur == bg || is_nan_v(cur) || cur < v) cur = v;
  } else if constexpr (FN == F_COUNT) {
    if (cur == bg || is_nan_v(cur)) cur = T(1); else cur = add_wrap(cur, T(1));
  } else {
    cur = T(1);
  }
}

// float64 fold with the comparisons on the integer pipe: `cur == bg`, NaN
// tests and `<`/`>` are decided on the bit patterns (IEEE: -0 == +0, NaN
// compares false), only the accumulating add of sum/count issues FP64.
using rzb::BgF64;
using rzb::bg_f64;
using rzb::eq_bg_f64;
using rzb::gt_f64;

template <int FN>
__device__ __forceinline__ void apply_px_f64(double& cur, double v, const BgF64& bg) {
  const unsigned long long c = f64_bits(cur);
  if constexpr (FN == F_SUM) {
    if (eq_bg_f64(c, bg) || nan_bits(c) || nan_bits(f64_bits(v))) cur = v; else cur = __dadd_rn(cur, v);
  } else if constexpr (FN == F_FIRST) {
    if (eq_bg_f64(c, bg) || nan_bits(c)) cur = v;
  } else if constexpr (FN == F_LAST) {
    cur = v;
  } else if constexpr (FN == F_MIN) {
    if (eq_bg_f64(c, bg) || nan_bits(c) || gt_f64(c, f64_bits(v))) cur = v;
  } else if constexpr (FN == F_MAX) {
    if (eq_bg_f64(c, bg) || nan_bits(c) || gt_f64(f64_bits(v), c)) cur = v;
  } else if constexpr (FN == F_COUNT) {
    if (eq_bg_f64(c, bg) || nan_bits(c)) cur = 1.0; else cur = __dadd_rn(cur, 1.0);
  } else {
    cur = 1.0;
  }
}

// one pixel-function step; for float64 the background is pre-classified
template <typename T, int FN>
__device__ __forceinline__ void apply_one(T& cur, T v, T bg, const BgF64& bgc) {
  if constexpr (std::is_same<T, double>::value) apply_px_f64<FN>(cur, v, bgc);
  else apply_px<T, FN>(cur, v, bg);
}

// The first write onto the background always takes the reset branch of
// every pixel function (cur == bg, or cur is NaN when bg is NaN): its result
// is the value itself, or 1 for count / any.  No arithmetic is issued, so
// the compiler cannot speculate an FP64 add for it.
template <typename T, int FN>
__device__ __forceinline__ T first_write(T v) {
  if constexpr (FN == F_COUNT || FN == F_ANY) return T(1);
  else return v;
}

// The burn value of a record: its part's value (values[geometry of the part],
// gathered once per part by the prep), or the call's single value.
template <typename T>
__device__ __forceinline__ T rec_value(const FillArgs& a, unsigned rec_x) {
  if (a.pvals) return static_cast<const T*>(a.pvals)[rec_x & REC_PART_MASK];
  return from_bits<T>(a.scalar);
}

// ---- order-free first / last ---------------------------------------------
// `last` leaves a pixel at the value of the largest part that writes it.
// `first` takes the first write and keeps it unless it is the background or
// NaN (pixel_functions.rs:56-122), and every part writes one value: so the
// pixel ends at the value of the smallest part whose value is neither
// ("sticky"), or -- when no written value is sticky -- at the value of the
// largest part (every write replaced the one before).  Both are reductions
// over the parts that write the pixel, and need no sort: one pass over the
// records in any order keeps, per pixel, the largest part (+1, 0 = none) and,
// for `first`, the smallest sticky part (~0u = none).
constexpr int OF_WARP_MAX = 1024;  // deeper buckets go to the per-word kernel

template <typename T>
__device__ __forceinline__ T part_value(const FillArgs& a, unsigned p) {
  if (a.pvals) return static_cast<const T*>(a.pvals)[p];
  return from_bits<T>(a.scalar);
}

template <typename T>
__device__ __forceinline__ bool first_resets(T v, T bg, const BgF64& bgc) {
  if constexpr (std::is_same<T, double>::value) {
    const unsigned long long b = f64_bits(v);
    return eq_bg_f64(b, bgc) || nan_bits(b);
  } else {
    return v == bg || is_nan_v(v);
  }
}

// A record for the order-free pass: the part, bit 31 set when its value is
// sticky for `first` (the DEDUP flag plays no role for first / last: a part
// writes one value, so repeated writes of a part change nothing).
template <typename T, int FN>
__device__ __forceinline__ unsigned of_key(unsigned rx, T v, T bg, const BgF64& bgc) {
  unsigned k = rx & REC_PART_MASK;
  if constexpr (FN == F_FIRST) {
    if (!first_resets<T>(v, bg, bgc)) k |= DEDUP_BIT;
  }
  return k;
}

template <int FN>
__device__ __forceinline__ void of_update(unsigned& maxp1, unsigned& ming, unsigned k) {
  const unsigned p = k & REC_PART_MASK;
  maxp1 = max(maxp1, p + 1u);
  if (FN == F_FIRST && (k & DEDUP_BIT)) ming = min(ming, p);
}

template <typename T, int FN>
__device__ __forceinline__ T of_result(const FillArgs& a, unsigned maxp1, unsigned ming, T bg) {
  if (FN == F_FIRST && ming != 0xFFFFFFFFu) return part_value<T>(a, ming);
  if (maxp1 == 0u) return bg;
  return part_value<T>(a, maxp1 - 1u);
}

// `min` / `max` (cur == bg || NaN || cur > v, resp. < v) are order-free
// too when no written value is the background or NaN: after the first write
// every step keeps the running minimum (maximum) and an equal value does not
// replace it, so the pixel ends at the value of the smallest part among those
// whose value equals the extreme (only -0.0 and +0.0 are equal with other
// bits).  A pass that meets such a value falls back to the sorted fold.
template <typename T, int FN>
__device__ __forceinline__ bool of_better(T v, unsigned p, T bv, unsigned bp) {
  if (bp == 0xFFFFFFFFu) return true;
  bool ahead, eq;
  if constexpr (std::is_same<T, double>::value) {
    const unsigned long long x = f64_bits(v), y = f64_bits(bv);
    ahead = FN == F_MIN ? gt_f64(y, x) : gt_f64(x, y);
    eq = x == y || ((x | y) & 0x7FFFFFFFFFFFFFFFull) == 0;
  } else {
    ahead = FN == F_MIN ? v < bv : v > bv;
    eq = v == bv;
  }
  return ahead || (eq && p < bp);
}

// A 32-bit key that orders values of at most four bytes (NaN aside, which
// falls back before a key is used): the larger key is the value `max`
// (`min`) ends at.
template <typename T, int FN>
__device__ __forceinline__ unsigned of_value_key(T v) {
  unsigned k = 0;
  if constexpr (std::is_same<T, float>::value) {
    k = __float_as_uint(v);
    k ^= (unsigned)((int)k >> 31) | 0x80000000u;
  } else if constexpr (std::is_integral<T>::value) {
    k = std::is_signed<T>::value ? (unsigned)(int)v ^ 0x80000000u : (unsigned)v;
  }
  return FN == F_MIN ? ~k : k;
}

template <typename T, int FN>
__device__ __forceinline__ T of_key_value(unsigned k) {
  if (FN == F_MIN) k = ~k;
  if constexpr (std::is_same<T, float>::value) return __uint_as_float(k >> 31 ? k ^ 0x80000000u : ~k);
  else if constexpr (std::is_signed<T>::value) return (T)(int)(k ^ 0x80000000u);
  else return (T)k;
}

template <typename T>
__device__ __forceinline__ bool of_minus_zero(T v) {
  if constexpr (std::is_same<T, float>::value) return __float_as_uint(v) == 0x80000000u;
  return false;
}

template <typename T>
__device__ __forceinline__ T shfl_val(T v, int src) {
  if constexpr (sizeof(T) == 8) {
    unsigned long long b;
    memcpy(&b, &v, 8);
    b = __shfl_sync(0xFFFFFFFFu, b, src);
    T r;
    memcpy(&r, &b, 8);
    return r;
  } else {
    unsigned b = 0;
    memcpy(&b, &v, sizeof(T));
    b = __shfl_sync(0xFFFFFFFFu, b, src);
    T r;
    memcpy(&r, &b, sizeof(T));
    return r;
  }
}



// Write a tile's `len` values by one warp with 16-byte stores: the values
// before the first 16-byte boundary and behind the last one go one by one
// (a raster whose rows are no multiple of 16 bytes starts its tiles anywhere).
// elem(i) is value i, vec(i) the 16 bytes from value i on.
template <typename T, typename Elem, typename Vec>
__device__ __forceinline__ void store_values(T* dst, int len, Elem&& elem, Vec&& vec) {
  constexpr int E = 16 / (int)sizeof(T);
  const int lane = threadIdx.x & 31;
  const int off = (int)(reinterpret_cast<uintptr_t>(dst) & 15);
  const int head = off ? min(len, (16 - off) / (int)sizeof(T)) : 0;
  if (lane < head) dst[lane] = elem(lane);
  const int nv = (len - head) / E;
  uint4* d4 = reinterpret_cast<uint4*>(dst + head);
  for (int i = lane; i < nv; i += 32) __stcs(d4 + i, vec(head + i * E));
  const int tail = head + nv * E + lane;
  if (tail < len) dst[tail] = elem(tail);
}

template <typename T>
__device__ __forceinline__ void store_bg(T* dst, int len, const uint4& bg16, T bg) {
  store_values<T>(dst, len, [&](int) { return bg; }, [&](int) { return bg16; });
}

// 16 bytes of values from the coverage bits of their pixels: 1 where a bit is
// set, the background elsewhere.
template <typename T>
__device__ __forceinline__ uint4 expand_any(unsigned bits, const uint4& bg16, T one) {
  unsigned w[4], b[4] = {bg16.x, bg16.y, bg16.z, bg16.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (sizeof(T) == 1) {  // four pixels a word: spread four bits to the bytes' low bits
      const unsigned x = ((bits >> (4 * i)) & 15u) * 0x00204081u & 0x01010101u;
      w[i] = x | (b[i] & ~(x * 255u));
    } else if constexpr (sizeof(T) == 2) {
      const unsigned x = ((bits >> (2 * i)) & 1u) | ((bits >> (2 * i + 1)) & 1u) << 16;
      w[i] = x | (b[i] & ~(x * 65535u));
    } else if constexpr (sizeof(T) == 4) {
      unsigned o;
      memcpy(&o, &one, 4);
      w[i] = (bits >> i) & 1u ? o : b[i];
    } else {
      unsigned long long o;
      memcpy(&o, &one, 8);
      w[i] = (bits >> (i / 2)) & 1u ? (unsigned)(i & 1 ? o >> 32 : o) : b[i];
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// One pixel-function step, with the FP64 add of a float64 sum issued only
// when some lane of the warp needs it (a write onto the background takes the
// reset branch of every pixel function and needs no arithmetic).
template <typename T, int FN>
__device__ __forceinline__ void apply_step(T& c, T v, bool on, T bg, const BgF64& bgc) {
  if constexpr (std::is_same<T, double>::value && (FN == F_SUM || FN == F_COUNT)) {
    const unsigned long long cb = f64_bits(c);
    const bool reset = eq_bg_f64(cb, bgc) || nan_bits(cb) || (FN == F_SUM && nan_bits(f64_bits(v)));
    if (on && reset) c = FN == F_SUM ? v : 1.0;
    const bool add = on && !reset;
    if (__any_sync(0xFFFFFFFFu, add)) {
      if (add) c = __dadd_rn(c, FN == F_SUM ? v : 1.0);
    }
  } else {
    if (on) apply_one<T, FN>(c, v, bg, bgc);
  }
}

// ---- warp fill -------------------------------------------------------------
// One warp per bucket.  A warp takes FILL_CHUNK consecutive buckets (one coalesced
// load of their offsets) and loads the next bucket's records and values
// while it works on the current one.
//
// Records of different words touch different pixels, so only the part
// order within a word matters.  Up to FILL_WARP_MAX records are sorted by
// (word, part) with a bitonic network in registers (two records per lane),
// up to the schedule's sort_max by sorted_tile, and then walked once:
// lane l keeps pixel l of the current word in a register, applies each
// record whose mask covers it, and stores the word when the walk moves on
// (words without records are background).  A pixel-function step that needs
// a float64 add issues it only when some lane of the warp needs it.  Records
// of one deduplicating part and word are adjacent in the order and write a
// pixel once (PixelCache).  Deeper buckets go to the per-word kernel.
//
// first / last, and min / max when no written value is the background or NaN,
// take an order-free pass instead (buckets of up to OF_WARP_MAX records).
constexpr int FILL_WARPS_PER_BLOCK = 8;
constexpr int FILL_CHUNK = 4;       // buckets per work grab, at least
constexpr int FILL_CHUNK_MAX = 32;  // and at most: a lane per bucket's offset
constexpr int OF_LIGHT = 8;         // order-free passes: pixels of a record its own lane takes one by one

// Shared memory of one k_fill_warp warp: the sort's keys (a
// power of two of entries, at least sort_max, so that the bitonic network's
// padding stays inside), or the order-free pass's per-pixel state.  A smaller sort_max lets more warps share an SM.
inline int fill_sort_cap(int sort_max) {
  int e = FILL_WARP_MAX;
  while (e < sort_max) e <<= 1;
  return e;
}

template <typename T>
inline int fill_warp_bytes(int fn, int sort_cap) {
  int b = sort_cap * 8;
  // the order-free passes never sort
  if (fn == F_LAST) b = WPT * 33 * 4;
  if (fn == F_FIRST) b = 2 * WPT * 33 * 4;
  if (fn == F_MIN || fn == F_MAX) b = sizeof(T) <= 4 ? WPT * 34 * 4 : WPT * 32 * ((int)sizeof(T) + 4);
  return (b + 15) & ~15;
}

// the two records (positions lane and lane + 32) of a bucket held by a lane
template <typename T>
struct LanePair {
  uint2 r0, r1;
  T v0, v1;
};

template <typename T>
__device__ __forceinline__ LanePair<T> load_pair(const FillArgs& a, unsigned o0, int n) {
  const int lane = threadIdx.x & 31;
  LanePair<T> p;
  p.r0 = p.r1 = make_uint2(0u, 0u);
  p.v0 = p.v1 = T(0);
  if (n <= FILL_WARP_MAX) {
    if (lane < n) {
      p.r0 = a.recs[o0 + lane];
      p.v0 = rec_value<T>(a, p.r0.x);
    }
    if (lane + 32 < n) {
      p.r1 = a.recs[o0 + lane + 32];
      p.v1 = rec_value<T>(a, p.r1.x);
    }
  }
  return p;
}

// Bitonic sort of one 32-bit key per lane, ascending or descending.
__device__ __forceinline__ unsigned warp_sort32(unsigned x, bool ascending) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int kk = 2; kk <= 32; kk <<= 1)
#pragma unroll
    for (int j = kk >> 1; j > 0; j >>= 1) {
      const unsigned y = __shfl_xor_sync(0xFFFFFFFFu, x, j);
      const bool up = ((lane & kk) == 0 || kk == 32) == ascending;  // kk == 32: one block
      x = ((lane & j) == 0) == up ? min(x, y) : max(x, y);
    }
  return x;
}

// Sort the keys at positions lane and lane + 32 ascending (two: both halves
// are in use).
__device__ __forceinline__ void warp_sort64(unsigned& x0, unsigned& x1, bool two) {
  const int lane = threadIdx.x & 31;
  x0 = warp_sort32(x0, true);
  if (!two) return;
  x1 = warp_sort32(x1, false);
  const unsigned lo = min(x0, x1), hi = max(x0, x1);  // a bitonic sequence in each half
  x0 = lo;
  x1 = hi;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const unsigned y0 = __shfl_xor_sync(0xFFFFFFFFu, x0, j), y1 = __shfl_xor_sync(0xFFFFFFFFu, x1, j);
    x0 = (lane & j) == 0 ? min(x0, y0) : max(x0, y0);
    x1 = (lane & j) == 0 ? min(x1, y1) : max(x1, y1);
  }
}

// 32 x 32 bit transpose across a warp: lane i holds row i on entry and
// column l (bit i = bit l of row i) in lane l on return.  Five butterfly
// stages, each swapping the off-diagonal j x j blocks of every 2j x 2j block.
__device__ __forceinline__ unsigned warp_transpose32(unsigned x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int j = 16 >> s;
    const unsigned m = s == 0 ? 0x0000FFFFu : s == 1 ? 0x00FF00FFu : s == 2 ? 0x0F0F0F0Fu : s == 3 ? 0x33333333u
                                                                                                    : 0x55555555u;
    const unsigned y = __shfl_xor_sync(0xFFFFFFFFu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y << j) & ~m));
  }
  return x;
}

// Apply the records in `bits` (this lane's pixel, in part order; record r is
// held by lane r: value v, x = part | DEDUP_BIT) to c.  Every step each lane
// takes its own next record, so a word costs as many steps as its deepest
// pixel has records, not as many as it has records.  `last`: the part that
// wrote the pixel last.  `fresh`: c is the background, and the first write
// takes the reset branch of every pixel function.
template <typename T, int FN, bool DEDUP>
__device__ __forceinline__ void fold_bits(unsigned bits, T v, unsigned x, bool fresh, T& c, unsigned& last, T bg,
                                          const BgF64& bgc) {
  if (fresh) {
    const int r = (__ffs(bits) - 1) & 31;
    const T vr = shfl_val<T>(v, r);
    const unsigned xr = DEDUP ? __shfl_sync(0xFFFFFFFFu, x, r) : 0u;
    if (bits) {
      c = first_write<T, FN>(vr);
      last = xr;
    }
    bits &= bits - 1u;
  }
  while (__any_sync(0xFFFFFFFFu, bits != 0u)) {
    const int r = (__ffs(bits) - 1) & 31;
    const T vr = shfl_val<T>(v, r);
    bool on = bits != 0u;
    if (DEDUP) {
      const unsigned xr = __shfl_sync(0xFFFFFFFFu, x, r);
      if (on) {
        on = !(xr & DEDUP_BIT) || xr != last;  // a deduplicating part writes a pixel once
        last = xr;
      }
    }
    apply_step<T, FN>(c, vr, on, bg, bgc);
    bits &= bits - 1u;
  }
}

// The fold of a tile's records in (word, part) order, 32 at a time: lane l
// keeps pixel l of the current word and stores the word when the records move
// on; words without records are background.
template <typename T, int FN, bool DEDUP>
struct TileFold {
  T* dst;
  int len;
  T bg;
  int cw = -1;  // current word
  T c;
  unsigned last = 0xFFFFFFFFu;

  __device__ __forceinline__ TileFold(T* d, int l, T b) : dst(d), len(l), bg(b), c(b) {}
  __device__ __forceinline__ void move_to(int w) {
    const int lane = threadIdx.x & 31;
    if (cw >= 0 && cw * 32 + lane < len) dst[cw * 32 + lane] = c;
    for (int ww = cw + 1; ww < w; ++ww)
      if (ww * 32 + lane < len) dst[ww * 32 + lane] = bg;
    cw = w;
    c = bg;
    last = 0xFFFFFFFFu;
  }
  // records of lanes 0..cnt-1, in order: x = part | word | DEDUP_BIT
  __device__ __forceinline__ void add(unsigned x, unsigned mask, T v, int cnt, const BgF64& bgc) {
    const int lane = threadIdx.x & 31;
    const bool in = lane < cnt;
    const unsigned t = warp_transpose32(in ? mask : 0u);
    const int w = in ? (int)((x >> REC_W_SHIFT) & 15u) : -1;
    unsigned rest = __ballot_sync(0xFFFFFFFFu, in);
    while (rest) {
      const int cur = __shfl_sync(0xFFFFFFFFu, w, __ffs(rest) - 1);
      const unsigned wm = __ballot_sync(0xFFFFFFFFu, w == cur);
      rest &= ~wm;
      const bool fresh = cur != cw;
      if (fresh) move_to(cur);
      fold_bits<T, FN, DEDUP>(t & wm, v, x & ~(15u << REC_W_SHIFT), fresh, c, last, bg, bgc);
    }
  }
  __device__ __forceinline__ void finish() { move_to(WPT); }
};

// The fold of a tile of n <= 64 records, two per lane, sorted in registers by
// one 32-bit key: word, part relative to the tile's smallest, position; false
// (nothing written) when the parts are 2^22 or more apart.
template <typename T, int FN, bool DEDUP>
__device__ __forceinline__ bool fold_pair(const LanePair<T>& pr, int n, T* dst, int len, T bg, const BgF64& bgc) {
  const int lane = threadIdx.x & 31;
  const unsigned p0 = pr.r0.x & REC_PART_MASK, p1 = pr.r1.x & REC_PART_MASK;
  const bool in0 = lane < n, in1 = lane + 32 < n;
  const unsigned lo = __reduce_min_sync(0xFFFFFFFFu, in0 ? (in1 ? min(p0, p1) : p0) : 0xFFFFFFFFu);
  const unsigned hi = __reduce_max_sync(0xFFFFFFFFu, in0 ? (in1 ? max(p0, p1) : p0) : 0u);
  if (hi - lo >= (1u << 22) - 1u) return false;
  auto key = [&](unsigned x, unsigned p, unsigned i) {
    return ((x >> REC_W_SHIFT) & 15u) << 28 | (p - lo) << 6 | i;
  };
  unsigned k0 = in0 ? key(pr.r0.x, p0, (unsigned)lane) : 0xFFFFFFFFu;
  unsigned k1 = in1 ? key(pr.r1.x, p1, (unsigned)lane + 32u) : 0xFFFFFFFFu;
  const unsigned nk0 = __shfl_down_sync(0xFFFFFFFFu, k0, 1), nk1 = __shfl_down_sync(0xFFFFFFFFu, k1, 1);
  const unsigned k1_first = __shfl_sync(0xFFFFFFFFu, k1, 0);
  const bool ord = k0 <= (lane == 31 ? k1_first : nk0) && (lane == 31 || k1 <= nk1);
  if (!__all_sync(0xFFFFFFFFu, ord)) warp_sort64(k0, k1, n > 32);
  // the record at sorted position lane (then lane + 32), from the lane that loaded it
  auto fetch = [&](unsigned k, unsigned& x, unsigned& m, T& v) {
    const int src = (int)(k & 31u);
    x = __shfl_sync(0xFFFFFFFFu, pr.r0.x, src);
    m = __shfl_sync(0xFFFFFFFFu, pr.r0.y, src);
    v = shfl_val<T>(pr.v0, src);
    if (n > 32) {
      const unsigned xb = __shfl_sync(0xFFFFFFFFu, pr.r1.x, src), mb = __shfl_sync(0xFFFFFFFFu, pr.r1.y, src);
      const T vb = shfl_val<T>(pr.v1, src);
      if (k & 32u) {
        x = xb;
        m = mb;
        v = vb;
      }
    }
  };
  unsigned x, m;
  T v;
  TileFold<T, FN, DEDUP> fold(dst, len, bg);
  fetch(k0, x, m, v);
  fold.add(x, m, v, min(n, 32), bgc);
  if (n > 32) {
    fetch(k1, x, m, v);
    fold.add(x, m, v, n - 32, bgc);
  }
  fold.finish();
  return true;
}

// ascending bitonic sort of k[0..np) (np = next power of two >= n, padded
// with ~0) by one warp in shared memory
__device__ __forceinline__ void warp_sort_u64(unsigned long long* k, int n) {
  int np = 1;
  while (np < n) np <<= 1;
  const int lane = threadIdx.x & 31;
  for (int i = n + lane; i < np; i += 32) k[i] = ~0ull;
  __syncwarp();
  for (int kk = 2; kk <= np; kk <<= 1) {
    for (int j = kk >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < np; i += 32) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long x = k[i], y = k[ixj];
          const bool up = (i & kk) == 0;
          if ((x > y) == up) {
            k[i] = y;
            k[ixj] = x;
          }
        }
      }
      __syncwarp();
    }
  }
}

// Sort 32 K keys ascending across a warp, lane l holding positions K l to
// K l + K - 1: bitonic, the steps below K inside a lane.  Descending runs are
// sorted with their keys inverted.
template <int K>
__device__ __forceinline__ void warp_sort_keys32(unsigned (&x)[K]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int kk = 2; kk <= 32 * K; kk <<= 1) {
    unsigned inv[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const bool down = kk < K ? (k & kk) != 0 : (lane & (kk / K)) != 0;
      inv[k] = down ? ~0u : 0u;
      x[k] ^= inv[k];
    }
#pragma unroll
    for (int j = kk >> 1; j > 0; j >>= 1) {
      if (j >= K) {
        const bool lower = (lane & (j / K)) == 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const unsigned y = __shfl_xor_sync(0xFFFFFFFFu, x[k], j / K);
          x[k] = lower ? min(x[k], y) : max(x[k], y);
        }
      } else {
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (k & j) continue;
          const unsigned lo = min(x[k], x[k | j]), hi = max(x[k], x[k | j]);
          x[k] = lo;
          x[k | j] = hi;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) x[k] ^= inv[k];
  }
}

// Write the positions of the n <= 32 K records of a tile or word to spos in
// (word, part) order, sorted in registers by word, part relative to the tile's
// smallest and position; false (nothing written) when the parts are too far
// apart for one 32-bit key.
template <int K>
__device__ __forceinline__ bool sort_positions(const uint2* recs, int n, unsigned char* spos) {
  constexpr int POS = K == 4 ? 7 : 8;  // bits of a position
  const int lane = threadIdx.x & 31;
  unsigned x[K], lo = 0xFFFFFFFFu, hi = 0u;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const bool in = k * 32 + lane < n;
    x[k] = in ? recs[k * 32 + lane].x : 0u;
    if (in) {
      lo = min(lo, x[k] & REC_PART_MASK);
      hi = max(hi, x[k] & REC_PART_MASK);
    }
  }
  lo = __reduce_min_sync(0xFFFFFFFFu, lo);
  hi = __reduce_max_sync(0xFFFFFFFFu, hi);
  if (hi - lo >= (1u << (28 - POS)) - 1u) return false;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const unsigned pos = (unsigned)(k * 32 + lane);
    x[k] = pos < (unsigned)n
               ? ((x[k] >> REC_W_SHIFT) & 15u) << 28 | ((x[k] & REC_PART_MASK) - lo) << POS | pos : 0xFFFFFFFFu;
  }
  warp_sort_keys32<K>(x);
  unsigned packed[(K + 3) / 4];
#pragma unroll
  for (int k = 0; k < K; k += 4)
    packed[k / 4] = (x[k] & 0xFFu) | (x[k + 1] & 0xFFu) << 8 | (x[k + 2] & 0xFFu) << 16 | x[k + 3] << 24;
#pragma unroll
  for (int k = 0; k < K / 4; ++k) reinterpret_cast<unsigned*>(spos)[lane * (K / 4) + k] = packed[k];
  return true;
}

// The fold of a tile of up to sort_max records, their places sorted in
// registers (up to 128: four keys a lane, up to 256: eight), or as 64-bit keys
// in shared memory where a tile's parts are 2^21 (2^20) or more apart.  Half
// of the 40 M records that a batch of uneven rasters sums lie in tiles of 65
// to 128: 2.05 ms with all of them sorted in shared memory and their records
// kept there (which left room for four blocks per SM), 1.33 ms so; 16 road
// networks 0.50 -> 0.33 ms.  Out of line: inlined, its registers and code
// slowed the order-free passes of min / max by a half.
template <typename T, int FN, bool DEDUP>
__device__ __noinline__ void sorted_tile(const FillArgs& a, unsigned o0, int n, unsigned long long* skey, T* dst,
                                         int len, T bg, const BgF64& bgc) {
  const int lane = threadIdx.x & 31;
  unsigned char* spos = reinterpret_cast<unsigned char*>(skey);
  __syncwarp();
  const bool regs = n <= 128 ? sort_positions<4>(a.recs + o0, n, spos) : sort_positions<8>(a.recs + o0, n, spos);
  if (!regs) {
    for (int i = lane; i < n; i += 32)
      skey[i] = ((unsigned long long)(a.recs[o0 + i].x & ~DEDUP_BIT) << 8) | (unsigned)i;
    warp_sort_u64(skey, n);
  }
  __syncwarp();
  TileFold<T, FN, DEDUP> fold(dst, len, bg);
  for (int i0 = 0; i0 < n; i0 += 32) {
    uint2 r = make_uint2(0u, 0u);
    T v = T(0);
    if (i0 + lane < n) {
      r = a.recs[o0 + (regs ? (unsigned)spos[i0 + lane] & (n <= 128 ? 0x7Fu : 0xFFu)
                            : (unsigned)skey[i0 + lane] & 0xFFu)];
      v = rec_value<T>(a, r.x);
    }
    fold.add(r.x, r.y, v, min(32, n - i0), bgc);
  }
  fold.finish();
  __syncwarp();
}

// Blocks per SM that the registers are cut to: the warps wait for records,
// values and stores, and 64 of them (32 registers) hide that best although
// the ordered folds then spill (large fill's float64 sum 1.21 -> 1.02 ms at 8,
// 1.06 at 6; a batch's sum 1.33 -> 1.27, its max 0.86 -> 0.80; 88 M records of
// max 1.74 -> 1.60).  0: left to the compiler, as first and last got slower
// (0.89 -> 0.92 ms), and 8-byte min / max have shared memory for four.
template <typename T, int FN>
constexpr int fill_warp_blocks() {
  return FN == F_FIRST || FN == F_LAST || ((FN == F_MIN || FN == F_MAX) && sizeof(T) > 4) ? 0 : 8;
}

template <typename T, int FN, bool DEDUP>
__global__ void __launch_bounds__(FILL_WARPS_PER_BLOCK * 32, fill_warp_blocks<T, FN>()) k_fill_warp(FillArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  // sum / count sort their tiles' records (prefetched, two a lane); the other
  // functions take the order-free passes.  Tiles that min / max of values of
  // up to four bytes have to fold in order are left to k_fill_big: with the
  // sorted fold in this kernel, in line or called, the compiler kept the warps
  // of the passes apart (100,000 polygons of float32 over 12,000 x 12,000
  // pixels, a max without such tiles: 1.01 ms a call, 1.41 with a call of
  // sorted_tile).  The wider passes lose nothing by the call (1.31 ms).
  constexpr bool PAIRS = FN == F_SUM || FN == F_COUNT;
  Ctrl* ctrl = a.ctrl;
  if (ctrl->err || ctrl->span_count > a.rec_cap) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* wbase = smem + warp * a.warp_bytes;
  const T bg = from_bits<T>(a.bg);
  const BgF64 bgc = bg_f64(a.bg);
  TileIter<T> it;
  while (true) {
    unsigned long long b0 = 0;
    if (lane == 0) b0 = atomicAdd(a.work, (unsigned long long)a.chunk);
    b0 = __shfl_sync(0xFFFFFFFFu, b0, 0);
    if (b0 >= a.nbuckets) break;
    const int nb = (int)min((unsigned long long)a.chunk, a.nbuckets - b0);
    it.init(a, a.bucket0 + b0);
    const unsigned off = a.offsets[b0 + (lane < nb ? lane : nb)];
    const unsigned off_end = a.offsets[b0 + nb];
    unsigned o_next = __shfl_sync(0xFFFFFFFFu, off, 0);
    int n_next = (int)((nb > 1 ? __shfl_sync(0xFFFFFFFFu, off, 1) : off_end) - o_next);
    LanePair<T> nxt;
    if constexpr (PAIRS) nxt = load_pair<T>(a, o_next, n_next);
    // order-free passes: the next tile's first 32 records, their keys or
    // values looked up when the current tile is done
    uint2 nrec = make_uint2(0u, 0u);
    constexpr bool AHEAD = !PAIRS && FN != F_LAST;  // last reads no values: 8 more registers cost it more
    if (AHEAD && lane < n_next) nrec = a.recs[o_next + lane];
    for (int k = 0; k < nb; ++k) {
      const unsigned long long b = b0 + k;
      const int n = n_next;
      const unsigned o_cur = o_next;
      LanePair<T> pr;
      if constexpr (PAIRS) pr = nxt;
      const uint2 rec0 = AHEAD || PAIRS ? nrec : (lane < n ? a.recs[o_cur + lane] : make_uint2(0u, 0u));
      T val0 = T(0);
      if ((FN == F_MIN || FN == F_MAX || FN == F_FIRST) && lane < n) val0 = rec_value<T>(a, rec0.x);
      if (k + 1 < nb) {  // prefetch the next bucket
        o_next = __shfl_sync(0xFFFFFFFFu, off, k + 1);
        n_next = (int)((k + 2 < nb ? __shfl_sync(0xFFFFFFFFu, off, (k + 2) & 31) : off_end) - o_next);
        if constexpr (PAIRS) nxt = load_pair<T>(a, o_next, n_next);
        else if constexpr (AHEAD) nrec = lane < n_next ? a.recs[o_next + lane] : make_uint2(0u, 0u);
      }
      int len;
      T* dst = it.tile(a, len);
      it.next(a);
      if (n == 0) {
        store_bg<T>(dst, len, a.bg16, bg);
        continue;
      }
      if constexpr (FN == F_FIRST || FN == F_LAST) {
        if (n > OF_WARP_MAX) {
          if (lane == 0) a.big[atomicAdd(a.nbig, 1u)] = (unsigned)b;
          continue;
        }
        // State per pixel (word w, bit l) at w * 32 + l, and per word at
        // WPT * 32 + w for the records that cover a whole word.  A record of
        // a whole word or of few pixels is taken by the lane that loaded it,
        // with shared-memory atomics; the others are broadcast to the warp,
        // each lane its pixel.  (Broadcasting all of them cost 20
        // instructions a record: 40,000 x 40,000 pixels of lines and
        // polygons, int32 max, which does the same: 3.9 ms, now 1.6.)
        unsigned* smax = reinterpret_cast<unsigned*>(wbase);
        unsigned* smin = smax + WPT * 33;
        __syncwarp();
        for (int x = lane; x < WPT * 33; x += 32) {
          smax[x] = 0u;
          if (FN == F_FIRST) smin[x] = 0xFFFFFFFFu;
        }
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += 32) {
          const int i = i0 + lane;
          unsigned kx = 0u, km = 0u, kw = 0u;
          if (i < n) {
            const uint2 r = i0 ? a.recs[o_cur + i] : rec0;
            kx = of_key<T, FN>(r.x, FN != F_FIRST ? T(0) : i0 ? rec_value<T>(a, r.x) : val0, bg, bgc);
            km = r.y;
            kw = (r.x >> REC_W_SHIFT) & 15u;
          }
          const bool whole = km == 0xFFFFFFFFu, heavy = !whole && __popc(km) > OF_LIGHT;
          auto take = [&](unsigned ix) {
            atomicMax(&smax[ix], (kx & REC_PART_MASK) + 1u);
            if (FN == F_FIRST && (kx & DEDUP_BIT)) atomicMin(&smin[ix], kx & REC_PART_MASK);
          };
          if (whole) take(WPT * 32u + kw);
          for (unsigned m = whole || heavy ? 0u : km; m; m &= m - 1u) take(kw * 32u + (unsigned)(__ffs(m) - 1));
          __syncwarp();  // the atomics are done before other lanes read and write the same words below
          unsigned hv = __ballot_sync(0xFFFFFFFFu, heavy);
          while (hv) {
            const int j = __ffs(hv) - 1;
            hv &= hv - 1u;
            const unsigned xj = __shfl_sync(0xFFFFFFFFu, kx, j), mj = __shfl_sync(0xFFFFFFFFu, km, j);
            const unsigned wj = __shfl_sync(0xFFFFFFFFu, kw, j);
            if ((mj >> lane) & 1u) {
              const unsigned ix = wj * 32u + (unsigned)lane;
              unsigned mx = smax[ix], mn = FN == F_FIRST ? smin[ix] : 0u;
              of_update<FN>(mx, mn, xj);
              smax[ix] = mx;
              if (FN == F_FIRST) smin[ix] = mn;
            }
          }
          __syncwarp();
        }
#pragma unroll
        for (int w = 0; w < WPT; ++w) {
          const int x = w * 32 + lane;
          if (x < len) {
            const unsigned mx = max(smax[x], smax[WPT * 32 + w]);
            const unsigned mn = FN == F_FIRST ? min(smin[x], smin[WPT * 32 + w]) : 0xFFFFFFFFu;
            dst[x] = of_result<T, FN>(a, mx, mn, bg);
          }
        }
        continue;
      }
      if constexpr ((FN == F_MIN || FN == F_MAX) && sizeof(T) <= 4) {
        if (n <= OF_WARP_MAX) {
          // as first / last, on ordered keys of the values: the extreme is
          // the largest key.  Pixels written are kept as one mask per word
          // (words covered whole: in their own mask), so no key is reserved.
          unsigned* skey = reinterpret_cast<unsigned*>(wbase);
          unsigned* sset = skey + WPT * 33;
          __syncwarp();
          for (int x = lane; x < WPT * 34; x += 32) skey[x] = 0u;
          __syncwarp();
          bool bad = false;
          for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            unsigned kv = 0u, km = 0u, kw = 0u;
            if (i < n) {
              const uint2 r = i0 ? a.recs[o_cur + i] : rec0;
              const T v = i0 ? rec_value<T>(a, r.x) : val0;
              kv = of_value_key<T, FN>(v);
              km = r.y;
              kw = (r.x >> REC_W_SHIFT) & 15u;
              // a value that resets the pixel, or -0 (equal to +0 with other bits)
              bad = bad || first_resets<T>(v, bg, bgc) || of_minus_zero<T>(v);
            }
            if (__any_sync(0xFFFFFFFFu, bad)) break;
            const bool whole = km == 0xFFFFFFFFu, heavy = !whole && __popc(km) > OF_LIGHT;
            if (km) atomicOr(&sset[kw], km);
            if (whole) atomicMax(&skey[WPT * 32u + kw], kv);
            for (unsigned m = whole || heavy ? 0u : km; m; m &= m - 1u)
              atomicMax(&skey[kw * 32u + (unsigned)(__ffs(m) - 1)], kv);
            __syncwarp();
            unsigned hv = __ballot_sync(0xFFFFFFFFu, heavy);
            while (hv) {
              const int j = __ffs(hv) - 1;
              hv &= hv - 1u;
              const unsigned vj = __shfl_sync(0xFFFFFFFFu, kv, j), mj = __shfl_sync(0xFFFFFFFFu, km, j);
              const unsigned wj = __shfl_sync(0xFFFFFFFFu, kw, j);
              const unsigned ix = wj * 32u + (unsigned)lane;
              const unsigned old = skey[ix];
              skey[ix] = (mj >> lane) & 1u ? max(old, vj) : old;
            }
            __syncwarp();
          }
          if (!__any_sync(0xFFFFFFFFu, bad)) {
            __syncwarp();
#pragma unroll
            for (int w = 0; w < WPT; ++w) {
              const int x = w * 32 + lane;
              // selected, not branched around: the warp stays together
              const T v = of_key_value<T, FN>(max(skey[x], skey[WPT * 32 + w]));
              const T o = (sset[w] >> lane) & 1u ? v : bg;
              if (x < len) dst[x] = o;
            }
            continue;
          }
        }
        // deep, or with a value that resets the pixel: the ordered fold of k_fill_big
        if (lane == 0) {
          if (n > a.sort_max) a.big[atomicAdd(a.nbig, 1u)] = (unsigned)b;
          else a.big[a.nbuckets - 1 - atomicAdd(a.nshallow, 1u)] = (unsigned)b;
        }
        continue;
      }
      if constexpr ((FN == F_MIN || FN == F_MAX) && sizeof(T) > 4) {
        if (n <= OF_WARP_MAX) {
          // per pixel (word w, lane l) at w * 32 + l: its extreme and part
          T* sval = reinterpret_cast<T*>(wbase);
          unsigned* spart = reinterpret_cast<unsigned*>(sval + WPT * 32);
#pragma unroll
          for (int w = 0; w < WPT; ++w) spart[w * 32 + lane] = 0xFFFFFFFFu;
          bool bad = false;
          for (int i0 = 0; i0 < n; i0 += 32) {
            const int i = i0 + lane;
            unsigned kx = 0u, km = 0u;
            T kv = T(0);
            if (i < n) {
              const uint2 r = a.recs[o_cur + i];
              kv = rec_value<T>(a, r.x);
              kx = r.x;
              km = r.y;
              bad = bad || first_resets<T>(kv, bg, bgc);
            }
            if (__any_sync(0xFFFFFFFFu, bad)) break;
            const int cnt = min(32, n - i0);
            for (int j = 0; j < cnt; ++j) {
              const unsigned xj = __shfl_sync(0xFFFFFFFFu, kx, j), mj = __shfl_sync(0xFFFFFFFFu, km, j);
              const T vj = shfl_val<T>(kv, j);
              if ((mj >> lane) & 1u) {
                const unsigned ix = ((xj >> REC_W_SHIFT) & 15u) * 32u + (unsigned)lane;
                const unsigned pj = xj & REC_PART_MASK;
                if (of_better<T, FN>(vj, pj, sval[ix], spart[ix])) {
                  sval[ix] = vj;
                  spart[ix] = pj;
                }
              }
            }
          }
          if (!__any_sync(0xFFFFFFFFu, bad)) {
#pragma unroll
            for (int w = 0; w < WPT; ++w) {
              const int x = w * 32 + lane;
              if (x < len) dst[x] = spart[x] == 0xFFFFFFFFu ? bg : sval[x];
            }
            continue;
          }
        }
        if (n <= a.sort_max)
          sorted_tile<T, FN, DEDUP>(a, o_cur, n, reinterpret_cast<unsigned long long*>(wbase), dst, len, bg, bgc);
        else if (lane == 0)
          a.big[atomicAdd(a.nbig, 1u)] = (unsigned)b;
        continue;
      }
      if constexpr (PAIRS) {
      if (n > a.sort_max) {
        if (lane == 0) a.big[atomicAdd(a.nbig, 1u)] = (unsigned)b;
        continue;
      }
      if (n <= FILL_WARP_MAX && fold_pair<T, FN, DEDUP>(pr, n, dst, len, bg, bgc)) continue;
      sorted_tile<T, FN, DEDUP>(a, o_cur, n, reinterpret_cast<unsigned long long*>(wbase), dst, len, bg, bgc);
      }
    }
  }
}

// The shallow tiles that min / max of values of up to four bytes leave to the
// ordered fold.  One warp per tile, as k_fill_warp's sum: up to 32 of them a
// warp at a time, the next tile's records loaded while one is folded.
template <typename T, int FN, bool DEDUP>
__device__ __forceinline__ void shallow_tiles(const FillArgs& a, unsigned w, unsigned warps, unsigned char* wbase, T bg,
                                              const BgF64& bgc) {
  const int lane = threadIdx.x & 31;
  const unsigned total = *a.nshallow;
  const unsigned group = min(32u, max(1u, total / (2u * warps)));
  for (unsigned g0 = w * group; g0 < total; g0 += warps * group) {
    unsigned b = 0, o = 0;
    int n = 0;
    if ((unsigned)lane < group && g0 + lane < total) {
      b = a.big[a.nbuckets - 1 - (g0 + lane)];
      o = a.offsets[b];
      n = (int)(a.offsets[b + 1] - o);
    }
    unsigned todo = __ballot_sync(0xFFFFFFFFu, n > 0);
    LanePair<T> nxt;
    auto load_next = [&]() {
      const int k = (__ffs(todo) - 1) & 31;
      const unsigned ok = __shfl_sync(0xFFFFFFFFu, o, k);
      const int nk = __shfl_sync(0xFFFFFFFFu, n, k);
      if (todo) nxt = load_pair<T>(a, ok, nk);
    };
    load_next();
    while (todo) {
      const int k = __ffs(todo) - 1;
      todo &= todo - 1u;
      const unsigned bk = __shfl_sync(0xFFFFFFFFu, b, k), ok = __shfl_sync(0xFFFFFFFFu, o, k);
      const int nk = __shfl_sync(0xFFFFFFFFu, n, k);
      const LanePair<T> pr = nxt;
      load_next();
      int len;
      T* dst = bucket_tile<T>(a, bk, len);
      if (nk > FILL_WARP_MAX || !fold_pair<T, FN, DEDUP>(pr, nk, dst, len, bg, bgc))
        sorted_tile<T, FN, DEDUP>(a, ok, nk, reinterpret_cast<unsigned long long*>(wbase), dst, len, bg, bgc);
    }
  }
}

// ---- deep buckets: one block per bucket, one warp per word ----------------
// The block first copies the bucket's records, grouped by word, to their own
// positions of `brecs` (counted and placed by all its warps), so that each
// word's warp reads only its own.  (One warp per bucket did this in a launch
// of its own: 0.48 ms of the 1.5 ms that 16 road networks spent here.)
// The word's records are taken in part order, at most big_cap() at a time: a
// histogram over the pending part ids picks the largest prefix range that
// fits, the range is gathered, sorted (bitonic, shared memory) and folded:
// lane l keeps pixel l of the word in a register and walks the sorted
// records to the next one covering its pixel, so every step applies one
// record per lane.  A single part with more than big_cap() records in the word
// is applied in chunks (its records share one value and their order does
// not change the result).  first / last, and min / max without a background
// or NaN value among the word's records, take one order-free pass instead.
// For min / max of values of up to four bytes the kernel takes their shallow
// tiles first; half the word's capacity and registers for three blocks per SM
// make those of 100,000 polygons, a value that resets the pixel in each, 0.42
// ms (one list for both kinds, which every block walked to its end, and two
// blocks: 0.82; the call 1.93 -> 1.42 ms).  The other functions of up to four
// bytes are held to two blocks (deep sums of 20,000 polygons over 600 x 600
// pixels 0.92 ms a call, 1.17 at one); 8-byte values have shared memory for one.
constexpr int BIG_WARPS = WPT;
constexpr int BIG_HIST = 256;

template <typename T, int FN>
constexpr bool big_takes_shallow() { return (FN == F_MIN || FN == F_MAX) && sizeof(T) <= 4; }

template <typename T, int FN>
constexpr int big_cap() { return big_takes_shallow<T, FN>() ? BIG_CAP / 2 : BIG_CAP; }

// The per-word state, or sorted_tile's (its sort entries are at most FILL_WARP_SORT).
template <typename T, int FN>
constexpr int big_warp_bytes() {
  const int word = big_cap<T, FN>() * (8 + (int)sizeof(T)) + BIG_HIST * 4;
  const int tile = FILL_WARP_SORT * 8;
  return ((word > tile ? word : tile) + 15) & ~15;
}

// ascending bitonic sort of k[0..np) with np = next power of two >= n
// (padded with ~0), carrying v along
template <typename T>
__device__ __forceinline__ void warp_sort_keys(unsigned long long* k, T* v, int n) {
  int np = 1;
  while (np < n) np <<= 1;
  const int lane = threadIdx.x & 31;
  for (int i = n + lane; i < np; i += 32) k[i] = ~0ull;
  __syncwarp();
  for (int kk = 2; kk <= np; kk <<= 1) {
    for (int j = kk >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < np; i += 32) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long x = k[i], y = k[ixj];
          const bool up = (i & kk) == 0;
          if ((x > y) == up) {
            k[i] = y;
            k[ixj] = x;
            const T t = v[i];
            v[i] = v[ixj];
            v[ixj] = t;
          }
        }
      }
      __syncwarp();
    }
  }
}

// Fold keys[0..m) (part << 33 | dedup << 32 | mask, part order) into this
// lane's pixel, 32 records at a time.
template <typename T, int FN, bool DEDUP>
__device__ __forceinline__ void fold_sorted(const unsigned long long* keys, const T* vals, int m, T& c,
                                            unsigned& last, T bg, const BgF64& bgc) {
  const int lane = threadIdx.x & 31;
  for (int j0 = 0; j0 < m; j0 += 32) {
    const bool in = j0 + lane < m;
    const unsigned long long k = in ? keys[j0 + lane] : 0ull;
    const T v = in ? vals[j0 + lane] : T(0);
    const unsigned x = (unsigned)(k >> 33) | ((unsigned)(k >> 32) & 1u) << 31;
    fold_bits<T, FN, DEDUP>(warp_transpose32((unsigned)k), v, x, false, c, last, bg, bgc);
  }
}

// Fold the n <= 256 records of one word into this lane's pixel, their places
// sorted in registers; false when their parts are too far apart for that.
// (16 road networks: 0.61 ms with every word sorted in shared memory, 0.41 so.)
template <typename T, int FN, bool DEDUP>
__device__ __noinline__ bool sorted_word(const FillArgs& a, const uint2* recs, int n, unsigned char* spos, T& c, T bg,
                                         const BgF64& bgc) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  if (!(n <= 128 ? sort_positions<4>(recs, n, spos) : sort_positions<8>(recs, n, spos))) return false;
  __syncwarp();
  unsigned last = 0xFFFFFFFFu;
  for (int i0 = 0; i0 < n; i0 += 32) {
    uint2 r = make_uint2(0u, 0u);
    T v = T(0);
    if (i0 + lane < n) {
      r = recs[(unsigned)spos[i0 + lane] & (n <= 128 ? 0x7Fu : 0xFFu)];
      v = rec_value<T>(a, r.x);
    }
    fold_bits<T, FN, DEDUP>(warp_transpose32(r.y), v, r.x & (REC_PART_MASK | DEDUP_BIT), false, c, last, bg, bgc);
  }
  return true;
}

// The parts of this lane's records i0 + lane, + 32, + 64, + 96 of a word (past
// the end: no part).  Four loads in flight: a word's records are looked through
// three times per big_cap() of them, one load's latency at a time else (50,000
// records in every word of some tiles 79 ms, 56 so).
__device__ __forceinline__ void load_parts(const uint2* recs, int n, int i0, unsigned (&p)[4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 4; ++k) p[k] = i0 + k * 32 + lane < n ? recs[i0 + k * 32 + lane].x & REC_PART_MASK : ~0u;
}

// Fold the n records of one word; x: this lane's pixel in the tile.
template <typename T, int FN, bool DEDUP>
__device__ __forceinline__ void big_word(const FillArgs& a, const uint2* recs, int n, T* dst, int x, int len,
                                         unsigned char* wbase, T bg, const BgF64& bgc) {
  constexpr int CAP = big_cap<T, FN>();
  const int lane = threadIdx.x & 31;
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(wbase);
  T* vals = reinterpret_cast<T*>(wbase + CAP * 8);
  unsigned* hist = reinterpret_cast<unsigned*>(wbase + CAP * 8 + CAP * sizeof(T));
  if constexpr (FN == F_FIRST || FN == F_LAST) {  // order-free: one pass, no sort
    unsigned maxp1 = 0u, ming = 0xFFFFFFFFu;
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      unsigned kx = 0u, km = 0u;
      if (i < n) {
        const uint2 r = recs[i];
        kx = of_key<T, FN>(r.x, FN == F_FIRST ? rec_value<T>(a, r.x) : T(0), bg, bgc);
        km = r.y;
      }
      const int cnt = min(32, n - i0);
      for (int j = 0; j < cnt; ++j) {
        const unsigned xj = __shfl_sync(0xFFFFFFFFu, kx, j), mj = __shfl_sync(0xFFFFFFFFu, km, j);
        if ((mj >> lane) & 1u) of_update<FN>(maxp1, ming, xj);
      }
    }
    if (x < len) dst[x] = of_result<T, FN>(a, maxp1, ming, bg);
    return;
  }
  if constexpr (FN == F_MIN || FN == F_MAX) {  // order-free unless a value resets the pixel
    T bv = bg;
    unsigned bp = 0xFFFFFFFFu;
    bool bad = false;
    for (int i0 = 0; i0 < n; i0 += 32) {
      const int i = i0 + lane;
      unsigned kx = 0u, km = 0u;
      T kv = T(0);
      if (i < n) {
        const uint2 r = recs[i];
        kv = rec_value<T>(a, r.x);
        kx = r.x;
        km = r.y;
        bad = bad || first_resets<T>(kv, bg, bgc);
      }
      if (__any_sync(0xFFFFFFFFu, bad)) break;
      const int cnt = min(32, n - i0);
      for (int j = 0; j < cnt; ++j) {
        const unsigned xj = __shfl_sync(0xFFFFFFFFu, kx, j), mj = __shfl_sync(0xFFFFFFFFu, km, j);
        const T vj = shfl_val<T>(kv, j);
        if ((mj >> lane) & 1u) {
          const unsigned pj = xj & REC_PART_MASK;
          if (of_better<T, FN>(vj, pj, bv, bp)) {
            bv = vj;
            bp = pj;
          }
        }
      }
    }
    if (!__any_sync(0xFFFFFFFFu, bad)) {
      if (x < len) dst[x] = bv;
      return;
    }
  }
  T c = bg;
  unsigned last_part = 0xFFFFFFFFu;
  unsigned lo_part = 0;  // parts < lo_part are done
  bool done = false;
  if (n <= 256) done = sorted_word<T, FN, DEDUP>(a, recs, n, wbase, c, bg, bgc);
  while (!done) {
    unsigned cnt = 0, pmin = 0xFFFFFFFFu, pmax = 0;
    for (int i0 = 0; i0 < n; i0 += 128) {
      unsigned p[4];
      load_parts(recs, n, i0, p);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p[k] >= lo_part && p[k] <= REC_PART_MASK) {
          ++cnt;
          pmin = min(pmin, p[k]);
          pmax = max(pmax, p[k]);
        }
    }
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    if (cnt == 0) break;
    pmin = __reduce_min_sync(0xFFFFFFFFu, pmin);
    pmax = __reduce_max_sync(0xFFFFFFFFu, pmax);
    unsigned hi = pmax + 1;  // parts [lo_part, hi) this round
    bool single = false;
    if (cnt > (unsigned)CAP) {
      unsigned span_lo = pmin, span_hi = pmax;  // inclusive
      while (true) {
        int shift = 0;
        while (((span_hi - span_lo) >> shift) >= (unsigned)BIG_HIST) ++shift;
        for (int h = lane; h < BIG_HIST; h += 32) hist[h] = 0u;
        __syncwarp();
        for (int i0 = 0; i0 < n; i0 += 128) {
          unsigned p[4];
          load_parts(recs, n, i0, p);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (p[k] >= span_lo && p[k] <= span_hi) atomicAdd(&hist[(p[k] - span_lo) >> shift], 1u);
        }
        __syncwarp();
        // largest prefix of bins with at most CAP records (lane 0)
        int jsel = -1;
        if (lane == 0) {
          unsigned cum = 0;
          for (int h = 0; h < BIG_HIST; ++h) {
            if (cum + hist[h] > (unsigned)CAP) break;
            cum += hist[h];
            jsel = h;
          }
        }
        jsel = __shfl_sync(0xFFFFFFFFu, jsel, 0);
        __syncwarp();
        if (jsel >= 0) {
          hi = span_lo + ((unsigned)(jsel + 1) << shift);
          break;
        }
        if (shift == 0) {  // one part alone exceeds CAP
          hi = span_lo + 1;
          single = true;
          break;
        }
        span_hi = span_lo + (1u << shift) - 1u;  // zoom into the first bin
      }
    }
    // gather [lo_part, hi) of this word (chunks of CAP for a single part)
    int m = 0;
    for (int b0 = 0; b0 < n; b0 += 128) {
      uint2 rs[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) rs[k] = b0 + k * 32 + lane < n ? recs[b0 + k * 32 + lane] : make_uint2(0u, 0u);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint2 r = rs[k];
        const unsigned part = r.x & REC_PART_MASK;
        const bool take = b0 + k * 32 + lane < n && part >= lo_part && part < hi;
        const unsigned mk = __ballot_sync(0xFFFFFFFFu, take);
        if (take) {
          const int pos = m + __popc(mk & ((1u << lane) - 1u));
          // part (order), then the DEDUP flag, then the mask
          keys[pos] = ((unsigned long long)part << 33) | ((unsigned long long)(r.x >> 31) << 32) | r.y;
          vals[pos] = rec_value<T>(a, r.x);
        }
        m += __popc(mk);
        if (single && m > CAP - 32) {  // fold a chunk of the single part
          __syncwarp();
          fold_sorted<T, FN, DEDUP>(keys, vals, m, c, last_part, bg, bgc);
          m = 0;
          __syncwarp();
        }
      }
    }
    __syncwarp();
    if (!single) warp_sort_keys(keys, vals, m);
    __syncwarp();
    fold_sorted<T, FN, DEDUP>(keys, vals, m, c, last_part, bg, bgc);
    __syncwarp();
    lo_part = hi;
  }
  if (x < len) dst[x] = c;
}

template <typename T, int FN, bool DEDUP>
__global__ void __launch_bounds__(BIG_WARPS * 32, big_takes_shallow<T, FN>() ? 3 : sizeof(T) <= 4 ? 2 : 0) k_fill_big(FillArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned s_cnt[WPT], s_pos[WPT];
  const Ctrl* ctrl = a.ctrl;
  if (block_skips(ctrl->err || ctrl->span_count > a.rec_cap)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* wbase = smem + warp * big_warp_bytes<T, FN>();
  const T bg = from_bits<T>(a.bg);
  const BgF64 bgc = bg_f64(a.bg);
  const unsigned nbig = *a.nbig;
  if constexpr (big_takes_shallow<T, FN>())
    shallow_tiles<T, FN, DEDUP>(a, blockIdx.x * BIG_WARPS + warp, gridDim.x * BIG_WARPS, wbase, bg, bgc);
  for (unsigned it = blockIdx.x; it < nbig; it += gridDim.x) {
    const unsigned b = a.big[it], o0 = a.offsets[b];
    const int n = (int)(a.offsets[b + 1] - o0);
    __syncthreads();  // the last bucket's words are done
    if (threadIdx.x < WPT) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    for (int place = 0; place < 2; ++place) {
      for (int i0 = warp * 32; i0 < n; i0 += BIG_WARPS * 32) {
        const int i = i0 + lane;
        uint2 r = make_uint2(0u, 0u);
        if (i < n) r = a.recs[o0 + i];
        const unsigned w = i < n ? (r.x >> REC_W_SHIFT) & 15u : 0xFFu;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, w);
        const int leader = __ffs(peers) - 1;
        unsigned base = 0;
        if (lane == leader && i < n) base = atomicAdd(place ? &s_pos[w] : &s_cnt[w], (unsigned)__popc(peers));
        base = __shfl_sync(0xFFFFFFFFu, base, leader);
        if (place && i < n) a.brecs[o0 + base + __popc(peers & ((1u << lane) - 1u))] = r;
      }
      __syncthreads();
      if (place == 0) {
        if (threadIdx.x < WPT) {
          unsigned before = 0;
          for (unsigned w = 0; w < threadIdx.x; ++w) before += s_cnt[w];
          s_pos[threadIdx.x] = before;
        }
        __syncthreads();
      }
    }
    int len;
    T* dst = bucket_tile<T>(a, b, len);
    // every word's cursor has moved to its end
    const int nw = (int)s_cnt[warp];
    big_word<T, FN, DEDUP>(a, a.brecs + o0 + s_pos[warp] - nw, nw, dst, warp * 32 + lane, len, wbase, bg, bgc);
  }
}

// ---- order-free fill: count / any --------------------------------------
// Integer `count` with background 0 (and float count with background 0 or
// NaN) equals the pixel's coverage depth: every write after the first adds
// one and no intermediate count can equal the background.  `any` is 1
// wherever the depth is non-zero.  Neither needs values or order.  One warp
// per bucket (FILL_CHUNK consecutive buckets per task, the next bucket's records
// loaded while the current one is counted); every record is broadcast to the
// warp and lane l adds its bit l to the counter of the record's word.
constexpr int DEPTH_WARPS = 8;

// `any`: the words' masks are joined in shared memory and expanded to values,
// 16 bytes a lane.  (One value per lane and word, as k_fill_depth writes
// them, took 2.8 ms for 16 uint8 bands of 20,000 x 20,000 pixels; so it takes
// 1.37 at six blocks per SM, 1.43 with the registers left to the compiler,
// 1.66 at eight.)
template <typename T>
__global__ void __launch_bounds__(DEPTH_WARPS * 32, 6) k_fill_any(FillArgs a) {
  __shared__ unsigned s_cov[DEPTH_WARPS][WPT + 1];
  Ctrl* ctrl = a.ctrl;
  if (ctrl->err || ctrl->span_count > a.rec_cap) return;
  const int lane = threadIdx.x & 31;
  unsigned* cov = s_cov[threadIdx.x >> 5];
  const T bg = from_bits<T>(a.bg);
  if (lane <= WPT) cov[lane] = 0u;
  __syncwarp();
  TileIter<T> it;
  while (true) {
    unsigned long long b0 = 0;
    if (lane == 0) b0 = atomicAdd(a.work, (unsigned long long)a.chunk);
    b0 = __shfl_sync(0xFFFFFFFFu, b0, 0);
    if (b0 >= a.nbuckets) break;
    const int nb = (int)min((unsigned long long)a.chunk, a.nbuckets - b0);
    it.init(a, a.bucket0 + b0);
    const unsigned off = a.offsets[b0 + (lane < nb ? lane : nb)];
    const unsigned off_end = a.offsets[b0 + nb];
    unsigned o_next = __shfl_sync(0xFFFFFFFFu, off, 0);
    unsigned e_next = nb > 1 ? __shfl_sync(0xFFFFFFFFu, off, 1) : off_end;
    uint2 nxt = lane < (int)(e_next - o_next) ? a.recs[o_next + lane] : make_uint2(0u, 0u);
    for (int k = 0; k < nb; ++k) {
      const unsigned o0 = o_next, n = e_next - o_next;
      uint2 r = nxt;
      if (k + 1 < nb) {
        o_next = __shfl_sync(0xFFFFFFFFu, off, k + 1);
        e_next = k + 2 < nb ? __shfl_sync(0xFFFFFFFFu, off, (k + 2) & 31) : off_end;
        nxt = lane < (int)(e_next - o_next) ? a.recs[o_next + lane] : make_uint2(0u, 0u);
      }
      int len;
      T* dst = it.tile(a, len);
      it.next(a);
      if (n == 0) {
        store_bg<T>(dst, len, a.bg16, bg);
        continue;
      }
      for (unsigned i0 = 0; i0 < n; i0 += 32) {
        if (i0 > 0) r = i0 + lane < n ? a.recs[o0 + i0 + lane] : make_uint2(0u, 0u);
        if (r.y) atomicOr(&cov[(r.x >> REC_W_SHIFT) & 15u], r.y);
      }
      __syncwarp();
      constexpr int E = 16 / (int)sizeof(T);
      store_values<T>(
          dst, len, [&](int i) { return (cov[i >> 5] >> (i & 31)) & 1u ? T(1) : bg; },
          [&](int i) {
            const unsigned bits = __funnelshift_r(cov[i >> 5], cov[(i >> 5) + 1], i & 31);
            return expand_any<T>(bits & ((1u << E) - 1u), a.bg16, T(1));
          });
      __syncwarp();
      if (lane < WPT) cov[lane] = 0u;
      __syncwarp();
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(DEPTH_WARPS * 32) k_fill_depth(FillArgs a) {
  Ctrl* ctrl = a.ctrl;
  if (ctrl->err || ctrl->span_count > a.rec_cap) return;
  const int lane = threadIdx.x & 31;
  const T bg = from_bits<T>(a.bg);
  TileIter<T> it;
  while (true) {
    unsigned long long b0 = 0;
    if (lane == 0) b0 = atomicAdd(a.work, (unsigned long long)a.chunk);
    b0 = __shfl_sync(0xFFFFFFFFu, b0, 0);
    if (b0 >= a.nbuckets) break;
    const int nb = (int)min((unsigned long long)a.chunk, a.nbuckets - b0);
    it.init(a, a.bucket0 + b0);
    const unsigned off = a.offsets[b0 + (lane < nb ? lane : nb)];
    const unsigned off_end = a.offsets[b0 + nb];
    unsigned o_next = __shfl_sync(0xFFFFFFFFu, off, 0);
    unsigned e_next = nb > 1 ? __shfl_sync(0xFFFFFFFFu, off, 1) : off_end;
    uint2 nxt = lane < (int)(e_next - o_next) ? a.recs[o_next + lane] : make_uint2(0u, 0u);
    for (int k = 0; k < nb; ++k) {
      const unsigned o0 = o_next, o1 = e_next;
      const int n = (int)(o1 - o0);
      uint2 r = nxt;
      if (k + 1 < nb) {
        o_next = __shfl_sync(0xFFFFFFFFu, off, k + 1);
        e_next = k + 2 < nb ? __shfl_sync(0xFFFFFFFFu, off, (k + 2) & 31) : off_end;
        nxt = lane < (int)(e_next - o_next) ? a.recs[o_next + lane] : make_uint2(0u, 0u);
      }
      int len;
      T* dst = it.tile(a, len);
      it.next(a);
      if (n == 0) {
        store_bg<T>(dst, len, a.bg16, bg);
        continue;
      }
      // 32 records at a time, bit-sliced: after the transpose lane l holds
      // bit l of every record's mask, so the depth of pixel (w, l) grows by
      // the records of word w among those bits (lanes past the end hold an
      // empty mask and add nothing)
      unsigned c[WPT];
#pragma unroll
      for (int w = 0; w < WPT; ++w) c[w] = 0u;
      for (int i0 = 0; i0 < n; i0 += 32) {
        if (i0 > 0) r = i0 + lane < n ? a.recs[o0 + i0 + lane] : make_uint2(0u, 0u);
        const unsigned wd = (r.x >> REC_W_SHIFT) & 15u;
        const unsigned t = warp_transpose32(r.y);
#pragma unroll
        for (int w = 0; w < WPT; ++w) c[w] += (unsigned)__popc(t & __ballot_sync(0xFFFFFFFFu, wd == (unsigned)w));
      }
      auto value = [&](unsigned d) {
        if (!d) return bg;
        if constexpr (std::is_integral<T>::value) return (T)(typename std::make_unsigned<T>::type)d;
        else return (T)d;
      };
      if constexpr (sizeof(T) < 4) {  // a lane's single values are narrow: staged, then 16 bytes a lane
        __shared__ __align__(16) T s_seg[DEPTH_WARPS][TW];
        T* seg = s_seg[threadIdx.x >> 5];
#pragma unroll
        for (int w = 0; w < WPT; ++w) seg[w * 32 + lane] = value(c[w]);
        __syncwarp();
        store_values<T>(
            dst, len, [&](int i) { return seg[i]; },
            [&](int i) {
              constexpr int E = 16 / (int)sizeof(T);
              uint4 q;
              T v[E];
#pragma unroll
              for (int e = 0; e < E; ++e) v[e] = seg[i + e];
              memcpy(&q, v, 16);
              return q;
            });
        __syncwarp();
      } else {
#pragma unroll
        for (int w = 0; w < WPT; ++w)
          if (w * 32 + lane < len) dst[w * 32 + lane] = value(c[w]);
      }
    }
  }
}

// Host launcher shared by the per-dtype translation units.
template <typename T>
bool depth_exact(const FillArgs& a, int fn, bool dedup) {
  if (fn == F_ANY) return true;
  if (fn != F_COUNT || dedup) return false;
  const T bg = from_bits_host<T>(a.bg);
  if constexpr (std::is_integral<T>::value) return bg == T(0);
  else return bg == T(0) || bg != bg;
}

// Blocks of a fill kernel that one SM holds with `smem` bytes of dynamic
// shared memory (at most `smem_max`, which is allowed once).  Asked of the
// driver once per device and size: the two queries cost a small call 5 us.
template <auto Kern>
int fill_occupancy(int threads, int smem, int smem_max) {
  static std::atomic<unsigned> known[64];
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<unsigned>& slot = known[dev & 63];
  const unsigned c = slot.load(std::memory_order_relaxed);
  if (dev < 64 && c && (int)(c >> 8) == smem) return (int)(c & 255u);
  if (smem_max) cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
  int bps = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, Kern, threads, smem);
  if (bps < 1) bps = 1;
  slot.store((unsigned)smem << 8 | (unsigned)bps, std::memory_order_relaxed);
  return bps;
}

template <typename T>
int launch_fill_t(const FillArgs& a, int fn, bool dedup, int num_sms, cudaStream_t s) {
  // persistent grids: as many blocks as fit on the GPU at once, chunks of
  // buckets handed out by an atomic counter.  About 32 grabs a warp:
  // fewer leave warps idle at the end (the large fill's 800,000 buckets),
  // more make the counter the bottleneck (12.8 M buckets, 4 at a time).  A
  // fill of few buckets gives every warp one at a time.
  auto persistent = [&](FillArgs& w, int bps, int per_block_units) {
    unsigned long long g = (unsigned long long)num_sms * bps;
    const unsigned long long grabs = a.nbuckets / (g * per_block_units * 32);
    const int least = a.nbuckets < g * per_block_units * FILL_CHUNK ? 1 : FILL_CHUNK;
    w.chunk = (int)(grabs < (unsigned)least ? least : grabs > FILL_CHUNK_MAX ? FILL_CHUNK_MAX : grabs);
    const unsigned long long units = (unsigned long long)per_block_units * w.chunk;
    const unsigned long long want = (a.nbuckets + units - 1) / units;
    if (want < g) g = want;
    return (unsigned)(g ? g : 1);
  };
  if (depth_exact<T>(a, fn, dedup)) {
    FillArgs aw = a;
    if (fn == F_ANY) {
      const unsigned grid = persistent(aw, fill_occupancy<k_fill_any<T>>(DEPTH_WARPS * 32, 0, 0), DEPTH_WARPS);
      k_fill_any<T><<<grid, DEPTH_WARPS * 32, 0, s>>>(aw);
    } else {
      const unsigned grid = persistent(aw, fill_occupancy<k_fill_depth<T>>(DEPTH_WARPS * 32, 0, 0), DEPTH_WARPS);
      k_fill_depth<T><<<grid, DEPTH_WARPS * 32, 0, s>>>(aw);
    }
    return 1;
  }
  int launches = 0;
#define RZ_FILL_CASE(FNV, DD)                                                                             \
  {                                                                                                       \
    FillArgs aw = a;                                                                                      \
    aw.sort_cap = fill_sort_cap(a.sort_max);                                                              \
    aw.warp_bytes = fill_warp_bytes<T>(FNV, aw.sort_cap);                                                 \
    constexpr int W = FILL_WARPS_PER_BLOCK;                                                               \
    const int ws = W * aw.warp_bytes, wmax = W * fill_warp_bytes<T>(FNV, FILL_WARP_SORT);                 \
    constexpr int bs = BIG_WARPS * big_warp_bytes<T, FNV>();                                                   \
    const int wbps = fill_occupancy<k_fill_warp<T, FNV, DD>>(W * 32, ws, wmax);                           \
    const int bbps = fill_occupancy<k_fill_big<T, FNV, DD>>(BIG_WARPS * 32, bs, bs);                      \
    const unsigned grid = persistent(aw, wbps, W);                                                        \
    k_fill_warp<T, FNV, DD><<<grid, W * 32, ws, s>>>(aw);                                                 \
    const unsigned long long bg = (unsigned long long)num_sms * bbps;                                     \
    k_fill_big<T, FNV, DD><<<(unsigned)(bg < a.nbuckets ? bg : a.nbuckets), BIG_WARPS * 32, bs, s>>>(aw); \
    launches += 2;                                                                                        \
  }
  switch (fn) {
    case F_SUM:
      if (dedup) RZ_FILL_CASE(F_SUM, true) else RZ_FILL_CASE(F_SUM, false)
      break;
    case F_FIRST: RZ_FILL_CASE(F_FIRST, false) break;
    case F_LAST: RZ_FILL_CASE(F_LAST, false) break;
    case F_MIN: RZ_FILL_CASE(F_MIN, false) break;
    case F_MAX: RZ_FILL_CASE(F_MAX, false) break;
    case F_COUNT:
      if (dedup) RZ_FILL_CASE(F_COUNT, true) else RZ_FILL_CASE(F_COUNT, false)
      break;
    default: break;  // any: depth_exact
  }
#undef RZ_FILL_CASE
  return launches;
}

}  // namespace rzd

#define RZ_DECLARE_FILL(NAME) \
  int NAME(const rzd::FillArgs& a, int fn, bool dedup, int num_sms, cudaStream_t s);
RZ_DECLARE_FILL(rz_fill_u8)
RZ_DECLARE_FILL(rz_fill_u16)
RZ_DECLARE_FILL(rz_fill_u32)
RZ_DECLARE_FILL(rz_fill_u64)
RZ_DECLARE_FILL(rz_fill_i8)
RZ_DECLARE_FILL(rz_fill_i16)
RZ_DECLARE_FILL(rz_fill_i32)
RZ_DECLARE_FILL(rz_fill_i64)
RZ_DECLARE_FILL(rz_fill_f32)
RZ_DECLARE_FILL(rz_fill_f64)
