// rz_sparse.cuh -- the sparse (COO) encoding: coverage records ordered by
// (band, part, row, word) and expanded into (row, col, value) triplets, one
// per written pixel (SparseArrayWriter, rust/src/encoding/writers.rs:86-131).
#pragma once

#include <type_traits>

#include "rz_device.cuh"

namespace rzd {

// sort keys of the parts by band (part order kept within a band)
__global__ void k_part_band_keys(const PartPlan* __restrict__ plan, unsigned long long P, unsigned long long* keys,
                                 unsigned* vals) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < P; p += stride) {
    keys[p] = ((unsigned long long)plan[p].band << 32) | p;
    vals[p] = (unsigned)p;
  }
}

__global__ void k_part_rank(const unsigned* __restrict__ sorted_parts, unsigned long long P, unsigned* prank) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < P; i += stride)
    prank[sorted_parts[i]] = (unsigned)i;
}

// key = band-major part rank << word_bits | word id within the band's raster
__global__ void k_rec_keys(RecBuf rb, unsigned long long n, const unsigned* __restrict__ prank,
                           const PartPlan* __restrict__ plan, int word_bits, unsigned long long* keys,
                           unsigned* vals) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    const unsigned part = rb.part[i] & REC_PART_MASK;
    const unsigned pr = prank ? prank[part] : part;
    keys[i] = ((unsigned long long)pr << word_bits) | (rb.wid[i] - plan[part].wid0);
    vals[i] = (unsigned)i;
  }
}

// pixels each ordered record writes: a deduplicating part writes a pixel of
// a word once (its records of one word are adjacent in the order)
__global__ void k_sparse_count(const unsigned long long* __restrict__ skeys, const unsigned* __restrict__ svals,
                               unsigned long long n, RecBuf rb, unsigned* eff, unsigned long long* counts) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    const unsigned rec = svals[i];
    unsigned m = rb.mask[rec];
    if (rb.part[rec] & DEDUP_BIT) {
      unsigned before = 0u;
      for (unsigned long long j = i; j > 0 && skeys[j - 1] == skeys[i]; --j) before |= rb.mask[svals[j - 1]];
      m &= ~before;
    }
    eff[i] = m;
    counts[i] = (unsigned long long)__popc(m);
  }
}

// The n-th set bit of m (n < popc(m)).
__device__ __forceinline__ unsigned nth_bit(unsigned m, unsigned n) {
  unsigned at = 0;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const unsigned c = (unsigned)__popc((m >> at) & ((1u << w) - 1u));
    if (n >= c) {
      n -= c;
      at += w;
    }
  }
  return at;
}

// The triplets of 32 records at a time: each lane finds the record and pixel
// of its own output place, so that rows, columns and values leave in runs of
// 32.  (A thread per record, writing its up to 32 triplets one after the
// other and counting each record on its band's one counter, took 1.1 ms for
// 20 M triplets.)
template <int VB>
__global__ void __launch_bounds__(256) k_sparse_emit(
    const unsigned long long* __restrict__ skeys, const unsigned* __restrict__ svals, unsigned long long n, RecBuf rb,
    const unsigned* __restrict__ eff, const unsigned long long* __restrict__ offsets,
    const PartPlan* __restrict__ plan, const void* __restrict__ values, const unsigned* __restrict__ part_geom,
    unsigned long long scalar_bits, int word_bits, unsigned long long* rows, unsigned long long* cols, void* tvals,
    unsigned long long* band_counts) {
  using V = typename std::conditional<VB == 1, unsigned char,
            typename std::conditional<VB == 2, unsigned short,
            typename std::conditional<VB == 4, unsigned, unsigned long long>::type>::type>::type;
  const unsigned lane = threadIdx.x & 31;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i0 = blockIdx.x * (unsigned long long)blockDim.x + (threadIdx.x & ~31u); i0 < n;
       i0 += stride) {
    const unsigned long long i = i0 + lane;
    unsigned m = 0, y = 0, x0 = 0, band = 0;
    V v = 0;
    if (i < n) {
      m = eff[i];
      const unsigned part = rb.part[svals[i]] & REC_PART_MASK;
      const unsigned lwid = (unsigned)(skeys[i] & ((1ull << word_bits) - 1ull));
      const unsigned wpr = plan[part].wpr;
      y = lwid / wpr;
      x0 = (lwid - y * wpr) * 32u;
      band = plan[part].band;
      v = values ? static_cast<const V*>(values)[part_geom[part]] : (V)scalar_bits;
    }
    const unsigned long long out0 = offsets[i0];
    unsigned incl = (unsigned)__popc(m);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= (unsigned)o) incl += t;
    }
    const unsigned excl = incl - (unsigned)__popc(m), total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    {  // one count per band among the records (they are ordered by band)
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, band);
      const unsigned c = __reduce_add_sync(peers, (unsigned)__popc(m));
      if (c && lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(&band_counts[band], (unsigned long long)c);
    }
    for (unsigned t0 = 0; t0 < total; t0 += 32) {
      // the record of place t0 + lane: the last non-empty one that starts at or before it
      const unsigned start = m && excl >= t0 && excl < t0 + 32 ? 1u << (excl - t0) : 0u;
      const unsigned starts = __reduce_or_sync(0xFFFFFFFFu, start);
      const unsigned full = __ballot_sync(0xFFFFFFFFu, m != 0u);
      const unsigned before = (unsigned)__popc(__ballot_sync(0xFFFFFFFFu, m != 0u && excl < t0));
      const unsigned q = before + (unsigned)__popc(starts & ((2u << lane) - 1u)) - 1u;  // among the non-empty ones
      const unsigned src = nth_bit(full, q) & 31u;
      const unsigned ms = __shfl_sync(0xFFFFFFFFu, m, src), es = __shfl_sync(0xFFFFFFFFu, excl, src);
      const unsigned ys = __shfl_sync(0xFFFFFFFFu, y, src), xs = __shfl_sync(0xFFFFFFFFu, x0, src);
      V vs;
      if constexpr (VB == 8) vs = (V)__shfl_sync(0xFFFFFFFFu, (unsigned long long)v, src);
      else vs = (V)__shfl_sync(0xFFFFFFFFu, (unsigned)v, src);
      const unsigned t = t0 + lane;
      if (t < total) {
        const unsigned long long pos = out0 + t;
        rows[pos] = ys;
        cols[pos] = xs + nth_bit(ms, t - es);
        static_cast<V*>(tvals)[pos] = vs;
      }
    }
  }
}

// ---- replay of a triplet stream (SparseArray::build_array) ----

// Key of every triplet of a chunk: the band comes from the band start
// offsets (bstart[b] <= t < bstart[b + 1] for stream index t), rows and
// columns are checked against the raster (the reference indexes the array and
// panics outside it; here the first bad stream index is reported).
template <typename K>
__global__ void k_replay_keys(const unsigned long long* __restrict__ rows, const unsigned long long* __restrict__ cols,
                              unsigned n, unsigned long long t0, const unsigned long long* __restrict__ bstart,
                              unsigned n_bands, unsigned long long nrows, unsigned long long ncols,
                              K* keys, unsigned* idx, Ctrl* ctrl) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned long long t = t0 + i;
    unsigned lo = 0, hi = n_bands - 1;  // the last band whose start is <= t
    while (lo < hi) {
      const unsigned mid = lo + (hi - lo + 1) / 2;
      if (bstart[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const unsigned long long r = rows[i], c = cols[i];
    unsigned long long key = 0;
    if (r < nrows && c < ncols) key = ((unsigned long long)lo * nrows + r) * ncols + c;
    else set_error(ctrl, ERR_TRIPLET, t);
    keys[i] = (K)key;
    idx[i] = i;
  }
}

// Background of a raster of n elements of VB bytes.
template <int VB>
__global__ void k_replay_bg(void* p, unsigned long long n, unsigned long long bg) {
  using U = typename std::conditional<VB == 1, unsigned char,
            typename std::conditional<VB == 2, unsigned short,
            typename std::conditional<VB == 4, unsigned, unsigned long long>::type>::type>::type;
  U* q = static_cast<U*>(p);
  const U v = (U)bg;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x)
    q[i] = v;
}

}  // namespace rzd
