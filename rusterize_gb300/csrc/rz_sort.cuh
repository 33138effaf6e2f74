// rz_sort.cuh -- stable least-significant-digit radix sort of (32- or 64-bit
// key, 32-bit value) pairs, up to 9 bits per pass: a per-tile digit histogram, one
// exclusive scan of the digit-major histogram table, and a scatter that
// orders its tile by digit in shared memory first, so that each digit's
// elements leave in runs.
//
// What bounds it: memory traffic, 24 B read and written per element and pass
// and 8 B read for the histogram.  With tiles of 1,024 elements written
// straight from their threads (four elements of a digit at a time) and 8 bits
// a pass, 23 M pixel keys of 25 bits took four passes of 330 + 64 us.
#pragma once

#include <cuda_runtime.h>

#include "rz_scan.cuh"

namespace rzd {

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 16;  // elements per thread
constexpr unsigned RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_MAX_BITS = 9;
constexpr int RS_BINS = 1 << RS_MAX_BITS;

template <typename K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const K* __restrict__ keys, unsigned n,
                                                         int shift, int bits, unsigned* __restrict__ hist,
                                                         unsigned nblocks) {
  __shared__ unsigned s_h[RS_BINS];
  const unsigned bins = 1u << bits;
  for (unsigned d = threadIdx.x; d < bins; d += RS_THREADS) s_h[d] = 0u;
  __syncthreads();
  const unsigned base = blockIdx.x * RS_TILE;
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const unsigned e = base + r * RS_THREADS + threadIdx.x;
    if (e < n) atomicAdd(&s_h[(unsigned)(keys[e] >> shift) & (bins - 1u)], 1u);
  }
  __syncthreads();
  for (unsigned d = threadIdx.x; d < bins; d += RS_THREADS) hist[d * nblocks + blockIdx.x] = s_h[d];
}

// Shared memory of k_rs_scatter: the tile's keys and values, and per-warp
// digit counts.
template <typename K>
constexpr int rs_scatter_smem() { return (int)RS_TILE * (4 + (int)sizeof(K)) + RS_WARPS * RS_BINS * 2; }

template <typename K>
__global__ void __launch_bounds__(RS_THREADS, 3) k_rs_scatter(const K* __restrict__ kin,
                                                            const unsigned* __restrict__ vin, K* __restrict__ kout,
                                                            unsigned* __restrict__ vout, unsigned n, int shift,
                                                            int bits, const unsigned* __restrict__ off,
                                                            unsigned nblocks) {
  extern __shared__ __align__(16) unsigned char smem[];
  K* s_k = reinterpret_cast<K*>(smem);
  unsigned* s_v = reinterpret_cast<unsigned*>(s_k + RS_TILE);
  unsigned short* s_w = reinterpret_cast<unsigned short*>(s_v + RS_TILE);  // [warp][digit]: counts, then prefixes
  __shared__ unsigned s_first[RS_BINS];  // the tile's first position of each digit
  __shared__ unsigned s_glob[RS_BINS];   // global position of that element, minus the tile's
  __shared__ unsigned s_tot[RS_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u, bins = 1u << bits;
  for (unsigned i = threadIdx.x; i < RS_WARPS * RS_BINS / 2; i += RS_THREADS) reinterpret_cast<unsigned*>(s_w)[i] = 0u;
  __syncthreads();
  // warp w takes elements [512 w, 512 (w + 1)) of the tile in order: an
  // element's rank is the number of equal digits before it in its warp
  const unsigned base = blockIdx.x * RS_TILE + warp * (32 * RS_ITEMS);
  K k[RS_ITEMS];
  unsigned v[RS_ITEMS];
  unsigned short rank[RS_ITEMS];
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const unsigned e = base + r * 32 + lane;
    k[r] = e < n ? kin[e] : K(0);
    v[r] = e < n ? vin[e] : 0u;
  }
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const bool valid = base + r * 32 + lane < n;
    const unsigned d = (unsigned)(k[r] >> shift) & (bins - 1u);
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, valid ? d : RS_BINS + (unsigned)lane);
    unsigned short* cnt = &s_w[warp * RS_BINS + d];
    const unsigned before = valid ? *cnt : 0u;
    rank[r] = (unsigned short)(before + __popc(peers & lt));
    __syncwarp();
    if (valid && (peers & lt) == 0u) *cnt = (unsigned short)(before + __popc(peers));
    __syncwarp();
  }
  __syncthreads();
  // per digit: exclusive prefix over the warps, then over the digits
  constexpr int PER = RS_BINS / RS_THREADS;
  unsigned tot[PER], sum = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const unsigned d = threadIdx.x * PER + j;
    unsigned acc = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      const unsigned c = s_w[w * RS_BINS + d];
      s_w[w * RS_BINS + d] = (unsigned short)acc;
      acc += c;
    }
    tot[j] = acc;
    sum += acc;
  }
  const unsigned incl = warp_inclusive_scan<unsigned>(sum);
  if (lane == 31) s_tot[warp] = incl;
  __syncthreads();
  unsigned first = incl - sum;
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) first += w < warp ? s_tot[w] : 0u;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const unsigned d = threadIdx.x * PER + j;
    s_first[d] = first;
    if (d < bins) s_glob[d] = off[d * nblocks + blockIdx.x] - first;
    first += tot[j];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    if (base + r * 32 + lane < n) {
      const unsigned d = (unsigned)(k[r] >> shift) & (bins - 1u);
      const unsigned at = s_first[d] + s_w[warp * RS_BINS + d] + rank[r];
      s_k[at] = k[r];
      s_v[at] = v[r];
    }
  }
  __syncthreads();
  const unsigned m = min(RS_TILE, n - blockIdx.x * RS_TILE);
  for (unsigned i = threadIdx.x; i < m; i += RS_THREADS) {
    const K key = s_k[i];
    const unsigned pos = s_glob[(unsigned)(key >> shift) & (bins - 1u)] + i;
    kout[pos] = key;
    vout[pos] = s_v[i];
  }
}

// Scratch (in 32-bit words) for radix_sort on n elements.
inline unsigned long long radix_sort_temp_words(unsigned long long n) {
  const unsigned long long nblocks = (n + RS_TILE - 1) / RS_TILE;
  const unsigned long long h = (unsigned long long)RS_BINS * (nblocks ? nblocks : 1);
  return 2 * h + 1 + scan_temp_elems(h);
}

// Sort keys[0..n) (bits [0, bits) significant) carrying vals; ktmp / vtmp are
// buffers of n elements.  Returns true when the sorted data ended up in
// ktmp / vtmp.  `launches` counts the kernels issued.
template <typename K>
bool radix_sort(K* keys, unsigned* vals, K* ktmp, unsigned* vtmp, unsigned n, int bits, unsigned* temp, cudaStream_t s,
                int& launches) {
  if (n == 0) return false;
  cudaFuncSetAttribute(k_rs_scatter<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, rs_scatter_smem<K>());
  const unsigned nblocks = (n + RS_TILE - 1) / RS_TILE;
  const int passes = (bits + RS_MAX_BITS - 1) / RS_MAX_BITS;
  bool in_tmp = false;
  for (int p = 0, shift = 0; p < passes; ++p) {
    const int w = (bits - shift + passes - p - 1) / (passes - p);  // the bits left, evenly over the passes left
    const unsigned long long h = (unsigned long long)nblocks << w;
    unsigned* hist = temp;
    unsigned* hoff = temp + h;
    unsigned* stmp = temp + 2 * h + 1;
    const K* kin = in_tmp ? ktmp : keys;
    const unsigned* vin = in_tmp ? vtmp : vals;
    k_rs_hist<K><<<nblocks, RS_THREADS, 0, s>>>(kin, n, shift, w, hist, nblocks);
    launches += 1 + scan<unsigned>(hist, hoff, h, stmp, s);
    k_rs_scatter<K><<<nblocks, RS_THREADS, rs_scatter_smem<K>(), s>>>(
        kin, vin, in_tmp ? keys : ktmp, in_tmp ? vals : vtmp, n, shift, w, hoff, nblocks);
    ++launches;
    in_tmp = !in_tmp;
    shift += w;
  }
  return in_tmp;
}

}  // namespace rzd
