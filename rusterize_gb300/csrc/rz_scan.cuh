// rz_scan.cuh -- exclusive prefix sums (reduce / scan / apply).  out has n+1
// elements; out[n] = total.
#pragma once

#include <cuda_runtime.h>

namespace rzd {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr unsigned long long SCAN_TILE = (unsigned long long)SCAN_THREADS * SCAN_ITEMS;

// A block covers SCAN_TILE elements; warp w of the block takes its SCAN_WROWS
// consecutive elements 32 at a time, so every load is one coalesced sweep,
// and a shuffle scan per group of 32 plus a running carry give the warp's
// prefixes.
constexpr int SCAN_WARPS = SCAN_THREADS / 32;
constexpr int SCAN_WROWS = (int)(SCAN_TILE / SCAN_WARPS);
constexpr int SCAN_GROUPS = SCAN_WROWS / 32;
// Up to this many blocks every apply block adds up the totals before it
// itself (16 KB of them at most), which saves the launch that scans them.
constexpr unsigned long long SCAN_FOLD_BLOCKS = 4096;

template <typename T>
__device__ __forceinline__ T warp_inclusive_scan(T x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += t;
  }
  return x;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xFFFFFFFFu, x, o);
  return x;
}

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const T* __restrict__ in, unsigned long long n,
                                                              T* __restrict__ sums) {
  __shared__ T s_tot[SCAN_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long r0 = (unsigned long long)blockIdx.x * SCAN_TILE + (unsigned long long)warp * SCAN_WROWS;
  T acc = 0;
#pragma unroll 4
  for (int gi = 0; gi < SCAN_GROUPS; ++gi) {
    const unsigned long long row = r0 + (unsigned long long)gi * 32 + lane;
    if (row < n) acc += in[row];
  }
  acc = warp_sum<T>(acc);
  if (lane == 0) s_tot[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    T total = 0;
    for (int w = 0; w < SCAN_WARPS; ++w) total += s_tot[w];
    sums[blockIdx.x] = total;
  }
}

// `sums`: the blocks' totals (FOLD) or their exclusive prefixes, or nullptr
// for a single block.  `cursor` (may be nullptr, may be `in`): a second copy
// of the prefixes, for a scatter to count up from.
template <typename T, bool FOLD>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply(const T* in, unsigned long long n,
                                                             const T* __restrict__ sums, T* __restrict__ out,
                                                             T* cursor) {
  __shared__ T s_tot[SCAN_WARPS], s_before[SCAN_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned long long r0 = (unsigned long long)blockIdx.x * SCAN_TILE + (unsigned long long)warp * SCAN_WROWS;
  T before = 0;  // total of the blocks before this one
  if (FOLD && sums) {
    for (unsigned b = threadIdx.x; b < blockIdx.x; b += SCAN_THREADS) before += sums[b];
    before = warp_sum<T>(before);
  } else if (sums) {
    before = threadIdx.x == 0 ? sums[blockIdx.x] : T(0);
  }
  T ex[SCAN_GROUPS];  // exclusive prefix of each of this lane's elements within the warp's
  T carry = 0;
#pragma unroll
  for (int gi = 0; gi < SCAN_GROUPS; ++gi) {
    const unsigned long long row = r0 + (unsigned long long)gi * 32 + lane;
    const T v = row < n ? in[row] : T(0);
    const T x = warp_inclusive_scan<T>(v);
    ex[gi] = carry + x - v;
    carry += __shfl_sync(0xFFFFFFFFu, x, 31);
  }
  if (lane == 0) {
    s_tot[warp] = carry;
    s_before[warp] = before;
  }
  __syncthreads();
  T off = 0, total = 0;
#pragma unroll
  for (int w = 0; w < SCAN_WARPS; ++w) {
    off += s_before[w] + (w < warp ? s_tot[w] : T(0));
    total += s_before[w] + s_tot[w];
  }
#pragma unroll
  for (int gi = 0; gi < SCAN_GROUPS; ++gi) {
    const unsigned long long row = r0 + (unsigned long long)gi * 32 + lane;
    if (row < n) {
      out[row] = off + ex[gi];
      if (cursor) cursor[row] = off + ex[gi];
    }
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = total;
}

// Scratch elements (of T) needed by scan() for n elements.
inline unsigned long long scan_temp_elems(unsigned long long n) {
  unsigned long long need = 0;
  while (true) {
    unsigned long long nblk = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (nblk <= 1) break;
    need += 2 * nblk + 1;
    n = nblk;
  }
  return need + 1;
}

// Returns the number of kernel launches issued.
template <typename T>
int scan(T* in, T* out, unsigned long long n, T* temp, cudaStream_t s, T* cursor = nullptr) {
  unsigned long long nblk = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (nblk <= 1) {
    k_scan_apply<T, false><<<1, SCAN_THREADS, 0, s>>>(in, n, nullptr, out, cursor);
    return 1;
  }
  T* sums = temp;
  k_scan_reduce<T><<<(unsigned)nblk, SCAN_THREADS, 0, s>>>(in, n, sums);
  if (nblk <= SCAN_FOLD_BLOCKS) {
    k_scan_apply<T, true><<<(unsigned)nblk, SCAN_THREADS, 0, s>>>(in, n, sums, out, cursor);
    return 2;
  }
  T* sums_out = temp + nblk;
  const int launches = scan<T>(sums, sums_out, nblk, sums_out + nblk + 1, s);
  k_scan_apply<T, false><<<(unsigned)nblk, SCAN_THREADS, 0, s>>>(in, n, sums_out, out, cursor);
  return launches + 2;
}

}  // namespace rzd
