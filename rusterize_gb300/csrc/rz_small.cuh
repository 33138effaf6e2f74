// rz_small.cuh -- the pipeline from the table check to the scatter as one
// cooperative launch, for small calls.
//
// A call of a few dozen polygons spent most of its time between kernels: ten
// launches of 1 to 10 us each, and the host needs about 5 us per launch (64
// polygons over 256 x 256 pixels: 153 us a call, 54 us of them kernels; as one
// launch 114 us, and 89 us with fewer queries and events around it).  Here
// the same bodies run one after the other in one grid, with grid-wide
// barriers between them.
#pragma once

#include "rz_kernels.cuh"
#include "rz_scan.cuh"

namespace rzd {

constexpr int SMALL_JOB_THREADS = 128;
constexpr int SMALL_JOB_WIDE_SMEM = BITMAP_WORDS * 4 + (SMALL_JOB_THREADS / 32) * POLY_WARP_QCAP * POLY_QENT;
constexpr int SMALL_JOB_LINE_SMEM = LINE_WARPS * line_warp_bytes<false>();
constexpr int SMALL_JOB_SMEM = SMALL_JOB_WIDE_SMEM > SMALL_JOB_LINE_SMEM ? SMALL_JOB_WIDE_SMEM : SMALL_JOB_LINE_SMEM;
static_assert(SMALL_JOB_SMEM >= SMALL_SMEM && SMALL_WARPS * 32 == SMALL_JOB_THREADS &&
              LINE_WARPS * 32 == SMALL_JOB_THREADS, "one block shape for every phase");

struct SmallArgs {
  Geo geo;
  Grid g;
  JobDims one;
  unsigned* part_geom;
  PartPlan* plan;
  Lists lists;
  PrepOut out;
  Tune tune;
  RecBuf sb;
  unsigned* bcount;
  unsigned* boff;
  unsigned* cursor;
  uint2* sorted;
  unsigned long long nbuckets;
  unsigned n_bands;  // 0: no band check
  int repeats;
  Ctrl* ctrl;
};

// Exclusive prefix sums of n counts by one block, and a second copy of them.
__device__ __forceinline__ void block_scan(const unsigned* in, unsigned n, unsigned* out, unsigned* cursor) {
  __shared__ unsigned s_tot[SMALL_JOB_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned base = 0;
  for (unsigned i0 = 0; i0 < n; i0 += SMALL_JOB_THREADS * 4) {
    const unsigned i = i0 + threadIdx.x * 4;
    unsigned v[4], sum = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = i + k < n ? in[i + k] : 0u;
      sum += v[k];
    }
    const unsigned incl = warp_inclusive_scan<unsigned>(sum);
    if (lane == 31) s_tot[warp] = incl;
    __syncthreads();
    unsigned before = base, total = 0;
#pragma unroll
    for (int w = 0; w < SMALL_JOB_THREADS / 32; ++w) {
      before += w < warp ? s_tot[w] : 0u;
      total += s_tot[w];
    }
    before += incl - sum;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < n) out[i + k] = cursor[i + k] = before;
      before += v[k];
    }
    base += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = base;
}

__global__ void __launch_bounds__(SMALL_JOB_THREADS, 4) k_small_job(SmallArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  cg::grid_group grid = cg::this_grid();
  Ctrl* ctrl = a.ctrl;
  __shared__ unsigned s_go;
  // After a barrier: whether the block goes on.  One thread decides for the
  // block, because another block may already be in the next phase and set
  // an error there while this one looks.
  auto go = [&]() {
    grid.sync();
    if (threadIdx.x == 0) s_go = *reinterpret_cast<volatile unsigned*>(&ctrl->err) == 0u;
    __syncthreads();
    const bool yes = s_go != 0u;
    __syncthreads();
    return yes;
  };
  tables_body(a.geo, a.part_geom, ctrl);
  bool ok = go();
  if (a.n_bands) {
    if (ok) bands_body(a.geo, a.n_bands, ctrl);
    ok = go();
  }
  if (ok) prep_body(a.geo, a.g, a.one, nullptr, 1, a.part_geom, a.plan, a.lists, a.out, a.tune, 1, ctrl);
  ok = go();
  if (ctrl->big_parts) {  // parts for k_part_prep_big: the call goes on with the kernels of its own
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ctrl->stopped = 1;
      ctrl->span_count = ~0ull;  // the fill does nothing
    }
    return;
  }
  const WorkList* l = a.lists.l;
  const bool lines = wl_total(ctrl->list[WL_LINE]) != 0;
  if (ok) {
    narrow_body(a.geo, a.g, a.plan, l[WL_NARROW], a.sb, a.bcount, a.tune.narrow_chunk, ctrl);
    __syncthreads();
    if (wl_total(ctrl->list[WL_WIDE]))
      wide_body<SMALL_JOB_THREADS>(a.geo, a.g, a.plan, l[WL_WIDE], a.sb, a.bcount, ctrl);
    __syncthreads();
    if (lines)
      line_body<false, 1>(a.geo, a.g, a.plan, l[WL_LINE], a.out.last_kept, a.repeats, a.sb, a.bcount, ctrl, smem);
    if (wl_total(ctrl->list[WL_POINT]))
      point_body(a.geo, a.g, a.one, 0, a.plan, a.part_geom, l[WL_POINT], a.sb, a.bcount, ctrl);
  }
  ok = go();
  if (lines) {
    if (ok) endpix_body(a.geo, a.g, a.plan, l[WL_LINE], a.out.last_kept, a.sb, a.bcount, ctrl);
    ok = go();
  }
  if (blockIdx.x == 0) block_scan(a.bcount, (unsigned)a.nbuckets, a.boff, a.cursor);
  ok = go();
  const unsigned long long n = *reinterpret_cast<volatile unsigned long long*>(&ctrl->span_count);
  if (ok && n <= a.sb.cap) scatter_body(a.sb, n, a.cursor, a.sorted);
}

}  // namespace rzd
