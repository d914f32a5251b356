// Cell neighbour list on the GPU: rebuild trigger, cell assignment, Morton
// counting sort and warp-ballot list build.
//
// Semantics follow the reference's NeighborList exactly (src/nbrlist.cpp):
//   * a rebuild happens on the first evaluation and whenever the two largest
//     anchor moves since the last build add up to more than the skin
//     (coordinates_changed, :51-77);
//   * a group's cell is round(x / l_cell) mod n per axis with
//     l_cell = L * (1.0 / n) (rebuild_periodic :228-234, Cubic/Orthorhombic
//     nearest_lattice_point src/bcond.cpp:31-34, include/pbc.h:25-31, 52-59);
//   * groups in the same cell are paired unconditionally (:243-244);
//   * groups in cells joined by the reference's cell stencil are paired when
//     their minimum-image distance squared is below (cutoff + width)^2
//     (:245-248, include/bcond.hpp:56-60).
// The arithmetic that decides membership (cell index, squared distance,
// displacement test) uses explicitly rounded FP64 operations so it cannot be
// contracted into FMAs: it is the same IEEE sequence the reference executes,
// and the pair set is identical, not merely close.  The list build first
// tests each candidate in FP32 against a band around (cutoff + width)^2 wide
// enough to hold every FP32 rounding error; only candidates inside the band
// take the FP64 test, so the decision is the FP64 one.
//
// The list is stored FULL (each unordered pair in both rows) so the pair
// kernels accumulate on their own rows only, without atomics.  Rows are
// indexed by sorted position (groups ordered by the Morton rank of their cell).

#include <algorithm>
#include <cmath>

#include "nbrlist.cuh"

namespace mmnb {

// merge two (largest, second largest) pairs of a multiset
__device__ __forceinline__ void top2_merge(double &a, double &b, double a2, double b2)
{
  const double hi = fmax(a, a2), lo = fmin(a, a2);
  b = fmax(lo, fmax(b, b2));
  a = hi;
}

constexpr int kCheckThreads = 256;

__device__ __forceinline__ void block_top2(double &a, double &b, double *sa, double *sb)
{
  sa[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      double x = sa[threadIdx.x], y = sb[threadIdx.x];
      top2_merge(x, y, sa[threadIdx.x + s], sb[threadIdx.x + s]);
      sa[threadIdx.x] = x;
      sb[threadIdx.x] = y;
    }
    __syncthreads();
  }
  a = sa[0];
  b = sb[0];
  __syncthreads();  // sa, sb may be reused at once
}

// Anchors of this evaluation, the two largest anchor moves since the last
// build, and the rebuild decision (first || forced || largest + second >
// width || fixed interval), all in one launch: each block reduces its share,
// the last block to finish merges the block results.  On a rebuild the last
// block also clears the cell counts for the rebuild kernel.
// flags[4] counts evaluations, flags[5] rebuilds, flags[6] is the block counter.
// With pruned rows (prune > 0; the rigid-water kernel) the same pass takes
// the two largest moves since the last prune (plast, sorted order of the
// build) and sets flags[kFlagPruneFull] when the pruned rows must be made
// again: after a rebuild, while they are not valid, or when those moves add
// up to more than the prune margin.
__global__ void __launch_bounds__(kCheckThreads) k_list_check(const double *__restrict__ r,
                                                              const int *__restrict__ group, int ngroup,
                                                              const double *__restrict__ last, double width,
                                                              int first, int force, int interval,
                                                              double *__restrict__ anchor,
                                                              double *__restrict__ partial, int *__restrict__ flags,
                                                              int *__restrict__ cell_count, int ncount,
                                                              double prune, const int *__restrict__ rank,
                                                              const double *__restrict__ plast)
{
  __shared__ double sa[kCheckThreads], sb[kCheckThreads];
  __shared__ bool last_block;
  double a = 0, b = 0, pa = 0, pb = 0;
  cudaTriggerProgrammaticLaunchCompletion();
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroup; g += gridDim.x * blockDim.x) {
    const int s0 = group[2 * g];
    const double x = r[3 * s0], y = r[3 * s0 + 1], z = r[3 * s0 + 2];
    anchor[3 * g] = x;
    anchor[3 * g + 1] = y;
    anchor[3 * g + 2] = z;
    const double dx = __dsub_rn(x, last[3 * g]);
    const double dy = __dsub_rn(y, last[3 * g + 1]);
    const double dz = __dsub_rn(z, last[3 * g + 2]);
    // squared moves: the square root (monotonic, correctly rounded) is
    // taken of the two largest only, in the last block
    const double d = exact_sq3(dx, dy, dz);
    if (d > a) {
      b = a;
      a = d;
    } else if (d > b) {
      b = d;
    }
    // before the first build there are no ranks to read (and the rows are made
    // anew whatever the moves)
    if (prune > 0 && !first) {
      const int p = rank[g];
      const double ex = x - plast[3 * p], ey = y - plast[3 * p + 1], ez = z - plast[3 * p + 2];
      const double e = ex * ex + ey * ey + ez * ez;
      if (e > pa) {
        pb = pa;
        pa = e;
      } else if (e > pb) {
        pb = e;
      }
    }
  }
  block_top2(a, b, sa, sb);
  if (prune > 0)
    block_top2(pa, pb, sa, sb);
  if (threadIdx.x == 0) {
    partial[4 * blockIdx.x] = a;
    partial[4 * blockIdx.x + 1] = b;
    partial[4 * blockIdx.x + 2] = pa;
    partial[4 * blockIdx.x + 3] = pb;
    __threadfence();
    last_block = atomicAdd(flags + 6, 1) == (int) gridDim.x - 1;
  }
  __syncthreads();
  if (!last_block)
    return;
  __threadfence();
  a = b = pa = pb = 0;
  for (int i = threadIdx.x; i < (int) gridDim.x; i += blockDim.x) {
    top2_merge(a, b, partial[4 * i], partial[4 * i + 1]);
    top2_merge(pa, pb, partial[4 * i + 2], partial[4 * i + 3]);
  }
  block_top2(a, b, sa, sb);
  block_top2(pa, pb, sa, sb);
  a = __dsqrt_rn(a);
  b = __dsqrt_rn(b);
  pa = sqrt(pa);
  pb = sqrt(pb);
  __shared__ int rebuild_s;
  if (threadIdx.x == 0) {
    const int count = flags[4];
    int rebuild = first || force || flags[kFlagForceRebuild] || (__dadd_rn(b, a) > width);
    flags[kFlagForceRebuild] = 0;
    if (interval > 0 && count % interval == 0)
      rebuild = 1;
    flags[kFlagRebuild] = rebuild;
    flags[4] = count + 1;
    if (rebuild)
      flags[5] += 1;  // rebuild counter
    flags[6] = 0;
    rebuild_s = rebuild;
    if (rebuild) {
      flags[kFlagPruneValid] = 0;
      flags[kFlagListTrunc] = 0;
    }
    flags[kFlagPruneFull] = prune > 0 ? (rebuild || !flags[kFlagPruneValid] || pa + pb > prune) : 1;
  }
  __syncthreads();
  if (rebuild_s)
    for (int c = threadIdx.x; c < ncount; c += blockDim.x)
      cell_count[c] = 0;
}

constexpr int kCellThreads = 256;       // blocks of the two-kernel cell sort
constexpr int kOneBlockThreads = 1024;  // the one-block cell sort

// Morton rank of group g's cell = round(x / l_cell) mod n per axis; the anchors become
// the new "last"
__device__ __forceinline__ int cell_assign(const RebuildArgs &a, int g)
{
  const int n = a.cg.n;
  int ijk[3];
  for (int d = 0; d < 3; d++) {
    const double x = a.anchor[3 * g + d];
    // a non-finite anchor converts to cell 0 (float-to-int conversion gives 0
    // for NaN and saturates): flagged, the host reports it
    if (!isfinite(x))
      a.flags[kFlagError] = MMNB_ERR_DEVICE;
    ijk[d] = (int) floor(__dadd_rn(__ddiv_rn(x, a.cg.lc[d]), 0.5));
    ijk[d] %= n;
    if (ijk[d] < 0)
      ijk[d] += n;
    a.last[3 * g + d] = x;
  }
  const int c = (ijk[0] * n + ijk[1]) * n + ijk[2];
  a.cell_of_group[g] = c;
  return a.cell_rank[c];
}

// Exclusive scan of the values of a block of T threads (one per thread): the
// thread's exclusive prefix and the block total.
template <int T>
__device__ __forceinline__ int block_exclusive_scan(int v, int *warp_tot, int &total)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o)
      incl += u;
  }
  if (lane == 31)
    warp_tot[w] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
  for (int k = 0; k < T / 32; k++) {
    const int t = warp_tot[k];
    before += k < w ? t : 0;
    total += t;
  }
  __syncthreads();
  return before + incl - v;
}

// group g at sorted position pos: its rank and the anchors the list is built from
__device__ __forceinline__ void place_group(const RebuildArgs &a, int g, int pos)
{
  a.sorted[pos] = g;
  a.rank[g] = pos;
  float w[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double x = a.anchor[3 * g + d];
    a.anchor_sorted[3 * pos + d] = x;
    w[d] = (float) (x - a.box.L[d] * floor(x * a.box.invL[d]));
  }
  a.anchor32[pos] = make_float4(w[0], w[1], w[2], 0.f);
}

// groups of the cells before cell k: those of the chunks before its own (`before`, in
// shared memory) and of the cells before it there
__device__ __forceinline__ int cell_offset(const RebuildArgs &a, const int *before, int k)
{
  const int c = k >> a.chunk_shift;
  int v = before[c];
#pragma unroll 4
  for (int i = c << a.chunk_shift; i < k; i += 4) {
    const int4 n = __ldcg(reinterpret_cast<const int4 *>(a.cell_count + i));
    v += n.x + (i + 1 < k ? n.y : 0) + (i + 2 < k ? n.z : 0) + (i + 3 < k ? n.w : 0);
  }
  return v;
}

// Cells and sorted order of a rebuild.  Without one due every block returns at once
// (the decision is read from device memory, so the launches sit in a CUDA graph
// unchanged).  As phases of one cooperative launch with the rows, separated by grid
// barriers, they cost every evaluation a wait for the whole grid's room (together with
// the site kernel's change: the 648-site k-sum box 90 -> 86 us per call, twelve
// replicas at once 3432 -> 3373 us per ten steps, 98,304 sites mixed 177 -> 175.5 us).
__global__ void __launch_bounds__(kCellThreads) k_list_assign(RebuildArgs a)
{
  after_previous();
  if (!a.flags[kFlagRebuild])
    return;
  const int g = blockIdx.x * kCellThreads + threadIdx.x;
  if (g >= a.ngroup)
    return;
  const int k = cell_assign(a, g);
  a.rank_of_group[g] = k;
  atomicAdd(a.cell_count + k, 1);
  atomicAdd(a.chunk + (k >> a.chunk_shift), 1);
  a.next[g] = atomicExch(a.head + k, g);
}

// Offsets of the cells, a thread each; then a thread per group, its place among its
// cell's groups in index order (deterministic lists).  A cell's groups hang on a list in
// order of arrival, and each walks it to count those before it: two on average, tens
// in a droplet or a cluster, whose few cells a thread per cell would leave to a few
// threads (32,768 waters as a droplet in 20 times the volume, mixed, list rebuilt in
// each call: 573 us so, 297 now; 302 with a cooperative launch for all phases).
// Past kWalk of them (all coordinates zero, or not finite) a block counts the cell's
// groups of the blocks before instead, in order.
constexpr int kWalk = 512;

__global__ void __launch_bounds__(kCellThreads) k_list_sort(RebuildArgs a)
{
  constexpr int T = kCellThreads;
  after_previous();
  if (!a.flags[kFlagRebuild])
    return;
  extern __shared__ int before[];  // nchunk
  __shared__ int warp_tot[T / 32], pick;
  int total, run = 0;
  for (int c0 = 0; c0 < a.nchunk; c0 += T) {
    const int c = c0 + threadIdx.x;
    const int ex = block_exclusive_scan<T>(c < a.nchunk ? a.chunk[c] : 0, warp_tot, total);
    if (c < a.nchunk)
      before[c] = run + ex;
    run += total;
  }
  __syncthreads();
  const int g0 = blockIdx.x * T, g = g0 + threadIdx.x;
  if (g < a.ncell3) {
    a.start[g] = cell_offset(a, before, g);
    if (g == a.ncell3 - 1)
      a.start[a.ncell3] = a.ngroup;
  }
  int k = 0, n = 0, at = 0;
  if (g < a.ngroup) {
    k = a.rank_of_group[g];
    n = a.cell_count[k];
    int h = a.head[k];
    at = cell_offset(a, before, k);
    if (n <= kWalk) {
      for (int i = 1; i < n; i++) {
        at += h < g;
        h = a.next[h];
      }
      at += h < g;
      place_group(a, g, at);
    }
  }
  bool crowd = n > kWalk;
  while (__syncthreads_or(crowd)) {
    if (threadIdx.x == 0)
      pick = a.ncell3;
    __syncthreads();
    if (crowd)
      atomicMin(&pick, k);
    __syncthreads();
    const int cell = pick;
    int v = 0;
    for (int j = threadIdx.x; j < g0; j += T)
      v += a.rank_of_group[j] == cell;
    int earlier;
    block_exclusive_scan<T>(v, warp_tot, earlier);
    const bool in = crowd && k == cell;
    const int ex = block_exclusive_scan<T>(in ? 1 : 0, warp_tot, total);
    if (in) {
      place_group(a, g, at + earlier + ex);
      crowd = false;
    }
  }
}

// The same by one block, for boxes it handles as fast as two launches would: counts and
// order in shared memory, the groups ordered by comparing all of their cell's.
constexpr int kOneBlockGroups = 2048, kOneBlockCells = 1024;
constexpr int kOneBlockEach = kOneBlockGroups / kOneBlockThreads;

__global__ void __launch_bounds__(kOneBlockThreads) k_list_cells(RebuildArgs a)
{
  static_assert(kOneBlockCells <= kOneBlockThreads, "a cell per thread");
  after_previous();
  if (!a.flags[kFlagRebuild])
    return;
  __shared__ int count[kOneBlockCells], start[kOneBlockCells], list[kOneBlockGroups], warp_tot[kOneBlockThreads / 32];
  const int t = threadIdx.x;
  if (t < kOneBlockCells)
    count[t] = 0;
  __syncthreads();
  int k[kOneBlockEach], slot[kOneBlockEach];
#pragma unroll
  for (int i = 0; i < kOneBlockEach; i++) {
    const int g = t + i * kOneBlockThreads;
    if (g < a.ngroup) {
      k[i] = cell_assign(a, g);
      slot[i] = atomicAdd(count + k[i], 1);
    }
  }
  __syncthreads();
  int total;
  const int at = block_exclusive_scan<kOneBlockThreads>(t < a.ncell3 ? count[t] : 0, warp_tot, total);
  if (t < a.ncell3)
    start[t] = a.start[t] = at;
  if (t == 0)
    a.start[a.ncell3] = a.ngroup;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kOneBlockEach; i++) {
    const int g = t + i * kOneBlockThreads;
    if (g < a.ngroup)
      list[start[k[i]] + slot[i]] = g;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kOneBlockEach; i++) {
    const int g = t + i * kOneBlockThreads;
    if (g < a.ngroup) {
      const int b = start[k[i]], n = count[k[i]];
      int r = 0;
#pragma unroll 4
      for (int j = 0; j < n; j++)
        r += list[b + j] < g;
      place_group(a, g, b + r);
    }
  }
}

cudaError_t launch_list_check(mmnb_handle *h, const double *d_r, int force)
{
  k_list_check<<<h->top2_blocks, kCheckThreads, 0, h->stream>>>(
      d_r, h->d_group, h->ngroup, h->d_last, h->nlw, h->first ? 1 : 0, force, h->cfg.rebuild_interval, h->d_anchor,
      h->d_top2, h->d_flags, h->d_cell_count, cell_words(h->ncell3), h->water ? h->prune_margin : 0.0, h->d_rank,
      h->d_plast);
  h->launches += 1;
  return cudaGetLastError();
}

RebuildArgs rebuild_args(const mmnb_handle *h)
{
  RebuildArgs a;
  a.ngroup = h->ngroup;
  a.ncell3 = h->ncell3;
  a.nstencil = h->nstencil;
  a.rowcap = h->rowcap;
  a.cg = h->cg;
  a.box = h->box;
  a.anchor = h->d_anchor;
  a.cell_rank = h->d_cell_rank;
  a.stencil = h->d_stencil;
  a.flags = h->d_flags;
  a.cell_of_group = h->d_cell_of_group;
  a.cell_count = h->d_cell_count;
  a.next = h->d_slot;
  a.head = h->d_cell_head;
  a.start = h->d_cell_start;
  a.sorted = h->d_sorted;
  a.rank = h->d_rank;
  a.last = h->d_last;
  a.anchor_sorted = h->d_anchor_sorted;
  a.nbr = h->d_nbr;
  a.nbr_count = h->d_nbr_count;
  a.anchor32 = h->d_anchor32;
  // the rows' counts are written last, by the list build: until then they
  // hold the rank of each group's cell
  a.rank_of_group = h->d_nbr_count;
  a.chunk_shift = chunk_shift(h->ncell3);
  a.chunk = h->d_cell_count + chunk_at(h->ncell3);
  a.nchunk = div_up(h->ncell3, 1 << a.chunk_shift);
  // bound of the FP32 squared-distance error: anchors wrapped into [0, L] and
  // rounded (<= 4 ulp(L) per component after the difference and the image
  // shift), propagated through |d|^2, plus the rounding of the sum; 8x margin
  double lmax = 0, lmin = 1e300;
  for (int d = 0; d < 3; d++) {
    a.Lf[d] = (float) h->box.L[d];
    a.invLf[d] = (float) h->box.invL[d];
    lmax = std::max(lmax, h->box.L[d]);
    lmin = std::min(lmin, h->box.L[d]);
  }
  const double c2 = h->cg.c2, ulp = std::ldexp(1.0, -23);
  const double tol = 8 * (2 * std::sqrt(3.0) * std::sqrt(c2) * 4 * ulp * lmax + 4 * ulp * c2);
  // the FP32 minimum image may pick another image only at |d| ~ L/2
  const bool safe = std::sqrt(c2) + 1.0 < 0.45 * lmin;
  a.c2lo = safe ? (float) (c2 - tol) : -1.0f;
  a.c2hi = safe ? (float) (c2 + tol) : 3.0e38f;
  // the cull keeps a 0.01 A margin over the FP32 rounding of the anchors and
  // cell centres (~1e-5 A here); boxes where the FP32 minimum image is not
  // safe keep every stencil cell
  for (int d = 0; d < 3; d++)
    a.lcf[d] = (float) h->cg.lc[d];
  const double cull = std::sqrt(c2) + 0.01;
  a.c2cull = safe ? (float) (cull * cull) : 3.0e38f;
  return a;
}

// The one-block sort up to kOneBlockGroups (of ncell3 <= ngroup / 2 + 3 cells): a launch
// less in every evaluation, and a faster rebuild up to about there.  Calls with the list
// rebuilt in each, one block against two kernels, mixed: 216 waters 38.7 and 42.8 us,
// 1,000 44.8 and 48.5, 1,500 49.4 and 49.4, 2,048 53.5 and 50.3; rebuilt every ten
// calls: 27.9 and 29.1, 32.0 and 32.7, 34.4 and 34.7, 36.7 and 36.9.
cudaError_t launch_list_cells(mmnb_handle *h)
{
  const RebuildArgs a = rebuild_args(h);
  if (h->ngroup <= kOneBlockGroups && h->ncell3 <= kOneBlockCells) {
    launch_after(h, k_list_cells, 1, kOneBlockThreads, 0, a);
    h->launches += 1;
  } else {
    launch_after(h, k_list_assign, div_up(h->ngroup, kCellThreads), kCellThreads, 0, a);
    launch_after(h, k_list_sort, div_up(std::max(h->ngroup, h->ncell3), kCellThreads), kCellThreads,
                 sizeof(int) * a.nchunk, a);
    h->launches += 2;
  }
  return cudaGetLastError();
}

}  // namespace mmnb
