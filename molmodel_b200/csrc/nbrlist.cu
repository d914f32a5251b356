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
                                                              int *__restrict__ cell_count, int ncell3,
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
    for (int c = threadIdx.x; c < ncell3; c += blockDim.x)
      cell_count[c] = 0;
}

constexpr int kCellThreads = 256;       // blocks of the two-kernel cell sort
constexpr int kOneBlockThreads = 1024;  // the one-block cell sort

// cell = round(x / l_cell) mod n per axis; the anchors become the new "last"
__device__ __forceinline__ void cell_assign(const RebuildArgs &a, int g)
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
  const int k = a.cell_rank[c];
  atomicAdd(a.cell_count + k, 1);
  a.next[g] = atomicExch(a.head + k, g);
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

// The cells of ranks [c0, c0 + T), a thread each: offsets from `base` on (the groups
// of the cells before), and the cells' groups in index order (deterministic lists).
// A cell's groups hang on a list in order of arrival; a few are ordered by walking
// it once per group, the groups of a crowded cell by the whole block.  Returns the
// offset after the last cell.
constexpr int kCrowd = 16;

template <int T>
__device__ int sort_cells(const RebuildArgs &a, int c0, int base, int *warp_tot)
{
  __shared__ int crowd[T], ncrowd;
  if (threadIdx.x == 0)
    ncrowd = 0;
  const int c = c0 + threadIdx.x;
  const int n = c < a.ncell3 ? __ldcg(a.cell_count + c) : 0;
  int total;
  const int at = base + block_exclusive_scan<T>(n, warp_tot, total);
  if (c < a.ncell3)
    a.start[c] = at;
  if (c == a.ncell3 - 1)
    a.start[a.ncell3] = at + n;
  const int head = n > 0 ? __ldcg(a.head + c) : 0;
  if (n == 1) {
    place_group(a, head, at);
  } else if (n > kCrowd) {
    int g = head;
    for (int k = 0; k < n; k++, g = __ldcg(a.next + g))
      a.scatter[at + k] = g;
    crowd[atomicAdd(&ncrowd, 1)] = threadIdx.x;
  } else if (n > 1) {
    int m[kCrowd];
    int g = head;
#pragma unroll
    for (int k = 0; k < kCrowd; k++) {
      m[k] = 0x7fffffff;
      if (k < n) {
        m[k] = g;
        if (k + 1 < n)
          g = __ldcg(a.next + g);
      }
    }
#pragma unroll
    for (int k = 0; k < kCrowd; k++) {
      if (k >= n)
        break;
      int r = 0;
#pragma unroll
      for (int j = 0; j < kCrowd; j++)
        r += m[j] < m[k];
      place_group(a, m[k], at + r);
    }
  }
  __syncthreads();
  for (int q = 0; q < ncrowd; q++) {
    const int cq = c0 + crowd[q], b = a.start[cq], e = b + __ldcg(a.cell_count + cq);
    for (int i = b + threadIdx.x; i < e; i += T) {
      const int g = a.scatter[i];
      int r = 0;
      for (int j = b; j < e; j++)
        r += a.scatter[j] < g;
      place_group(a, g, b + r);
    }
  }
  __syncthreads();
  return base + total;
}

// Cells and sorted order of a rebuild.  Without one due every block returns at once
// (the decision is read from device memory, so the launches sit in a CUDA graph
// unchanged).  As phases of one cooperative launch with the rows, separated by grid
// barriers, they cost every evaluation a wait for the whole grid's room: the 648-site
// k-sum box 90 -> 80 us per call, twelve replicas at once 3700 -> 3410 us per ten
// steps, 98,304 sites mixed 186 -> 178 us.
__global__ void __launch_bounds__(kCellThreads) k_list_assign(RebuildArgs a)
{
  after_previous();
  if (!a.flags[kFlagRebuild])
    return;
  const int g = blockIdx.x * kCellThreads + threadIdx.x;
  if (g < a.ngroup)
    cell_assign(a, g);
}

__global__ void __launch_bounds__(kCellThreads) k_list_sort(RebuildArgs a)
{
  after_previous();
  if (!a.flags[kFlagRebuild])
    return;
  __shared__ int warp_tot[kCellThreads / 32];
  // groups of the blocks before
  const int c0 = blockIdx.x * kCellThreads;
  int v = 0, base;
#pragma unroll 8
  for (int i = threadIdx.x; i < c0; i += kCellThreads)
    v += __ldcg(a.cell_count + i);
  block_exclusive_scan<kCellThreads>(v, warp_tot, base);
  sort_cells<kCellThreads>(a, c0, base, warp_tot);
}

// both steps by one block, for boxes it handles as fast as two launches would
__global__ void __launch_bounds__(kOneBlockThreads) k_list_cells(RebuildArgs a)
{
  after_previous();
  if (!a.flags[kFlagRebuild])
    return;
  __shared__ int warp_tot[kOneBlockThreads / 32];
  for (int g = threadIdx.x; g < a.ngroup; g += kOneBlockThreads)
    cell_assign(a, g);
  __syncthreads();
  int base = 0;
  for (int c0 = 0; c0 < a.ncell3; c0 += kOneBlockThreads)
    base = sort_cells<kOneBlockThreads>(a, c0, base, warp_tot);
}

cudaError_t launch_list_check(mmnb_handle *h, const double *d_r, int force)
{
  k_list_check<<<h->top2_blocks, kCheckThreads, 0, h->stream>>>(
      d_r, h->d_group, h->ngroup, h->d_last, h->nlw, h->first ? 1 : 0, force, h->cfg.rebuild_interval, h->d_anchor,
      h->d_top2, h->d_flags, h->d_cell_count, h->ncell3, h->water ? h->prune_margin : 0.0, h->d_rank,
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
  // hold the groups in cell order
  a.scatter = h->d_nbr_count;
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

// The one-block sort up to this many groups: a launch less in every evaluation
// (~1.3 us), against a slower rebuild (profiled cold, 512 groups: 9 us in one block;
// 4,096 groups: 33 us against 5 + 12; 32,768 in one block 147 us against 5 + 15)
constexpr int kOneBlockGroups = 2048;

cudaError_t launch_list_cells(mmnb_handle *h)
{
  const RebuildArgs a = rebuild_args(h);
  if (h->ngroup <= kOneBlockGroups) {
    launch_after(h, k_list_cells, 1, kOneBlockThreads, 0, a);
    h->launches += 1;
  } else {
    launch_after(h, k_list_assign, div_up(h->ngroup, kCellThreads), kCellThreads, 0, a);
    launch_after(h, k_list_sort, div_up(h->ncell3, kCellThreads), kCellThreads, 0, a);
    h->launches += 2;
  }
  return cudaGetLastError();
}

}  // namespace mmnb
