// The list build's rows, run by the kernels that prepare the pair kernels' sites.
#pragma once

#include "mmnb_internal.cuh"

namespace mmnb {

__device__ __forceinline__ double exact_wrap(double x, double L, double invL)
{
  // x - L * floor(x * (1/L) + 0.5)   (include/pbc.h:8-14)
  return __dsub_rn(x, __dmul_rn(L, floor(__dadd_rn(__dmul_rn(x, invL), 0.5))));
}

__device__ __forceinline__ double exact_sq3(double x, double y, double z)
{
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

struct RebuildArgs {
  int ngroup, ncell3, nstencil, rowcap;
  CellGeom cg;
  Box box;
  const double *anchor;      // this evaluation's anchors (original order)
  const int *cell_rank;      // reference cell index -> Morton rank
  const int *stencil;        // 3 per offset, components in [0, n)
  int *flags;
  int *cell_of_group, *cell_count, *next, *start, *sorted, *rank;  // next: the group that arrived before
  double *last, *anchor_sorted;
  int *nbr, *nbr_count;
  // FP32 pre-test of the list build: sorted anchors wrapped into the box, and
  // squared distances that are certainly inside (< c2lo) or outside (> c2hi)
  // of (cutoff + width)^2 whatever the FP32 rounding; only the rest take the
  // exact FP64 test, so the pair set is the same
  float4 *anchor32;
  float Lf[3], invLf[3];
  float c2lo, c2hi;
  // per-row cull of stencil cells: a cell whose every point is farther than
  // sqrt(c2cull) > cutoff + width from the row's anchor holds no partner
  float lcf[3], c2cull;
  int *head;                 // per rank: the cell's last group to arrive
  int *rank_of_group;        // scratch, ngroup: the Morton rank of each group's cell
  int *chunk;                // groups of each 2^chunk_shift cells (ranks)
  int chunk_shift, nchunk;
};

// one warp per sorted group.  Per batch of 32 stencil cells the members are
// laid out in one candidate sequence (cell order, then member order; a warp
// scan of the cells' counts gives each cell's offset), the lanes test
// consecutive candidates, and the accepted ones are compacted into the row
// with a ballot.  Rows are in a fixed order (deterministic lists).
constexpr int kCand = 128;  // candidates staged per warp at a time
constexpr int kSeg = 256;   // stencil cells whose member ranges a warp fetches at a time

__device__ __forceinline__ void build_row(const RebuildArgs &a, int p, int lane, int *cand, int2 *ranges)
{
  const int n = a.cg.n;
  const int gi = a.sorted[p];
  const int ci = a.cell_of_group[gi];
  const int ix = ci / (n * n), iy = (ci / n) % n, iz = ci % n;
  const double xi = a.anchor_sorted[3 * p], yi = a.anchor_sorted[3 * p + 1], zi = a.anchor_sorted[3 * p + 2];
  const float4 wi = a.anchor32[p];
  int *row = a.nbr + (size_t) p * a.rowcap;
  const unsigned below = (1u << lane) - 1;
  int count = 0;
  for (int g0 = 0; g0 < a.nstencil; g0 += kSeg) {
    // the member ranges of a segment of stencil cells, fetched with independent
    // loads (one dependent chain per cell instead of one per batch of 32);
    // the cells that can hold a partner and are not empty are compacted in
    // stencil order, so the batches below see only them (the own cell, stencil
    // entry 0, always has the row's group and comes first)
    const int segn = min(kSeg, a.nstencil - g0);
    int kept = 0;
#pragma unroll 2
    for (int t0 = 0; t0 < segn; t0 += 32) {
      const int t = t0 + lane;
      int2 rg = make_int2(0, 0);
      if (t < segn) {
        const int s = g0 + t;
        // cell and stencil components are in [0, n): one conditional subtraction wraps
        int jx = ix + a.stencil[3 * s], jy = iy + a.stencil[3 * s + 1], jz = iz + a.stencil[3 * s + 2];
        jx -= jx >= n ? n : 0;
        jy -= jy >= n ? n : 0;
        jz -= jz >= n ? n : 0;
        // lower bound of the distance from this row's anchor (wrapped into the
        // box) to the cell's slab [c l - l/2, c l + l/2] on each axis, minimum image
        float dx = wi.x - (float) jx * a.lcf[0], dy = wi.y - (float) jy * a.lcf[1], dz = wi.z - (float) jz * a.lcf[2];
        dx = fmaxf(fabsf(dx - a.Lf[0] * rintf(dx * a.invLf[0])) - 0.5f * a.lcf[0], 0.f);
        dy = fmaxf(fabsf(dy - a.Lf[1] * rintf(dy * a.invLf[1])) - 0.5f * a.lcf[1], 0.f);
        dz = fmaxf(fabsf(dz - a.Lf[2] * rintf(dz * a.invLf[2])) - 0.5f * a.lcf[2], 0.f);
        if (s == 0 || dx * dx + dy * dy + dz * dz <= a.c2cull) {
          const int rj = a.cell_rank[(jx * n + jy) * n + jz];
          rg = make_int2(a.start[rj], a.start[rj + 1]);
        }
      }
      const bool keep = rg.y > rg.x;
      const unsigned kb = __ballot_sync(0xffffffffu, keep);
      if (keep)
        ranges[kept + __popc(kb & below)] = rg;
      kept += __popc(kb);
    }
    __syncwarp();
    for (int b0 = 0; b0 < kept; b0 += 32) {
      const int s0 = g0 + b0;
      int beg = 0, end = 0;
      if (b0 + lane < kept) {
        const int2 rg = ranges[b0 + lane];
        beg = rg.x;
        end = rg.y;
      }
      const int c = end - beg;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
          incl += v;
      }
      const int excl = incl - c;
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      // stencil entry 0 is the group's own cell: its members pair unconditionally
      const int own = s0 == 0 ? __shfl_sync(0xffffffffu, incl, 0) : 0;
      for (int base = 0; base < total; base += kCand) {
        const int lo = max(excl, base), hi = min(incl, base + kCand);
        for (int k = lo; k < hi; k++)
          cand[k - base] = beg + (k - excl);
        __syncwarp();
        const int nb = min(kCand, total - base);
        for (int k0 = 0; k0 < nb; k0 += 32) {
          const int k = k0 + lane;
          bool take = false;
          int q = 0;
          if (k < nb) {
            q = cand[k];
            if (q != p) {
              if (base + k < own) {
                take = true;
              } else {
                const float4 wj = a.anchor32[q];
                float fx = wi.x - wj.x, fy = wi.y - wj.y, fz = wi.z - wj.z;
                fx -= a.Lf[0] * rintf(fx * a.invLf[0]);
                fy -= a.Lf[1] * rintf(fy * a.invLf[1]);
                fz -= a.Lf[2] * rintf(fz * a.invLf[2]);
                const float f2 = fx * fx + fy * fy + fz * fz;
                if (f2 < a.c2lo) {
                  take = true;
                } else if (f2 <= a.c2hi) {
                  const double dx = exact_wrap(__dsub_rn(xi, a.anchor_sorted[3 * q]), a.box.L[0], a.box.invL[0]);
                  const double dy = exact_wrap(__dsub_rn(yi, a.anchor_sorted[3 * q + 1]), a.box.L[1], a.box.invL[1]);
                  const double dz = exact_wrap(__dsub_rn(zi, a.anchor_sorted[3 * q + 2]), a.box.L[2], a.box.invL[2]);
                  take = exact_sq3(dx, dy, dz) < a.cg.c2;
                }
              }
            }
          }
          const unsigned bal = __ballot_sync(0xffffffffu, take);
          if (take) {
            const int idx = count + __popc(bal & below);
            if (idx < a.rowcap)
              row[idx] = q;
          }
          count += __popc(bal);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  }
  if (lane == 0) {
    a.nbr_count[p] = min(count, a.rowcap);
    if (count > a.rowcap) {
      atomicMax(&a.flags[kFlagOverflow], count);
      a.flags[kFlagListTrunc] = 1;
    }
    atomicMax(&a.flags[kFlagMaxRow], count);
  }
}

// All rows, by every block of a launch of 256-thread blocks, when this evaluation
// rebuilds the list (the cells and sorted order are in place).  The kernels that
// sort the sites call it after their own work: neither reads the other's output, and
// on an evaluation without a rebuild it costs one read of the flag.
constexpr int kRowWarps = 8;

__device__ __forceinline__ void build_rows(const RebuildArgs &a)
{
  if (!a.flags[kFlagRebuild])
    return;
  __shared__ int cand[kRowWarps * kCand];
  __shared__ int2 ranges[kRowWarps * kSeg];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int p = blockIdx.x * kRowWarps + w; p < a.ngroup; p += gridDim.x * kRowWarps)
    build_row(a, p, lane, cand + w * kCand, ranges + w * kSeg);
}

RebuildArgs rebuild_args(const mmnb_handle *h);

// blocks of a site-sorting launch over n slots: enough warps for the rows as well
inline int sort_blocks(const mmnb_handle *h, int n)
{
  const int rows = div_up(h->ngroup, kRowWarps), full = 5 * 148;
  return div_up(n, 32 * kRowWarps) > rows ? div_up(n, 32 * kRowWarps)
         : div_up(n, 32 * kRowWarps) > full ? div_up(n, 32 * kRowWarps)
         : rows < full ? rows : full;
}

}  // namespace mmnb
