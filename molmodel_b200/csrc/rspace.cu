// Real-space Ewald + Lennard-Jones, FP64 form.
//
// Replaces RSpaceEwald (src/rspace.c:382-558).  Semantics kept from the
// reference:
//   * cutoff, switching and minimum image are decided per GROUP pair from the
//     two anchor sites; every site pair of the group pair uses the anchors'
//     image shift (src/rspace.c:423-478);
//   * the quintic switch S(z), z = (r^2 - rlo^2)/(rhi^2 - rlo^2), multiplies
//     both Coulomb and LJ terms; the switch derivative times the summed
//     unswitched energy acts on the anchors only (:479-489);
//   * erfc(eta r)/r and its -2 d/d(r^2) come from the reference's own
//     512-segment Chebyshev table inside its range, from erfc/exp outside
//     (:104-156);
//   * excluded site pairs are skipped only inside group pairs that contain an
//     exclusion (group_excluded, :422, 446, 465), and every excluded charged
//     pair gets the -erf(eta r)/r correction (:492-521);
//   * 1-4 pairs get scaled plain Coulomb + LJ (:522-557).
//
// Layout: the neighbour list is full (both directions); one warp, or a team of up
// to four for small systems, owns one group row and takes the next from a
// counter.  Three queues in shared memory keep every lane busy whatever the
// groups hold:
//   * the list is walked 32 entries at a time (a lane per partner: anchor
//     displacement, cutoff), the partners inside the cutoff queued;
//   * queued partners are expanded to their sites, a lane per site (so the site
//     records are read in whole lines, one batch ahead), charged sites and LJ
//     sites each to a queue of their own with the partner's switch and
//     displacement folded in;
//   * queued charged sites are evaluated against the row's charged sites, queued LJ
//     sites against its LJ sites: lane = (row site, partner site), 32 / n of the
//     partners' sites per step for n row sites.  No lane holds a site that lacks
//     the term, so the sums of a lane are one site's: 12 doubles at most, and the
//     kernel is the same for groups of one site and of eight.
// The reference's table is in shared memory, the cubic alone: b1 is -2 / dx times its
// derivative, which is how the reference stores it; below the table (r^2 < 4)
// ewald_short, past it (r^2 > 1.2 rc^2) polynomials of degree seven that are the
// function to rounding, where the reference takes erfc and exp (which a few lanes of
// nearly every step would take, the others waiting: 17^3 cells of solution, per call,
// 134 us with the functions, 127 with these).
// Lanes' sums are added in a fixed order: no atomics, bitwise reproducible whichever
// warp takes a row.
//
// Bound by latency (12 warps of 168 registers per SM; 16 of 128 spill and were
// slower, 86 against 115 us) and the shared-memory pipe.  Measured on 17^3 cells of
// solution (14,100 sites in groups of two to four, exclusions across groups): a
// warp per row with a lane per partner GROUP over all its padded site pairs, erfc
// branch and exclusion searches included, 484 us; this layout 86 us.  On 32^3 cells
// (94,000 sites): 455 us.  A lane per partner site over all the row's sites, in
// registers, took 152 us on the smaller box (idle lanes of padded groups, spills).
// Rigid water has its own kernel (rspace_water64.cu), which is faster there (44
// against 68 us on 4,096 waters, 191 against 392 us on 32,768).

#include "nbrlist.cuh"

#include <algorithm>

namespace mmnb {

constexpr int kP64Warps = 12;  // at most, per block: 168 registers a thread, no spills
constexpr int kP64Ring = 64;   // entries per queue: at most 31 carried over and 32 new

struct PairArgs {
  int ngroup, rowcap, geometric, G, width, batch, split, copies, series, half;  // half: entries to the (c2, c3)
  Box box;
  double rlo2, rhi2, inv_sw, eta, eta2, cerf;  // cerf = 2 eta / sqrt(pi)
  double cmin, inv_dx, dscale, inv_dscale;     // dscale = -2 / segment width
  const double2 *table;                        // (c0, c1) of each segment, from `half` on (c2, c3)
  const double2 *tail;                         // past the table: 4 per segment, powers 0..7 of its position
  double tmin, tail_inv, tail_nseg, tscale;    // tscale: b1 / dscale from the position's derivative
  const double4 *anchor;  // sorted groups: anchor, packed first site and site masks
  const double4 *sr;      // slots: offset from the anchor, charge
  const double4 *sp;      // slots: sig, sqrt(eps), rscreen, -
  const int *nbr, *nbr_count, *sorted;
  const int *gexcl_ptr, *gexcl_idx, *excl_ptr, *excl_idx;
  unsigned long long *counter;  // next row; zeroed by k_sort_sites
  double *phi, *evec, *ljf, *lj_row;
  double *vir_row;        // per row: the virial's pair term (mmnb_virial)
  const double *cheb_d;   // 512 x 4: cubics of -eta d/d(eta) of the table (mmnb_virial)
};

// bytes of a warp's queues
constexpr int p64_warp_bytes(bool screen, bool gexcl, bool vir)
{
  return kP64Ring * (16 * 2 + 16 * 4 + 16 * 4 + 8 + (vir ? 16 : 0) + (screen ? 8 : 0) + 4 * 2 + (gexcl ? 4 * 3 : 0)) +
         (gexcl ? 8 * kMaxGroup : 0);
}

// b0 = erfc(eta r)/r and g with b1 = dscale g, b1 = -2 d b0 / d(r^2); seg and f:
// table segment and position in it, seg = -1 outside the table
__device__ __forceinline__ void ewald_p64(const PairArgs &a, const double2 *t0, const double2 *t1, double r2,
                                          double &b0, double &g, int &seg, double &f)
{
  const double x = (r2 - a.cmin) * a.inv_dx;
  if (x > 0 && x < kCheb) {
    // floor(x) exactly: x + 2^52 rounded down holds floor(x) in its low word
    const double t = __dadd_rd(x, 4503599627370496.0);
    const int i = __double2loint(t);
    f = x - (t - 4503599627370496.0);
    seg = i;
    const double2 c01 = t0[i * a.copies], c23 = t1[i * a.copies];
    b0 = ((c23.y * f + c23.x) * f + c01.y) * f + c01.x;
    g = fma(fma(c23.y, 3 * f, c23.x + c23.x), f, c01.y);
    return;
  }
  seg = -1;
  f = 0;
  const double y = (r2 - a.tmin) * a.tail_inv;
  if (x <= 0 && a.series) {
    ewald_short(a.eta2, a.cerf, r2, b0, g);
    g *= a.inv_dscale;
  } else if (x > 0 && y < a.tail_nseg) {
    const int i = (int) y;
    const double u = fma(2.0, y - i, -1.0);
    const double2 *const c = a.tail + 4 * i;
    const double2 c01 = __ldg(c), c23 = __ldg(c + 1), c45 = __ldg(c + 2), c67 = __ldg(c + 3);
    const double k[8] = {c01.x, c01.y, c23.x, c23.y, c45.x, c45.y, c67.x, c67.y};
    double p = k[7], d = 0;
#pragma unroll
    for (int n = 6; n >= 0; n--) {
      d = fma(d, u, p);
      p = fma(p, u, k[n]);
    }
    b0 = p;
    g = d * a.tscale;
  } else {
    const double r = sqrt(r2);
    const double er = a.eta * r;
    b0 = erfc(er) / r;
    g = (b0 + a.cerf * exp(-(er * er))) / r2 * a.inv_dscale;
  }
}

__device__ __forceinline__ int nth_bit(int m, int n)
{
  for (; n > 0; n--)
    m &= m - 1;
  return __ffs(m) - 1;
}

__device__ __forceinline__ void team_sync(int team, int threads)
{
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(threads) : "memory");
}

template <bool SCREEN, bool GEXCL, bool VIR>
__global__ void __launch_bounds__(32 * kP64Warps, 1) k_pair_fp64(PairArgs a)
{
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int next_row[kP64Warps];
  constexpr int kMask = kP64Ring - 1, kBytes = p64_warp_bytes(SCREEN, GEXCL, VIR);
  double2 *const tab = reinterpret_cast<double2 *>(smem);
  for (int i = threadIdx.x; i < 2 * kCheb * a.copies; i += blockDim.x) {
    const int k = i / a.copies;
    tab[i] = a.table[k < kCheb ? k : a.half + k - kCheb];
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // this lane's copy of the table
  const double2 *const t0 = tab + lane % a.copies, *const t1 = t0 + kCheb * a.copies;
  unsigned char *const base_w = smem + sizeof(double2) * 2 * kCheb * a.copies;
  auto queues = [&](int warp) { return reinterpret_cast<double2 *>(base_w + (size_t) warp * kBytes); };
  // queued partners: (x, y), (z, r^2) of the anchor displacement
  double2 *const ga = queues(w), *const gb = ga + kP64Ring;
  // queued charged sites: position relative to the row's anchor, q, q S and the
  // switch derivative times the displacement: (ux, uy), (uz, q), (q S, gx), (gy, gz)
  double2 *const q0 = gb + kP64Ring, *const q1 = q0 + kP64Ring, *const q2 = q1 + kP64Ring, *const q3 = q2 + kP64Ring;
  // queued LJ sites: (ux, uy), (uz, sig), (sqrt(eps), S), (gx, gy), gz
  double2 *const l0 = q3 + kP64Ring, *const l1 = l0 + kP64Ring, *const l2 = l1 + kP64Ring, *const l3 = l2 + kP64Ring;
  double *const l4 = reinterpret_cast<double *>(l3 + kP64Ring);
  double *const qg = l4 + kP64Ring, *const lg = qg + (VIR ? kP64Ring : 0);  // VIR: dS r^2
  double *const qrs = lg + (VIR ? kP64Ring : 0);
  int *const gj = reinterpret_cast<int *>(qrs + (SCREEN ? kP64Ring : 0)), *const gm = gj + kP64Ring;
  // group exclusions: the partner's first site; 1 + site of a queued site that may be excluded
  int *const gs = gm + kP64Ring, *const qx = gs + kP64Ring, *const lx_ = qx + kP64Ring;
  unsigned long long *const xmask = reinterpret_cast<unsigned long long *>(lx_ + kP64Ring);  // per row site
  // sums of a row: per-lane values over the charged sites' queue, the totals over the LJ sites'
  double *const red = reinterpret_cast<double *>(q0);
  double *const tot = reinterpret_cast<double *>(l0);
  static_assert(32 * 13 * sizeof(double) <= 4 * kP64Ring * sizeof(double2), "sums do not fit");
  const unsigned below = (1u << lane) - 1;
  const int split = a.split, sub = w & (split - 1), team = w / split;
  const int eg = lane / a.width, ek = lane - eg * a.width;  // expansion: partner and site of this lane
  __syncthreads();
  for (;;) {
    int p = 0;
    if (split == 1) {
      if (lane == 0)
        p = (int) atomicAdd(a.counter, 1ull);
      p = __shfl_sync(0xffffffffu, p, 0);
    } else {
      if (sub == 0 && lane == 0)
        next_row[team] = (int) atomicAdd(a.counter, 1ull);
      team_sync(team, 32 * split);
      p = next_row[team];
    }
    if (p >= a.ngroup)
      break;
    const double4 ai = a.anchor[p];
    const long long info = __double_as_longlong(ai.w);
    const int si0 = (int) (info >> 32), ns = (int) info & 0xff, qm = ((int) info >> 8) & 0xff,
              lm = ((int) info >> 16) & 0xff;
    // sites excluded in other groups: whether any; where the row's lists are (first: what
    // the row's set-up waits for)
    const bool row_gx = GEXCL && ((int) info >> 24) & 1;
    int xb = 0, xe = 0;
    if (row_gx && lane < ns) {
      xb = a.excl_ptr[si0 + lane];
      xe = a.excl_ptr[si0 + lane + 1];
    }
    const int cnt = a.nbr_count[p];
    const int *row = a.nbr + (size_t) p * a.rowcap;
    const int step = 32 * split;
    // entries past the row end read the row's own group (a valid address)
    int base = 32 * sub;
    int jc = base + lane < cnt ? row[base + lane] : p;
    int jn = base + step + lane < cnt ? row[base + step + lane] : p;
    double4 ac = a.anchor[jc];
    const int nq = __popc(qm), nl = __popc(lm);
    const int Pq = nq ? 32 / nq : 0, Pl = nl ? 32 / nl : 0;
    // this lane's row sites and the partner site it takes of a step
    const int iq = nq ? lane / Pq : 0, il = nl ? lane / Pl : 0;
    const int sq = lane - iq * Pq, sl = lane - il * Pl;
    const bool aq = iq < nq, al = il < nl;
    const int kq = aq ? nth_bit(qm, iq) : 0, kl = al ? nth_bit(lm, il) : 0;
    const double4 vq = a.sr[(size_t) p * a.G + kq], vl = a.sr[(size_t) p * a.G + kl];
    const double4 pl = a.sp[(size_t) p * a.G + kl];
    const double rsi = SCREEN ? a.sp[(size_t) p * a.G + kq].z : 0.0;
    // The first and the last site that any site of the row excludes.  Up to 64 sites apart,
    // each row site's as a mask from the first on; a row of one site then drops what it
    // excludes before the queues.  (A search per partner and per site pair, chains of
    // dependent loads that the other lanes wait for, in chains of 64,000 single sites that
    // exclude three to each side: the pair kernel 1247 us, 820 so.)
    int xlo = 1 << 30, xhi = -1;
    unsigned long long xone = 0;
    if (row_gx) {
      if (xb < xe) {
        xlo = a.excl_idx[xb];
        xhi = a.excl_idx[xe - 1];
      }
      xlo = __reduce_min_sync(0xffffffffu, xlo);
      xhi = __reduce_max_sync(0xffffffffu, xhi);
    }
    const bool masks = xhi - xlo < 64, single = masks && ns == 1;
    if (row_gx && single) {
      const int b = __shfl_sync(0xffffffffu, xb, 0), e = __shfl_sync(0xffffffffu, xe, 0);
      for (int n = b + lane; n < e; n += 32)
        xone |= 1ull << (a.excl_idx[n] - xlo);
      xone = (unsigned long long) __reduce_or_sync(0xffffffffu, (unsigned) (xone >> 32)) << 32 |
             __reduce_or_sync(0xffffffffu, (unsigned) xone);
    } else if (row_gx && masks && lane < ns) {
      unsigned long long m = 0;
      for (int n = xb; n < xe; n++)
        m |= 1ull << (a.excl_idx[n] - xlo);
      xmask[lane] = m;
    }
    const bool late = row_gx && !single;  // site pairs are looked at in the queues
    // whether site k of the row excludes site j
    auto excluded = [&](int k, int j) {
      return masks ? (unsigned) (j - xlo) < 64u && (xmask[k] >> (j - xlo)) & 1
                   : csr_has(a.excl_ptr, a.excl_idx, si0 + k, j);
    };
    double ph = 0, ex = 0, ey = 0, ez = 0, sx = 0, sy = 0, sz = 0;  // charges; s: switch force / q_i
    double lx = 0, ly = 0, lz = 0, tx = 0, ty = 0, tz = 0, elj = 0, vir = 0;
    int gh = 0, gn = 0, qh = 0, qn = 0, lh = 0, ln = 0;
    // walk the list until a batch of partners is queued
    auto fill = [&]() {
      while (gn < a.batch && base < cnt) {
        const int e2 = base + 2 * step + lane;
        const int jnn = e2 < cnt ? row[e2] : p;
        const double4 an = a.anchor[jn];
        double x, y, z, hx, hy, hz;
        const double r2a = anchor_disp(a.box, ai, ac, x, y, z, hx, hy, hz);
        const bool take = base + lane < cnt && r2a <= a.rhi2;
        const unsigned bal = __ballot_sync(0xffffffffu, take);
        if (take) {
          const int k = (gh + gn + __popc(bal & below)) & kMask;
          ga[k] = make_double2(x, y);
          gb[k] = make_double2(z, r2a);
          gj[k] = jc;
          int m = (int) __double_as_longlong(ac.w) & 0xffffff;
          if (row_gx) {
            const int s0 = (int) (__double_as_longlong(ac.w) >> 32);
            gs[k] = s0;
            if (s0 <= xhi && s0 + (m & 0xff) > xlo &&
                (masks || csr_has(a.gexcl_ptr, a.gexcl_idx, a.sorted[p], a.sorted[jc])))
              m |= 1 << 24;
          }
          gm[k] = m;
        }
        gn += __popc(bal);
        base += step;
        jc = jn;
        jn = jnn;
        ac = an;
      }
      __syncwarp();
    };
    // a batch's site records, on their way while the queue before them is evaluated
    double4 s = make_double4(0, 0, 0, 0), sp = s;
    int em = 0, en = 0;  // site mask bits (1: charge, 2: LJ, 4: may be excluded), partners of the batch
    auto load = [&]() {
      en = min(gn, a.batch);
      em = 0;
      if (eg < en) {
        const int k = (gh + eg) & kMask, m = gm[k];
        em = ((m >> (8 + ek)) & 1 && nq ? 1 : 0) | ((m >> (16 + ek)) & 1 && nl ? 2 : 0);
        if (em) {
          const size_t slot = (size_t) gj[k] * a.G + ek;
          s = a.sr[slot];
          if (SCREEN || (em & 2))
            sp = a.sp[slot];
          if (GEXCL && (m >> 24) & 1) {
            const unsigned d = gs[k] + ek - xlo;
            em = !single ? em | 4 : d < 64 && (xone >> d) & 1 ? 0 : em;
          }
        }
      }
    };
    auto push = [&]() {
      const unsigned bq = __ballot_sync(0xffffffffu, em & 1), bl = __ballot_sync(0xffffffffu, em & 2);
      if (em) {
        const int k = (gh + eg) & kMask;
        const double2 xy = ga[k], zr = gb[k];
        const double zz = fmax(zr.y - a.rlo2, 0.0) * a.inv_sw;
        const double S = ((-6 * zz + 15) * zz - 10) * zz * zz * zz + 1;
        const double ds = ((60 * zz - 120) * zz + 60) * zz * zz * a.inv_sw;
        const double ux = s.x - xy.x, uy = s.y - xy.y, uz = s.z - zr.x;
        if (em & 1) {
          const int e = (qh + qn + __popc(bq & below)) & kMask;
          q0[e] = make_double2(ux, uy);
          q1[e] = make_double2(uz, s.w);
          q2[e] = make_double2(s.w * S, ds * xy.x);
          q3[e] = make_double2(ds * xy.y, ds * zr.x);
          if (VIR)
            qg[e] = ds * zr.y;
          if (SCREEN)
            qrs[e] = sp.z;
          if (late)
            qx[e] = em & 4 ? gs[k] + ek + 1 : 0;
        }
        if (em & 2) {
          const int e = (lh + ln + __popc(bl & below)) & kMask;
          l0[e] = make_double2(ux, uy);
          l1[e] = make_double2(uz, sp.x);
          l2[e] = make_double2(sp.y, S);
          l3[e] = make_double2(ds * xy.x, ds * xy.y);
          l4[e] = ds * zr.x;
          if (VIR)
            lg[e] = ds * zr.y;
          if (late)
            lx_[e] = em & 4 ? gs[k] + ek + 1 : 0;
        }
      }
      qn += __popc(bq);
      ln += __popc(bl);
      gh = (gh + en) & kMask;
      gn -= en;
      __syncwarp();
    };
    auto eval_q = [&](int n) {
      if (aq && sq < n) {
        const int e = (qh + sq) & kMask;
        const double2 e0 = q0[e], e1 = q1[e], e2 = q2[e], e3 = q3[e];
        const bool out = late && qx[e] && excluded(kq, qx[e] - 1);
        if (!out) {
          const double dx = vq.x - e0.x, dy = vq.y - e0.y, dz = vq.z - e1.x;
          const double r2 = dx * dx + dy * dy + dz * dz;
          double b0, g, f;
          int seg;
          ewald_p64(a, t0, t1, r2, b0, g, seg, f);
          if (VIR && seg >= 0) {
            // the table is refitted for each eta: its eta derivative along the
            // volume-move path is the fitted cubic, not b1 r^2 - b0, the identity
            // of the exact function that mmnb_virial's scale covariance assumes
            const double2 *dc = reinterpret_cast<const double2 *>(a.cheb_d) + 2 * seg;
            const double2 d01 = __ldg(dc), d23 = __ldg(dc + 1);
            const double dd = ((d23.y * f + d23.x) * f + d01.y) * f + d01.x;
            vir -= 0.5 * vq.w * e2.x * (dd - (g * a.dscale * r2 - b0));
          }
          if (SCREEN) {
            const double rs = rsi + qrs[e];
            if (r2 < rs * rs) {
              const double invr = 1.0 / sqrt(r2), inv3 = 1.0 / (rs * rs * rs);
              b0 += (-0.5 * r2 * inv3 + 1.5 / rs) - invr;
              g += (inv3 - invr * invr * invr) * a.inv_dscale;
            }
          }
          const double qb = e1.y * b0, fb = e2.x * g;
          ph += e2.x * b0;
          ex += fb * dx;
          ey += fb * dy;
          ez += fb * dz;
          sx += qb * e2.y;
          sy += qb * e3.x;
          sz += qb * e3.y;
          if (VIR)
            vir += 0.5 * vq.w * qb * qg[e];
        }
      }
      qh = (qh + n) & kMask;
      qn -= n;
    };
    auto eval_l = [&](int n) {
      if (al && sl < n) {
        const int e = (lh + sl) & kMask;
        const double2 e0 = l0[e], e1 = l1[e], e2 = l2[e], e3 = l3[e];
        const double gz = l4[e];
        const bool out = late && lx_[e] && excluded(kl, lx_[e] - 1);
        if (!out) {
          const double dx = vl.x - e0.x, dy = vl.y - e0.y, dz = vl.z - e1.x;
          const double ir2 = 1.0 / (dx * dx + dy * dy + dz * dz);
          const double sg = a.geometric ? pl.x * e1.y : (0.5 * (pl.x + e1.y)) * (0.5 * (pl.x + e1.y));
          const double s6 = sg * sg * sg;
          const double b = 4 * (pl.y * e2.x) * s6;
          const double ir6 = ir2 * ir2 * ir2;
          const double b6 = b * ir6, a12 = b * s6 * ir6 * ir6;
          const double u = a12 - b6;
          const double du6 = (12 * a12 - 6 * b6) * e2.y;  // force scalar times r^2, switched
          const double du = du6 * ir2;
          elj += 0.5 * (u * e2.y);
          lx += du * dx;
          ly += du * dy;
          lz += du * dz;
          tx += u * e3.x;
          ty += u * e3.y;
          tz += u * gz;
          if (VIR)
            vir += 0.5 * (du6 + u * lg[e]);
        }
      }
      lh = (lh + n) & kMask;
      ln -= n;
    };
    fill();
    load();
    while (en > 0) {
      push();
      fill();
      load();
      while (nq && qn >= Pq)
        eval_q(Pq);
      while (nl && ln >= Pl)
        eval_l(Pl);
      __syncwarp();  // the slots are free again only after every lane has read them
    }
    if (qn > 0)
      eval_q(qn);
    if (ln > 0)
      eval_l(ln);
    __syncwarp();
    // the row's sums: charged site i over lanes [i Pq, (i + 1) Pq), LJ site i over
    // [i Pl, ...), the anchor's switch force and the energies over all lanes
    {
      double *const v = red + lane * 13;
      v[0] = ph;
      v[1] = ex;
      v[2] = ey;
      v[3] = ez;
      v[4] = lx;
      v[5] = ly;
      v[6] = lz;
      v[7] = vq.w * sx + tx;
      v[8] = vq.w * sy + ty;
      v[9] = vq.w * sz + tz;
      v[10] = elj;
      v[11] = vir;
    }
    __syncwarp();
    const int nt = 4 * nq + 3 * nl + 5;
    for (int t = lane; t < nt; t += 32) {
      int c, from, n;
      if (t < 4 * nq) {
        c = t & 3;
        from = (t >> 2) * Pq;
        n = Pq;
      } else if (t < 4 * nq + 3 * nl) {
        const int i = (t - 4 * nq) / 3;
        c = 4 + t - 4 * nq - 3 * i;
        from = i * Pl;
        n = Pl;
      } else {
        c = 7 + t - 4 * nq - 3 * nl;
        from = 0;
        n = 32;
      }
      double sum = 0;
#pragma unroll 8
      for (int l = 0; l < n; l++)
        sum += red[(from + l) * 13 + c];
      tot[t] = sum;
    }
    if (split == 1) {
      __syncwarp();
    } else {
      team_sync(team, 32 * split);
      if (sub == 0) {
        for (int t = lane; t < nt; t += 32) {
          double sum = tot[t];
          for (int o = 1; o < split; o++)
            sum += reinterpret_cast<const double *>(queues(w + o) + (l0 - ga))[t];
          tot[t] = sum;
        }
        __syncwarp();
      }
    }
    if (sub == 0) {
      const int tl = 4 * nq, tt = tl + 3 * nl;
      for (int o = lane; o < 7 * ns; o += 32) {
        const int k = o / 7, c = o - 7 * k, site = si0 + k, before = (1 << k) - 1;
        if (c < 4) {
          const double x = (qm >> k) & 1 ? tot[4 * __popc(qm & before) + c] : 0.0;
          if (c == 0)
            a.phi[site] = x;
          else
            a.evec[3 * site + c - 1] = x * a.dscale;
        } else {
          double x = (lm >> k) & 1 ? tot[tl + 3 * __popc(lm & before) + c - 4] : 0.0;
          if (k == 0)
            x += tot[tt + c - 4];
          a.ljf[3 * site + c - 4] = x;
        }
      }
      if (lane == 0) {
        a.lj_row[p] = tot[tt + 3];
        if (VIR)
          a.vir_row[p] = tot[tt + 4];
      }
    }
    if (split == 1)
      __syncwarp();  // the queues are the next row's again only after every lane has read them
    // (a team's warps meet again before the next row's first write: the row's number)
  }
}

// Sorted FP64 site data for the pair kernel: slots of (offset from the anchor,
// charge) and (sigma, sqrt(epsilon), r_screen, -), and per group the anchor with
// its first site (high word) and number of sites, charged sites and LJ sites (a
// byte each of the low word: bit k for site k), and bit 24 for exclusions across groups
// (gexcl_ptr, or null without any).  Clears the row counter.
__device__ __forceinline__ void sort_sites(const double *__restrict__ r, const double *__restrict__ q,
                             const double *__restrict__ sig, const double *__restrict__ eps,
                             const double *__restrict__ rscreen, const int *__restrict__ mask,
                             const int *__restrict__ sorted, const int *__restrict__ group,
                             const int *__restrict__ gexcl_ptr, int ngroup, int G,
                             double4 *__restrict__ sr, double4 *__restrict__ sp, double4 *__restrict__ anchor,
                             unsigned long long *__restrict__ counter, int *__restrict__ flags)
{
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0)
    *counter = 0ull;
  if (s >= ngroup * G)
    return;
  const int p = s / G, k = s % G;
  const int g = sorted[p];
  const int s0 = group[2 * g], n = group[2 * g + 1] - s0;
  const double ax = r[3 * s0], ay = r[3 * s0 + 1], az = r[3 * s0 + 2];
  if (k == 0) {
    unsigned m = n;
    if (gexcl_ptr && gexcl_ptr[g + 1] > gexcl_ptr[g])
      m |= 1u << 24;
    for (int j = 0; j < n; j++) {
      const int b = mask[s0 + j];
      m |= (b & MMNB_SITE_HAS_Q ? 1u << (8 + j) : 0u) | (b & MMNB_SITE_HAS_LJ ? 1u << (16 + j) : 0u);
    }
    anchor[p] = make_double4(ax, ay, az, __longlong_as_double((long long) s0 << 32 | m));
  }
  if (k < n) {
    const int site = s0 + k;
    const double x = r[3 * site], y = r[3 * site + 1], z = r[3 * site + 2];
    if (!isfinite(x) || !isfinite(y) || !isfinite(z))
      flags[kFlagError] = MMNB_ERR_DEVICE;
    sr[s] = make_double4(x - ax, y - ay, z - az, q[site]);
    sp[s] = make_double4(sig[site], sqrt(eps[site]), rscreen[site], 0.0);
  }
}

__global__ void __launch_bounds__(32 * kRowWarps)
k_sort_sites(const double *__restrict__ r, const double *__restrict__ q, const double *__restrict__ sig,
             const double *__restrict__ eps, const double *__restrict__ rscreen, const int *__restrict__ mask,
             const int *__restrict__ sorted, const int *__restrict__ group, const int *__restrict__ gexcl_ptr,
             int ngroup, int G, double4 *__restrict__ sr, double4 *__restrict__ sp, double4 *__restrict__ anchor,
             unsigned long long *__restrict__ counter, int *__restrict__ flags, RebuildArgs rows)
{
  after_previous();
  sort_sites(r, q, sig, eps, rscreen, mask, sorted, group, gexcl_ptr, ngroup, G, sr, sp, anchor, counter, flags);
  build_rows(rows);
}

cudaError_t launch_sort_sites(mmnb_handle *h, const double *d_r)
{
  const int n = h->ngroup * h->G;
  launch_after(h, k_sort_sites, sort_blocks(h, n), 32 * kRowWarps, 0, d_r, h->d_q, h->d_sig, h->d_eps,
               h->d_rscreen, h->d_mask, h->d_sorted, h->d_group, h->any_gexcl ? h->d_gexcl_ptr : nullptr,
               h->ngroup, h->G, h->d_sr, h->d_sp, h->d_sanchor, h->d_wsum + 3, h->d_flags, rebuild_args(h));
  h->launches += 1;
  return cudaGetLastError();
}

template <bool SCREEN, bool GEXCL, bool VIR>
static cudaError_t launch_pair64(mmnb_handle *h, PairArgs &a)
{
  cudaError_t e;
  int nsm = 0, optin = 0;
  if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->dev)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->dev)) != cudaSuccess)
    return e;
  // small systems: teams of two or four warps per row, as long as the chip holds
  // every team at once (9^3 cells of solution: 27 us with 2, 41 us with 4, where it
  // does not), and blocks no larger than it takes to cover the SMs
  const long chip = (long) nsm * kP64Warps;
  a.split = h->ngroup * 4L <= chip ? 4 : h->ngroup * 2L <= chip ? 2 : 1;
  int warps = std::min(kP64Warps, (div_up((long) h->ngroup * a.split, nsm) + 3) / 4 * 4);
  const int per = p64_warp_bytes(SCREEN, GEXCL, VIR);
  const size_t table = sizeof(double2) * 2 * kCheb, room = (size_t) optin - 1024;
  while (warps > 4 && table + (size_t) warps * per > room)
    warps -= 4;
  // a second copy of the table, interleaved so that two lanes of a 16-byte access
  // phase seldom meet in a bank, where it fits and a warp takes enough rows to fill
  // it for (465 -> 455 us on 32^3 cells of solution)
  a.copies = (long) h->ngroup >= 2L * nsm * warps && 2 * table + (size_t) warps * per <= room ? 2 : 1;
  const size_t smem = a.copies * table + (size_t) warps * per;
  if ((e = cudaFuncSetAttribute(k_pair_fp64<SCREEN, GEXCL, VIR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int) room)) != cudaSuccess)
    return e;
  const int grid = std::min(nsm, div_up((long) h->ngroup * a.split, warps));
  launch_after(h, k_pair_fp64<SCREEN, GEXCL, VIR>, grid, 32 * warps, smem, a);
  h->launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_rspace_fp64(mmnb_handle *h)
{
  PairArgs a;
  a.ngroup = h->ngroup;
  a.rowcap = h->rowcap;
  a.geometric = h->cfg.geometric_combining_for_sigma;
  a.G = h->G;
  a.width = h->maxgs;
  a.batch = 32 / h->maxgs;
  a.half = h->cheb_w_nseg;
  a.tail = reinterpret_cast<const double2 *>(h->d_cheb_w) + 2 * h->cheb_w_nseg;
  a.tmin = h->cheb_max;
  a.tail_inv = h->tail_inv;
  a.tail_nseg = h->tail_nseg;
  a.tscale = 2 * h->tail_inv * (-2.0) / (-2 * h->cheb_inv_dx);
  a.series = h->eta * sqrt(h->cheb_min) <= kErfSeriesMax;
  a.box = h->box;
  a.rlo2 = h->rlo2;
  a.rhi2 = h->rhi2;
  a.inv_sw = h->inv_sw;
  a.eta = h->eta;
  a.eta2 = h->eta * h->eta;
  a.cerf = h->eta * M_2_SQRTPI;
  a.cmin = h->cheb_min;
  a.inv_dx = h->cheb_inv_dx;
  a.dscale = -2 * h->cheb_inv_dx;
  a.inv_dscale = 1.0 / a.dscale;
  a.table = reinterpret_cast<const double2 *>(h->d_cheb_w);
  a.anchor = h->d_sanchor;
  a.sr = h->d_sr;
  a.sp = h->d_sp;
  a.nbr = h->d_nbr;
  a.nbr_count = h->d_nbr_count;
  a.sorted = h->d_sorted;
  a.gexcl_ptr = h->d_gexcl_ptr;
  a.gexcl_idx = h->d_gexcl_idx;
  a.excl_ptr = h->d_excl_ptr;
  a.excl_idx = h->d_excl_idx;
  a.counter = h->d_wsum + 3;
  a.phi = h->d_phi;
  a.evec = h->d_evec;
  a.ljf = h->d_ljf;
  a.lj_row = h->d_lj_row;
  a.vir_row = h->d_vir_row;
  a.cheb_d = h->d_cheb_d;
  if (h->want_virial) {
    // (mmnb_virial refuses screened charges)
    return h->any_gexcl ? launch_pair64<false, true, true>(h, a) : launch_pair64<false, false, true>(h, a);
  }
  if (h->has_rscreen)
    return h->any_gexcl ? launch_pair64<true, true, false>(h, a) : launch_pair64<true, false, false>(h, a);
  return h->any_gexcl ? launch_pair64<false, true, false>(h, a) : launch_pair64<false, false, false>(h, a);
}

}  // namespace mmnb
