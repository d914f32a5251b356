// Real-space Ewald + Lennard-Jones for rigid 3-site water, FP64 form.
//
// The group-pair semantics of RSpaceEwald (src/rspace.c:413-491), evaluated
// for groups [O(q, LJ), H(q), H(q)] (ElecLJ's groups for water,
// src/eleclj.cpp:654-676):
//   * the anchor (O) displacement, its minimum-image shift and the cutoff test
//     use the reference's rounding (anchor_disp), so the evaluated group pairs
//     are the reference's;
//   * every site pair uses the anchors' image shift; the quintic switch S and
//     dS/dr^2 come from the anchor distance, multiply the Coulomb and LJ terms,
//     and dS times the summed unswitched energy acts on the anchors (:479-489);
//   * b0 = erfc(eta r)/r comes from the reference's 512-segment Chebyshev cubic
//     in r^2 (src/rspace.c:25-37, src/cheby.c:7-45) and b1 = -2 db0/d(r^2) from
//     the derivative of that same cubic -- the reference stores the derivative
//     coefficients (-2 c1, -4 c2, -6 c3)/(b - a) beside the cubic; here they are
//     formed from the cubic's own coefficients and the segment width, which
//     agrees to rounding (the table's b1 is not the exact field term: it differs
//     from it by up to ~1e-5 relative at short range, so the table, not an exact
//     erfc, is what reproduces the reference);
//   * past the table's upper end (r^2 > 1.2 rc^2, which only site pairs of
//     water reach) the table continues with segments of the same construction
//     where that is as good as the erfc and exp the reference evaluates there
//     (table_segments), and below its lower end (r^2 < 4) they are exact
//     (ewald_short).
//
// Layout: a persistent grid, one block of up to kW64Warps warps per SM; each
// warp takes the next row group from a counter and walks its list 32 entries
// at a time (anchor test per lane, ballot compaction into a 128-slot ring of
// anchor displacements, cp.async of the partner's record -- its H offsets where
// every water has the same parameters -- into the same slot, an array per 16-byte
// word), evaluating 32 queued group pairs at a time.  The table's two halves,
// (c0, c1) and (c2, c3) per segment, sit in shared memory as two arrays of
// 16-byte entries in up to eight interleaved copies (a lane reads copy lane mod
// copies, so that the eight lanes of an access phase meet in a bank less often;
// four fit beside twelve warps' rings at rc 9).  Row totals are summed over the
// lanes in a fixed order (transpose through shared memory), so results do not
// depend on which warp or SM took the row.
//
// Bound by the shared-memory pipe and FP64 latency at 12 warps per SM.  On 32,768
// waters: 259 us with 32-byte ring words, one table and erfc below it; 226 with
// erf's series there (ewald_short); 191 with word arrays, records of H offsets and
// four copies.  On one row per warp the table's copy-in shows: asynchronous, 21 -> 17
// us on 216 waters.

#include "nbrlist.cuh"

#include <algorithm>

namespace mmnb {

// warps per block the kernel is compiled for (its register budget: 12 warps
// of 384 threads leave 170 registers a thread); a launch may use fewer when
// the rings and the table do not fit in shared memory
constexpr int kW64Warps = 12;
// a batch of 32 is queued before the oldest 32 are evaluated, so the ring
// holds up to 63 + 32 entries
constexpr int kW64Ring = 128;
constexpr int kW64Acc = 17;  // phi (3), field (9), LJ + switch force on O (3), LJ energy, virial term

struct Water64Args {
  int ngroup, rowcap, geometric, nseg, copies, series;
  Box box;
  double rlo2, rhi2, inv_sw, eta;
  double cmin, inv_dx, dscale, nsegd;  // dscale = -2 / segment width
  const double2 *table;                // [nseg] (c0, c1), then [nseg] (c2, c3)
  const double4 *anchor;               // sorted groups: anchor (x, y, z, -)
  const double2 *rec;                  // sorted groups: 6 x double2, layout in k_sort_water64
  double qO, qH, sig, seps;            // uniform water: charges and LJ parameters
  const int *nbr, *nbr_count, *sorted, *group;
  unsigned long long *counter;         // next row; zeroed by k_sort_water64
  double *phi, *evec, *ljf, *lj_row;
  double *vir_row;                     // per row: the virial's pair term (mmnb_virial), or null
  const double *cheb_d;                // 512 x 4: cubics of -eta d/d(eta) of the table (mmnb_virial)
};

// b0 = erfc(eta r)/r and b1 = (b0 + 2 eta/sqrt(pi) exp(-eta^2 r^2)) / r^2;
// seg and f: the table segment and the position in it, seg = -1 outside the table
__device__ __forceinline__ void ewald_w64(const Water64Args &a, const double2 *t0, const double2 *t1, double r2,
                                          double &b0, double &b1, int &seg, double &f)
{
  const double x = (r2 - a.cmin) * a.inv_dx;
  if (x > 0 && x < a.nsegd) {
    // floor(x) exactly: x + 2^52 rounded down holds floor(x) in its low word
    const double t = __dadd_rd(x, 4503599627370496.0);
    const int i = __double2loint(t);
    f = x - (t - 4503599627370496.0);
    seg = i;
    const double2 c01 = t0[i * a.copies], c23 = t1[i * a.copies];
    b0 = ((c23.y * f + c23.x) * f + c01.y) * f + c01.x;
    b1 = a.dscale * ((3 * c23.y * f + 2 * c23.x) * f + c01.y);
  } else {
    seg = -1;
    f = 0;
    if (x <= 0 && a.series) {
      ewald_short(a.eta * a.eta, a.eta * M_2_SQRTPI, r2, b0, b1);
    } else {
      const double r = sqrt(r2);
      const double er = a.eta * r;
      b0 = erfc(er) / r;
      b1 = (b0 + a.eta * M_2_SQRTPI * exp(-(er * er))) / r2;
    }
  }
}

// one site pair: d = displacement, qj = partner charge, qjs = qj S.
// VIR: the site pair's part of the virial that scale covariance misses --
// the table is refitted for each eta, so its eta derivative is the fitted
// cubic D of -eta d/d(eta) erfc(eta r)/r, not b1 r^2 - b0 (the identity the
// exact function obeys); qis = q_i S, added to the virial term with the
// factor -1/2 (the full list sees each pair twice)
template <bool VIR>
__device__ __forceinline__ void site_w64(const Water64Args &a, const double2 *t0, const double2 *t1, double dx,
                                         double dy, double dz, double r2, double qj, double qjs, double &ph,
                                         double &ex, double &ey, double &ez, double &tq, double qis, double &vir)
{
  double b0, b1, f;
  int seg;
  ewald_w64(a, t0, t1, r2, b0, b1, seg, f);
  tq += qj * b0;
  ph += qjs * b0;
  const double fb = qjs * b1;
  ex += fb * dx;
  ey += fb * dy;
  ez += fb * dz;
  if (VIR && seg >= 0 && seg < kCheb) {
    const double2 *dc = reinterpret_cast<const double2 *>(a.cheb_d) + 2 * seg;
    const double2 d01 = __ldg(dc), d23 = __ldg(dc + 1);
    const double dd = ((d23.y * f + d23.x) * f + d01.y) * f + d01.x;
    vir -= 0.5 * qis * qj * (dd - (b1 * r2 - b0));
  }
}

__device__ __forceinline__ void cp16(void *dst, const void *src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"((unsigned) __cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// 16-byte words of a queued partner: anchor displacement and r^2, H offsets and,
// unless every water has the same parameters, charges and LJ parameters
constexpr int w64_words(bool uni) { return uni ? 5 : 8; }

// UNI: every water has the same parameters (taken from the arguments)
template <bool VIR, bool UNI>
__global__ void __launch_bounds__(kW64Warps * 32, 1) k_pair_water64(Water64Args a)
{
  after_previous();
  constexpr int kWords = w64_words(UNI);
  extern __shared__ __align__(16) unsigned char smem[];
  // per warp: ring of (x, y), (z, r^2) of the anchor displacement and the partner's
  // record, one array per 16-byte word: consecutive lanes read consecutive words
  double2 *ring = reinterpret_cast<double2 *>(smem);  // [warps][kWords][kW64Ring]
  double2 *tab = ring + (size_t) kWords * kW64Ring * (blockDim.x >> 5);
  // the table is on its way while the first rows are walked: each warp waits for it
  // (and meets the block) before its first evaluation
  bool table_ready = false;
  if (a.copies == 1) {
    for (int i = threadIdx.x; i < 2 * a.nseg; i += blockDim.x)
      cp16(tab + i, a.table + i);
  } else {
    for (int i = threadIdx.x; i < 2 * a.nseg * a.copies; i += blockDim.x)
      tab[i] = a.table[i / a.copies];
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  auto wait_table = [&]() {
    if (table_ready)
      return;
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    table_ready = true;
  };
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const double2 *const tc01 = tab + lane % a.copies, *const tc23 = tc01 + a.nseg * a.copies;
  double2 *const q = ring + (size_t) w * kWords * kW64Ring;
  const unsigned below = (1u << lane) - 1;
  for (;;) {
    int p = 0;
    if (lane == 0)
      p = (int) atomicAdd(a.counter, 1ull);
    p = __shfl_sync(0xffffffffu, p, 0);
    if (p >= a.ngroup)
      break;
    const double4 ai = a.anchor[p];
    // record: (h1x, h1y), (h1z, h2x), (h2y, h2z), (qO, qH1), (qH2, sigma), (sqrt(eps), -)
    const double2 *const rp = a.rec + 6 * (size_t) p;
    const double2 r0 = rp[0], r1 = rp[1], r2 = rp[2];
    double2 r3 = make_double2(a.qO, a.qH), r4 = make_double2(a.qH, a.sig), r5 = make_double2(a.seps, 0.0);
    if (!UNI) {
      r3 = rp[3];
      r4 = rp[4];
      r5 = rp[5];
    }
    const double h1x = r0.x, h1y = r0.y, h1z = r1.x, h2x = r1.y, h2y = r2.x, h2z = r2.y;
    const double qO = r3.x, qH1 = r3.y, qH2 = r4.x, sgO = r4.y, seO = r5.x;
    double acc[kW64Acc];
#pragma unroll
    for (int c = 0; c < kW64Acc; c++)
      acc[c] = 0;
    auto compute = [&](int k) {
      const double2 *const e = q + k;
      const double2 d0 = e[0], d1 = e[kW64Ring], j0 = e[2 * kW64Ring], j1 = e[3 * kW64Ring], j2 = e[4 * kW64Ring];
      double2 j3 = make_double2(a.qO, a.qH), j4 = make_double2(a.qH, a.sig);
      double sej = a.seps;
      if (!UNI) {
        j3 = e[(UNI ? 0 : 5) * kW64Ring];
        j4 = e[(UNI ? 0 : 6) * kW64Ring];
        sej = e[(UNI ? 0 : 7) * kW64Ring].x;
      }
      const double4 da = make_double4(d0.x, d0.y, d1.x, d1.y);
      const double j1x = j0.x, j1y = j0.y, j1z = j1.x, j2x = j1.y, j2y = j2.x, j2z = j2.y;
      const double qjO = j3.x, qj1 = j3.y, qj2 = j4.x, sgj = j4.y;
      const double r2a = da.w;
      // switch (zero width inside rc - width: s = 1 and ds = 0 exactly there)
      const double zz = fmax(r2a - a.rlo2, 0.0) * a.inv_sw;
      const double s = ((-6 * zz + 15) * zz - 10) * zz * zz * zz + 1;
      const double ds = ((60 * zz - 120) * zz + 60) * zz * zz * a.inv_sw;
      const double qjOs = qjO * s, qj1s = qj1 * s, qj2s = qj2 * s;
      const double qOs = qO * s, qH1s = qH1 * s, qH2s = qH2 * s;
      double tO = 0, t1 = 0, t2 = 0;
      // row O
      site_w64<VIR>(a, tc01, tc23, da.x, da.y, da.z, r2a, qjO, qjOs, acc[0], acc[3], acc[4], acc[5], tO, qOs, acc[16]);
      {
        const double dx = da.x - j1x, dy = da.y - j1y, dz = da.z - j1z;
        site_w64<VIR>(a, tc01, tc23, dx, dy, dz, dx * dx + dy * dy + dz * dz, qj1, qj1s, acc[0], acc[3], acc[4], acc[5], tO, qOs, acc[16]);
      }
      {
        const double dx = da.x - j2x, dy = da.y - j2y, dz = da.z - j2z;
        site_w64<VIR>(a, tc01, tc23, dx, dy, dz, dx * dx + dy * dy + dz * dz, qj2, qj2s, acc[0], acc[3], acc[4], acc[5], tO, qOs, acc[16]);
      }
      // row H1
      {
        const double cx = da.x + h1x, cy = da.y + h1y, cz = da.z + h1z;
        site_w64<VIR>(a, tc01, tc23, cx, cy, cz, cx * cx + cy * cy + cz * cz, qjO, qjOs, acc[1], acc[6], acc[7], acc[8], t1, qH1s, acc[16]);
        double dx = cx - j1x, dy = cy - j1y, dz = cz - j1z;
        site_w64<VIR>(a, tc01, tc23, dx, dy, dz, dx * dx + dy * dy + dz * dz, qj1, qj1s, acc[1], acc[6], acc[7], acc[8], t1, qH1s, acc[16]);
        dx = cx - j2x;
        dy = cy - j2y;
        dz = cz - j2z;
        site_w64<VIR>(a, tc01, tc23, dx, dy, dz, dx * dx + dy * dy + dz * dz, qj2, qj2s, acc[1], acc[6], acc[7], acc[8], t1, qH1s, acc[16]);
      }
      // row H2
      {
        const double cx = da.x + h2x, cy = da.y + h2y, cz = da.z + h2z;
        site_w64<VIR>(a, tc01, tc23, cx, cy, cz, cx * cx + cy * cy + cz * cz, qjO, qjOs, acc[2], acc[9], acc[10], acc[11], t2, qH2s, acc[16]);
        double dx = cx - j1x, dy = cy - j1y, dz = cz - j1z;
        site_w64<VIR>(a, tc01, tc23, dx, dy, dz, dx * dx + dy * dy + dz * dz, qj1, qj1s, acc[2], acc[9], acc[10], acc[11], t2, qH2s, acc[16]);
        dx = cx - j2x;
        dy = cy - j2y;
        dz = cz - j2z;
        site_w64<VIR>(a, tc01, tc23, dx, dy, dz, dx * dx + dy * dy + dz * dz, qj2, qj2s, acc[2], acc[9], acc[10], acc[11], t2, qH2s, acc[16]);
      }
      // O-O Lennard-Jones (src/rspace.c:258-297)
      const double sg = a.geometric ? sgO * sgj : (0.5 * (sgO + sgj)) * (0.5 * (sgO + sgj));
      const double s6 = sg * sg * sg;
      const double b = 4 * (seO * sej) * s6;
      const double aa = b * s6;
      const double invr2 = 1.0 / r2a;
      const double invr6 = invr2 * invr2 * invr2;
      const double binvr6 = b * invr6;
      const double ainvr12 = aa * invr6 * invr6;
      const double du = 12 * ainvr12 * invr2 - 6 * binvr6 * invr2;
      const double u = ainvr12 - binvr6;
      const double tmps = qO * tO + qH1 * t1 + qH2 * t2 + u;
      acc[15] += 0.5 * (u * s);
      const double g = du * s + ds * tmps;
      acc[12] += g * da.x;
      acc[13] += g * da.y;
      acc[14] += g * da.z;
      // the part of dU/ds (box scaling) the site forces do not carry: the LJ and
      // switch force scalar times R^2 (each pair is seen from both rows: half)
      acc[16] += 0.5 * g * r2a;
    };
    const int cnt = a.nbr_count[p];
    const int *row = a.nbr + (size_t) p * a.rowcap;
    // entries past the row end read the row's own group (a valid address)
    int jc = lane < cnt ? row[lane] : p;
    int jn = lane + 32 < cnt ? row[lane + 32] : p;
    double4 ac = a.anchor[jc];
    int head = 0, qn = 0;
    for (int base = 0; base < cnt; base += 32) {
      const int e2 = base + 64 + lane;
      const int jnn = e2 < cnt ? row[e2] : p;
      const double4 an = a.anchor[jn];
      double x, y, z, sx, sy, sz;
      const double r2a = anchor_disp(a.box, ai, ac, x, y, z, sx, sy, sz);
      const bool take = base + lane < cnt && r2a <= a.rhi2;
      const unsigned bal = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int slot = (head + qn + __popc(bal & below)) & (kW64Ring - 1);
        double2 *const e = q + slot;
        e[0] = make_double2(x, y);
        e[kW64Ring] = make_double2(z, r2a);
        const double2 *src = a.rec + 6 * (size_t) jc;
#pragma unroll
        for (int k = 0; k < kWords - 2; k++)
          cp16(e + (2 + k) * kW64Ring, src + k);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      const bool run = qn >= 32;
      qn += __popc(bal);
      if (run) {
        wait_table();
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncwarp();
        compute((head + lane) & (kW64Ring - 1));
        __syncwarp();
        head = (head + 32) & (kW64Ring - 1);
        qn -= 32;
      }
      jc = jn;
      jn = jnn;
      ac = an;
    }
    wait_table();
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncwarp();
    for (; qn > 0; qn -= 32, head = (head + 32) & (kW64Ring - 1))
      if (lane < qn)
        compute((head + lane) & (kW64Ring - 1));
    // row totals: lanes' values transposed through the warp's ring, each of
    // lanes 0..15 adds one column over the 32 lanes in lane order
    __syncwarp();
    double(*red)[kW64Acc + 1] = reinterpret_cast<double(*)[kW64Acc + 1]>(q);
    static_assert(32 * (kW64Acc + 1) * sizeof(double) <= kWords * kW64Ring * sizeof(double2), "ring too small");
#pragma unroll
    for (int c = 0; c < kW64Acc; c++)
      red[lane][c] = acc[c];
    __syncwarp();
    const int si0 = a.group[2 * a.sorted[p]];
    if (lane < kW64Acc) {
      double t = 0;
      for (int l = 0; l < 32; l++)
        t += red[l][lane];
      if (lane < 3)
        a.phi[si0 + lane] = t;
      else if (lane < 12)
        a.evec[3 * si0 + (lane - 3)] = t;
      else if (lane < 15)
        a.ljf[3 * si0 + (lane - 12)] = t;
      else if (lane == 15)
        a.lj_row[p] = t;
      else if (a.vir_row)
        a.vir_row[p] = t;
    } else if (lane < kW64Acc + 6) {
      // the H sites carry no LJ force
      a.ljf[3 * si0 + 3 + (lane - kW64Acc)] = 0;
    }
    __syncwarp();  // the ring is the next row's again only after every lane has read it
  }
  wait_table();  // warps without a row meet the others here
}

// Per step: sorted FP64 anchors and the 96-byte records of the partner side,
// (h1x, h1y, h1z, h2x), (h2y, h2z, qO, qH1), (qH2, sigma_O, sqrt(eps_O), 0) with
// the H positions taken from the anchor O; the row counter is cleared and a
// non-finite coordinate is flagged.
__device__ __forceinline__ void sort_water64(const double *__restrict__ r, const double *__restrict__ q,
                               const double *__restrict__ sig, const double *__restrict__ eps,
                               const int *__restrict__ sorted, const int *__restrict__ group, int ngroup,
                               double4 *__restrict__ anchor, double2 *__restrict__ rec,
                               unsigned long long *__restrict__ counter, int *__restrict__ flags)
{
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p == 0)
    *counter = 0ull;
  if (p >= ngroup)
    return;
  const int a0 = group[2 * sorted[p]];
  const double ax = r[3 * a0], ay = r[3 * a0 + 1], az = r[3 * a0 + 2];
  const double *h1 = r + 3 * (a0 + 1), *h2 = r + 3 * (a0 + 2);
  if (!isfinite(ax + ay + az + h1[0] + h1[1] + h1[2] + h2[0] + h2[1] + h2[2]))
    flags[kFlagError] = MMNB_ERR_DEVICE;
  anchor[p] = make_double4(ax, ay, az, 0.0);
  double2 *const o = rec + 6 * (size_t) p;
  o[0] = make_double2(h1[0] - ax, h1[1] - ay);
  o[1] = make_double2(h1[2] - az, h2[0] - ax);
  o[2] = make_double2(h2[1] - ay, h2[2] - az);
  o[3] = make_double2(q[a0], q[a0 + 1]);
  o[4] = make_double2(q[a0 + 2], sig[a0]);
  o[5] = make_double2(sqrt(eps[a0]), 0.0);
}

__global__ void __launch_bounds__(32 * kRowWarps)
k_sort_water64(const double *__restrict__ r, const double *__restrict__ q, const double *__restrict__ sig,
               const double *__restrict__ eps, const int *__restrict__ sorted, const int *__restrict__ group,
               int ngroup, double4 *__restrict__ anchor, double2 *__restrict__ rec,
               unsigned long long *__restrict__ counter, int *__restrict__ flags, RebuildArgs rows)
{
  after_previous();
  sort_water64(r, q, sig, eps, sorted, group, ngroup, anchor, rec, counter, flags);
  build_rows(rows);
}

cudaError_t launch_sort_water64(mmnb_handle *h, const double *d_r)
{
  launch_after(h, k_sort_water64, sort_blocks(h, h->ngroup), 32 * kRowWarps, 0, d_r, h->d_q, h->d_sig,
               h->d_eps, h->d_sorted, h->d_group, h->ngroup, h->d_sp, reinterpret_cast<double2 *>(h->d_sr),
               h->d_wsum + 3, h->d_flags, rebuild_args(h));
  h->launches += 1;
  return cudaGetLastError();
}

template <bool VIR, bool UNI>
static cudaError_t launch_water64(mmnb_handle *h, Water64Args &a)
{
  cudaError_t e;
  int optin = 0, nsm = 0;
  if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->dev)) != cudaSuccess ||
      (e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->dev)) != cudaSuccess)
    return e;
  // the tuned warps per block, fewer if the rings and this box's table do not fit
  // (the table grows as rc falls)
  const size_t ring = sizeof(double2) * w64_words(UNI) * kW64Ring, table = sizeof(double2) * 2 * (size_t) a.nseg;
  // (and on a small box no more than it takes to cover the SMs: a block's warps
  // share one SM's pipes)
  int warps = std::min(std::min(h->tune.water64_warps, kW64Warps), std::max(4, (div_up(h->ngroup, nsm) + 1) / 2 * 2));
  while (warps > 4 && ring * warps + table > (size_t) optin)
    warps -= 2;
  // as many copies of the table as fit, where a warp takes enough rows to fill
  // them for (below about two, one copy)
  a.copies = (long) h->ngroup >= 2L * nsm * warps ? 8 : 1;
  while (a.copies > 1 && ring * warps + table * a.copies > (size_t) optin)
    a.copies >>= 1;
  if ((e = cudaFuncSetAttribute(k_pair_water64<VIR, UNI>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin)) !=
      cudaSuccess)
    return e;
  launch_after(h, k_pair_water64<VIR, UNI>, std::min(nsm, div_up(h->ngroup, warps)), 32 * warps,
               ring * warps + table * a.copies, a);
  h->launches += 1;
  return cudaGetLastError();
}

cudaError_t launch_rspace_water64(mmnb_handle *h)
{
  Water64Args a;
  a.ngroup = h->ngroup;
  a.rowcap = h->rowcap;
  a.geometric = h->cfg.geometric_combining_for_sigma;
  a.nseg = h->cheb_w_nseg;
  a.series = h->eta * sqrt(h->cheb_min) <= kErfSeriesMax;
  a.box = h->box;
  a.rlo2 = h->rlo2;
  a.rhi2 = h->rhi2;
  a.inv_sw = h->inv_sw;
  a.eta = h->eta;
  a.cmin = h->cheb_min;
  a.inv_dx = h->cheb_inv_dx;
  a.dscale = -2 * h->cheb_inv_dx;
  a.nsegd = table_segments(h);
  a.table = reinterpret_cast<const double2 *>(h->d_cheb_w);
  a.anchor = h->d_sp;
  a.rec = reinterpret_cast<const double2 *>(h->d_sr);
  a.qO = h->uni64[0];
  a.qH = h->uni64[1];
  a.sig = h->uni64[2];
  a.seps = h->uni64[3];
  a.nbr = h->d_nbr;
  a.nbr_count = h->d_nbr_count;
  a.sorted = h->d_sorted;
  a.group = h->d_group;
  a.counter = h->d_wsum + 3;
  a.phi = h->d_phi;
  a.evec = h->d_evec;
  a.ljf = h->d_ljf;
  a.lj_row = h->d_lj_row;
  a.vir_row = h->want_virial ? h->d_vir_row : nullptr;
  a.cheb_d = h->d_cheb_d;
  if (h->want_virial)
    return h->water_uni ? launch_water64<true, true>(h, a) : launch_water64<true, false>(h, a);
  return h->water_uni ? launch_water64<false, true>(h, a) : launch_water64<false, false>(h, a);
}

}  // namespace mmnb
