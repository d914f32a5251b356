// Ordinary Ewald reciprocal sum (replaces kspace_new / kspace_field,
// src/kspace.c:35-174; kspace_phi at points, :176-250): the evaluation's
// reciprocal space when use_p3m is off, the potential at points, and the
// adjoint's dipole solve.
//
// Wave vectors are the half space of integer n with |n|^2 <= kc^2 + 1e-8,
// k = 2 pi n / L, a_k = (4 pi / V) exp(-k^2 / 4 eta^2) / k^2.  With
// S(k) = sum_i q_i exp(i k.r_i), a site or point at r gets
//   phi += sum_k 2 a_k Re(S(k) exp(-i k.r)),  E += sum_k 2 a_k k Im(...).
//
// exp(i k.r) is the product of three axis phases exp(2 pi i n x / L), so a
// tile's phases (n = 0..nmax per axis) are tabulated in shared memory -- one
// sine and cosine per site and axis, the powers by products of two lower ones,
// about log2(n) roundings deep -- and a (k, site) term costs two complex
// products (8 FP64 operations) where a sine and cosine of k.r cost ~70.  The
// wave vectors are kept as rows of consecutive n_z at one (n_x, n_y): the
// summing kernel forms the (x, y) phase once per row and +n_z, -n_z from the
// same four products.
//
//   * k_ewald_structure: a thread per wave vector and a tile of sites in the
//     table, one partial S(k) per block of tiles;
//   * k_ewald_reduce: the partials in block order (bitwise reproducible), times
//     2 a_k;
//   * k_ewald_sum: a lane per site or point, the rows dealt to the block's
//     warps, the warps' sums added in warp order.
//
// Bound by latency at these sizes (a warp's chain of table reads and FP64
// products).  Measured against a sine and cosine per (k, site) with one thread per
// site over all wave vectors: 648 sites, 709 wave vectors: the field 256 -> 11 us
// (its six blocks walked a serial chain of 709 terms), the structure factor 6.3
// -> 7.2 + 3.9 us but now beside the list and pair kernels; 12,288 sites and 5,000
// points, 462 wave vectors: structure factor 49 -> 15.3 + 6.9 us, potential 154 ->
// 8.9 us.  S(k) staged in shared memory: 15.2 -> 11.0 and 11.8 -> 8.9 us of that.

#include "mmnb_internal.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace mmnb {

constexpr int kEwThreads = 256;          // structure factor: wave vectors per block
constexpr int kEwWarps = 8;              // summing kernel: warps per block of 32 sites
constexpr int kEwTable = 36 << 10;       // bytes of a block's phase tables of more than one site
// kspace_cutoff from which the wave vectors, 2/3 pi n^3, are more than an int counts; below
// it one site's table and the structure factor's dipole weights fit the default 48 KB
constexpr int kEwMaxCut = 1008;
static_assert(3 * kEwMaxCut * sizeof(double2) + 32 * 3 * sizeof(double) <= (48u << 10), "phase table too large");

struct EwaldArgs {
  int n, nk, nrow, nmax, tile;  // n: sites or points
  double invL[3], rec[3];
  const double *r, *w;          // positions; charges
  const double *g;              // dipole form: w_i g_i . k instead of w_i
  const int4 *row;              // (n_x, n_y, n_z of the first entry, its index)
  const short4 *kint;           // n_x, n_y, n_z of each wave vector
  const double *ak2;            // 2 a_k
  double2 *part, *sk;
};

// exp(2 pi i n x / L), n = 0..nmax, into t[0], t[stride], ...
__device__ __forceinline__ void axis_phases(double x, double invL, int nmax, double2 *t, int stride)
{
  double f = x * invL;
  f -= rint(f);
  double2 p;
  sincospi(2 * f, &p.y, &p.x);
  t[0] = make_double2(1.0, 0.0);
  if (nmax > 0)
    t[stride] = p;
  for (int n = 2; n <= nmax; n++) {
    const double2 a = t[(n >> 1) * stride], b = t[(n - (n >> 1)) * stride];
    t[n * stride] = make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
  }
}

// sites per table of the structure factor (a power of two, at most 32)
static int ewald_tile(int nmax)
{
  int t = 32;
  while (t > 1 && (size_t) t * 3 * (nmax + 1) * sizeof(double2) > (size_t) kEwTable)
    t >>= 1;
  return t;
}

template <bool DIPOLE>
__global__ void __launch_bounds__(kEwThreads) k_ewald_structure(EwaldArgs a)
{
  extern __shared__ __align__(16) double2 tab[];  // [site][axis][n]
  __shared__ double sw[32][DIPOLE ? 3 : 1];
  const int len = a.nmax + 1, width = 3 * len;
  const int k = blockIdx.x * kEwThreads + threadIdx.x;
  int nx = 0, ny = 0, nz = 0;
  if (k < a.nk) {
    const short4 n = a.kint[k];
    nx = n.x;
    ny = n.y;
    nz = n.z;
  }
  const int ox = nx, oy = len + abs(ny), oz = 2 * len + abs(nz);
  const double sy = ny < 0 ? -1 : 1, sz = nz < 0 ? -1 : 1;
  double c = 0, s = 0;
  for (int t0 = blockIdx.y * a.tile; t0 < a.n; t0 += gridDim.y * a.tile) {
    const int m = min(a.tile, a.n - t0);
    __syncthreads();
    if (threadIdx.x < 3 * m) {
      const int site = threadIdx.x / 3, d = threadIdx.x - 3 * site;
      const size_t i = (size_t) t0 + site;
      axis_phases(a.r[3 * i + d], a.invL[d], a.nmax, tab + site * width + d * len, 1);
      if (DIPOLE)
        sw[site][d] = a.w[i] * a.g[3 * i + d] * a.rec[d];
      else if (d == 0)
        sw[site][0] = a.w[i];
    }
    __syncthreads();
    if (k < a.nk) {
#pragma unroll 4
      for (int i = 0; i < m; i++) {
        const double2 *t = tab + i * width;
        const double2 x = t[ox];
        double2 y = t[oy], z = t[oz];
        y.y *= sy;
        z.y *= sz;
        double w = sw[i][0];
        if (DIPOLE)
          w = w * nx + sw[i][DIPOLE ? 1 : 0] * ny + sw[i][DIPOLE ? 2 : 0] * nz;
        const double px = w * (x.x * y.x - x.y * y.y), py = w * (x.x * y.y + x.y * y.x);
        c += px * z.x - py * z.y;
        s += px * z.y + py * z.x;
      }
    }
  }
  if (k < a.nk)
    a.part[(size_t) blockIdx.y * a.nk + k] = make_double2(c, s);
}

// sk[k] = 2 a_k S(k) (dipole form: of D(k) turned so that k_ewald_sum's
// potential is that of the dipoles), 32 wave vectors by kEwSlices slices of the partials
constexpr int kEwSlices = 32;
template <bool DIPOLE>
__global__ void __launch_bounds__(32 * kEwSlices) k_ewald_reduce(EwaldArgs a, int nb)
{
  __shared__ double2 sh[kEwSlices][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  const int per = (nb + kEwSlices - 1) / kEwSlices, lo = min(nb, w * per), hi = min(nb, lo + per);
  double c = 0, s = 0;
  if (k < a.nk)
#pragma unroll 4
    for (int b = lo; b < hi; b++) {
      const double2 v = a.part[(size_t) b * a.nk + k];
      c += v.x;
      s += v.y;
    }
  sh[w][lane] = make_double2(c, s);
  __syncthreads();
  if (w == 0 && k < a.nk) {
    for (int j = 1; j < min(kEwSlices, nb); j++) {
      c += sh[j][lane].x;
      s += sh[j][lane].y;
    }
    const double f = a.ak2[k];
    a.sk[k] = DIPOLE ? make_double2(f * s, -f * c) : make_double2(f * c, f * s);
  }
}

// phi (and with FIELD the field) of a lane's site or point
// STAGED: S(k) and the rows come from shared memory (each warp's walk over them is a
// chain of dependent reads)
template <bool FIELD, bool STAGED>
__global__ void __launch_bounds__(32 * kEwWarps) k_ewald_sum(EwaldArgs a, double neutral, bool add,
                                                             double *__restrict__ phi, double *__restrict__ evec)
{
  extern __shared__ __align__(16) double2 tab[];  // [axis][n][site], then S(k) and the rows
  __shared__ double sum[kEwWarps][FIELD ? 4 : 1][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int len = a.nmax + 1, T = a.tile;
  const size_t i0 = (size_t) blockIdx.x * T;
  const bool live = lane < T && i0 + lane < (size_t) a.n;
  const double2 *sk0 = a.sk;
  const int4 *rows = a.row;
  if (STAGED) {
    double2 *s = tab + 3 * len * T;
    int4 *r = reinterpret_cast<int4 *>(s + a.nk);
    for (int k = threadIdx.x; k < a.nk; k += 32 * kEwWarps)
      s[k] = a.sk[k];
    for (int k = threadIdx.x; k < a.nrow; k += 32 * kEwWarps)
      r[k] = a.row[k];
    sk0 = s;
    rows = r;
  }
  if (w < 3 && lane < T)
    axis_phases(live ? a.r[3 * (i0 + lane) + w] : 0.0, a.invL[w], a.nmax, tab + w * len * T + lane, T);
  __syncthreads();
  double p = 0, gx = 0, gy = 0, gz = 0;
  if (lane < T) {
    const double2 *tx = tab + lane, *ty = tx + len * T, *tz = ty + len * T;
    for (int j = w; j < a.nrow; j += kEwWarps) {
      const int4 row = rows[j];
      const int end = (j + 1 < a.nrow ? rows[j + 1].w : a.nk) - row.w;  // entries of the row
      const double2 x = tx[row.x * T];
      double2 y = ty[abs(row.y) * T];
      y.y = row.y < 0 ? -y.y : y.y;
      const double px = x.x * y.x - x.y * y.y, py = x.x * y.y + x.y * y.x;
      // entry of n_z = 0 (the row n_x = n_y = 0 starts at n_z = 1)
      const double2 *sk = sk0 + row.w - row.z;
      const int m = row.z + end - 1;
      double im_row = 0;
      if (row.z <= 0) {
        const double2 s = *sk;
        p += s.x * px + s.y * py;
        im_row = s.x * py - s.y * px;
      }
#pragma unroll 2
      for (int n = 1; n <= m; n++) {
        const double2 z = tz[n * T];
        const double ac = px * z.x, bd = py * z.y, ad = px * z.y, bc = py * z.x;
        const double2 s = sk[n];
        const double c1 = ac - bd, s1 = ad + bc;
        p += s.x * c1 + s.y * s1;
        double up = 0, um = 0;
        if (FIELD)
          up = s.x * s1 - s.y * c1;
        if (row.z < 0) {
          const double2 t = sk[-n];
          const double c2 = ac + bd, s2 = bc - ad;
          p += t.x * c2 + t.y * s2;
          if (FIELD)
            um = t.x * s2 - t.y * c2;
        }
        if (FIELD) {
          im_row += up + um;
          gz += n * (up - um);
        }
      }
      if (FIELD) {
        gx += row.x * im_row;
        gy += row.y * im_row;
      }
    }
  }
  sum[w][0][lane] = p;
  if constexpr (FIELD) {
    sum[w][1][lane] = gx;
    sum[w][2][lane] = gy;
    sum[w][3][lane] = gz;
  }
  __syncthreads();
  if (w < (FIELD ? 4 : 1) && live) {
    double v = sum[0][w][lane];
    for (int j = 1; j < kEwWarps; j++)
      v += sum[j][w][lane];
    const size_t i = i0 + lane;
    if (w == 0)
      phi[i] = ((add ? phi[i] : 0.0) + v) + neutral;
    else
      evec[3 * i + w - 1] = (add ? evec[3 * i + w - 1] : 0.0) + v * a.rec[w - 1];
  }
}

// ---- wave vectors ------------------------------------------------------------------

void ewald_free(EwaldSum &e)
{
  if (e.row)
    cudaFree(e.row);  // the first array of the one allocation
  e = EwaldSum();
}

// blocks of site tiles of the structure factor: enough to fill the chip with
// the blocks of wave vectors, no more partials than that
static int ewald_blocks(const EwaldSum &e, int nsite)
{
  const int tiles = div_up(nsite, ewald_tile(e.nmax)), kb = div_up(e.nk, kEwThreads);
  return std::max(1, std::min(tiles, std::max(1, 592 / kb)));
}

cudaError_t ewald_make(mmnb_handle *h, EwaldSum &e)
{
  ewald_free(e);
  const double kc = h->cfg.kspace_cutoff, n2max = kc * kc + 1e-8;
  if (kc >= kEwMaxCut)
    return cudaErrorInvalidValue;
  const int nmax = std::max(0, (int) floor(kc));
  std::vector<int4> row;
  std::vector<short4> kint;
  std::vector<double> ak2;
  const double c = 0.25 / (h->eta * h->eta), f = 4 * M_PI / h->volume;
  for (int d = 0; d < 3; d++)
    e.rec[d] = 2 * M_PI * (1.0 / h->box.L[d]);
  for (int nx = 0; nx <= nmax; nx++)
    for (int ny = (nx == 0 ? 0 : -nmax); ny <= nmax; ny++) {
      const int first = (int) ak2.size();
      int lo = 0;
      for (int nz = (nx == 0 && ny == 0 ? 1 : -nmax); nz <= nmax; nz++) {
        if ((double) nx * nx + (double) ny * ny + (double) nz * nz > n2max)
          continue;
        if ((int) ak2.size() == first)
          lo = nz;
        const double kx = e.rec[0] * nx, ky = e.rec[1] * ny, kz = e.rec[2] * nz;
        const double k2 = kx * kx + ky * ky + kz * kz;
        ak2.push_back(2 * (f * exp(-k2 * c) / k2));
        kint.push_back(make_short4((short) nx, (short) ny, (short) nz, 0));
      }
      if ((int) ak2.size() > first)
        row.push_back(make_int4(nx, ny, lo, first));
    }
  e.nk = (int) ak2.size();
  e.nrow = (int) row.size();
  e.nmax = nmax;
  e.made = true;
  if (e.nk == 0)
    return cudaSuccess;
  // one allocation: the rows, 2 a_k and the integer vectors (one copy), S(k), the partials
  const size_t nk = e.nk, nb = ewald_blocks(e, h->nsite);
  const size_t o_ak = sizeof(int4) * e.nrow, o_kint = o_ak + sizeof(double) * nk;
  const size_t o_sk = (o_kint + sizeof(short4) * nk + 15) / 16 * 16;
  std::vector<char> host(o_sk);
  std::copy(row.begin(), row.end(), reinterpret_cast<int4 *>(host.data()));
  std::copy(ak2.begin(), ak2.end(), reinterpret_cast<double *>(host.data() + o_ak));
  std::copy(kint.begin(), kint.end(), reinterpret_cast<short4 *>(host.data() + o_kint));
  char *dev = nullptr;
  cudaError_t s = cudaMalloc((void **) &dev, o_sk + sizeof(double2) * nk * (1 + nb));
  if (s != cudaSuccess) {
    e = EwaldSum();
    return s;
  }
  e.row = reinterpret_cast<int4 *>(dev);
  e.ak2 = reinterpret_cast<double *>(dev + o_ak);
  e.kint = reinterpret_cast<short4 *>(dev + o_kint);
  e.sk = reinterpret_cast<double2 *>(dev + o_sk);
  e.part = e.sk + nk;
  // on the handle's stream, whose kernels read it
  if ((s = cudaMemcpyAsync(dev, host.data(), host.size(), cudaMemcpyHostToDevice, h->stream)) != cudaSuccess ||
      (s = cudaStreamSynchronize(h->stream)) != cudaSuccess)
    ewald_free(e);
  return s;
}

static EwaldArgs ewald_args(const mmnb_handle *h, const EwaldSum &e)
{
  EwaldArgs a{};
  a.nk = e.nk;
  a.nrow = e.nrow;
  a.nmax = e.nmax;
  a.tile = ewald_tile(e.nmax);
  for (int d = 0; d < 3; d++) {
    a.invL[d] = 1.0 / h->box.L[d];
    a.rec[d] = e.rec[d];
  }
  a.row = e.row;
  a.kint = e.kint;
  a.ak2 = e.ak2;
  a.part = e.part;
  a.sk = e.sk;
  return a;
}

static size_t ewald_table_bytes(const EwaldArgs &a) { return (size_t) a.tile * 3 * (a.nmax + 1) * sizeof(double2); }

cudaError_t launch_ewald_structure(mmnb_handle *h, const EwaldSum &e, const double *d_r, const double *d_g)
{
  if (e.nk == 0)
    return cudaSuccess;
  EwaldArgs a = ewald_args(h, e);
  a.n = h->nsite;
  a.r = d_r;
  a.w = h->d_q;
  a.g = d_g;
  const int nb = ewald_blocks(e, h->nsite);
  const dim3 grid(div_up(e.nk, kEwThreads), nb);
  const size_t smem = ewald_table_bytes(a);
  if (d_g) {
    k_ewald_structure<true><<<grid, kEwThreads, smem, h->stream>>>(a);
    k_ewald_reduce<true><<<div_up(e.nk, 32), 32 * kEwSlices, 0, h->stream>>>(a, nb);
  } else {
    k_ewald_structure<false><<<grid, kEwThreads, smem, h->stream>>>(a);
    k_ewald_reduce<false><<<div_up(e.nk, 32), 32 * kEwSlices, 0, h->stream>>>(a, nb);
  }
  h->launches += 2;
  return cudaGetLastError();
}

cudaError_t launch_ewald_sum(mmnb_handle *h, const EwaldSum &e, int n, const double *d_pts, double neutral,
                             double *d_phi, double *d_evec, bool add)
{
  EwaldArgs a = ewald_args(h, e);
  a.n = n;
  a.r = d_pts;
  // up to 92 KB in all (two blocks per SM): about 5,000 wave vectors
  size_t smem = ewald_table_bytes(a);
  const size_t staged = smem + sizeof(double2) * e.nk + sizeof(int4) * e.nrow;
  const bool stage = staged <= (92u << 10);
  if (stage)
    smem = staged;
  auto *k = d_evec ? (stage ? k_ewald_sum<true, true> : k_ewald_sum<true, false>)
                   : (stage ? k_ewald_sum<false, true> : k_ewald_sum<false, false>);
  if (smem > (36u << 10)) {
    const cudaError_t s = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 92 << 10);
    if (s != cudaSuccess)
      return s;
  }
  k<<<div_up(n, a.tile), 32 * kEwWarps, smem, h->stream>>>(a, neutral, add, d_phi, d_evec);
  h->launches += 1;
  return cudaGetLastError();
}

// Adjoint: sum_j q_j g_j . dE_j/dq_i for the reciprocal sum.  With
// E_j = sum_k 2 a_k k (C sin k.r_j - S cos k.r_j) and C, S linear in the
// charges, dE_j/dq_i = sum_k 2 a_k k sin(k.(r_j - r_i)), so the sum is
// sum_k 2 a_k (Ds cos k.r_i - Dc sin k.r_i) with the dipole structure factor
// Dc + i Ds = sum_j q_j (k . g_j) exp(i k.r_j).
cudaError_t launch_kspace_dipole(mmnb_handle *h, const double *d_r, const double *d_g, double *d_psi)
{
  if (h->ew.nk == 0)
    return cudaSuccess;
  const cudaError_t e = launch_ewald_structure(h, h->ew, d_r, d_g);
  return e != cudaSuccess ? e : launch_ewald_sum(h, h->ew, h->nsite, d_r, 0.0, d_psi, nullptr, true);
}

}  // namespace mmnb
