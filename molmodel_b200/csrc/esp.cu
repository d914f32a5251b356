// Electrostatic potential at points away from the sites (replaces
// ElecLJ::electrostatic_potential_at_gridpoints, src/eleclj.cpp:1302-1340, its
// periodic branch).  Three terms, each optional as in the reference:
//   * real space (RSpaceEwaldPhiAtGridpoints, src/rspace.c:892-967): every
//     site with a nonzero mask against every point, minimum image with the
//     reference's rounding, cut at rc on the SITE-point distance, switched
//     over [rc - w, rc], erfc(eta r)/r from the Chebyshev table inside its
//     range, the short-range screening of the site's own r_screen;
//   * reciprocal space (kspace_new + kspace_phi, src/kspace.c:35-71, 176-250):
//     the ordinary Ewald k-sum over kspace_cutoff wave vectors, whatever the
//     handle uses for forces (P3M or the k-sum); the points carry no charge, so
//     the structure factor is that of the sites alone;
//   * the neutralising term -pi/(eta^2 V) sum q when the sites are not neutral
//     (src/eleclj.cpp:1330-1338).
// There is no self term: a point is not a charge.
//
// Layout of the real-space part: the sites are binned into cells (counting
// sort; within a cell in site order, so the sums are bitwise reproducible) and
// one warp takes a point.  It walks the columns of cells within reach along z
// -- a column's cells hold consecutive sites --, tests 32 sites at a time in
// FP32 against a cutoff widened past every FP32 rounding, queues the few that
// pass (one in nine of the sites of a sphere's bounding cells) and evaluates 32
// of them at a time in FP64, the reference's cutoff test included: neither the
// test of far sites nor the FP64 arithmetic runs with idle lanes.  The k-sum is
// kspace.cu's, its structure factor that of the sites.
//
// One thread per point over all sites (40 blocks for 5,000 points, each thread a
// serial loop of 12,288 FP64 minimum images): 3292 us; this layout: 43.6 us with
// 16 us of binning (12,288 sites, rc 9 A), and the work grows with the sites
// near a point instead of with all of them.  Columns one after the other and one
// queue (a lane or two taking erfc in nearly every batch): 65 us.

#include <algorithm>
#include <cmath>
#include <string>

#include "mmnb_internal.cuh"

namespace mmnb {

constexpr int kEspThreads = 256;
constexpr int kEspWarps = kEspThreads / 32;
constexpr int kEspMaxCells = 8192;  // their counts are scanned in shared memory

struct EspArgs {
  int nsite, npoint;
  Box box;
  double rlo2, rhi2, inv_sw, eta;
  double cheb_min, cheb_max, cheb_inv_dx;
  const double2 *t0, *t1;  // the table's cubics
  const double *r, *q, *rscreen, *pts;
  const int *mask;
  double *phi;
  // cells: n per axis, their edges, how many of them the cutoff reaches across
  int n[3], reach[3], ncell;
  float Lf[3], edge[3], reach2, low2;
  int *cell, *slot, *ids, *count, *start, *far;  // far: set when a site is far away (esp_near)
  float4 *near;    // sorted sites wrapped into the box
  double4 *site;   // sorted sites: position and charge
  double *screen;  // sorted sites: r_screen
};

// b0 = erfc(eta r)/r: the table inside its range, the closed form outside
__device__ __forceinline__ double esp_b0(const EspArgs &a, double r2)
{
  if (a.cheb_min < r2 && r2 < a.cheb_max) {
    double x = (r2 - a.cheb_min) * a.cheb_inv_dx;
    const unsigned i = (unsigned) x;
    const double2 c01 = __ldg(a.t0 + i), c23 = __ldg(a.t1 + i);
    x -= i;
    return ((c23.y * x + c23.x) * x + c01.y) * x + c01.x;
  }
  const double rm = sqrt(r2);
  return erfc(a.eta * rm) / rm;
}

// Whether a coordinate is near enough to be wrapped: 2^30 box lengths away the wrapped
// value is off by 2^-22 of one, within the margin of `reach`.  A point or a site
// farther out (or not finite) has no cell that means anything, and what the minimum
// image makes of it is rounding: such a point, and every point when a site is such,
// takes all sites one by one.
__device__ __forceinline__ bool esp_near(const EspArgs &a, double x, double y, double z)
{
  const double m = 1073741824.0;
  return fabs(x * a.box.invL[0]) <= m && fabs(y * a.box.invL[1]) <= m && fabs(z * a.box.invL[2]) <= m;
}

// position wrapped into [0, L] and its cell along one axis, both in range whatever the
// coordinate (a conversion of NaN gives 0 and others saturate), right for a near one
__device__ __forceinline__ int esp_cell(const EspArgs &a, int d, double x, float &w)
{
  const double f = x - a.box.L[d] * floor(x * a.box.invL[d]);
  w = fminf(fmaxf((float) f, 0.f), a.Lf[d]);
  return min(max((int) (f * a.box.invL[d] * a.n[d]), 0), a.n[d] - 1);
}

// cell of each site that acts on points, its place there in order of arrival
__global__ void __launch_bounds__(kEspThreads) k_esp_count(EspArgs a)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nsite)
    return;
  int c = -1;
  if (a.mask[i]) {
    float w;
    const double x = a.r[3 * i], y = a.r[3 * i + 1], z = a.r[3 * i + 2];
    c = (esp_cell(a, 0, x, w) * a.n[1] + esp_cell(a, 1, y, w)) * a.n[2] + esp_cell(a, 2, z, w);
    if (!esp_near(a, x, y, z))
      *a.far = 1;
    a.slot[i] = atomicAdd(a.count + c, 1);
  }
  a.cell[i] = c;
}

// sites by cell; every block scans the counts for itself
__global__ void __launch_bounds__(kEspThreads) k_esp_scatter(EspArgs a)
{
  extern __shared__ int start[];  // ncell + 1
  __shared__ int warp_sum[kEspWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per = (a.ncell + kEspThreads - 1) / kEspThreads;
  const int lo = min(a.ncell, (int) threadIdx.x * per), hi = min(a.ncell, lo + per);
  int v = 0;
  for (int c = lo; c < hi; c++)
    v += a.count[c];
  int incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o)
      incl += u;
  }
  if (lane == 31)
    warp_sum[w] = incl;
  __syncthreads();
  int run = incl - v;
  for (int k = 0; k < w; k++)
    run += warp_sum[k];
  for (int c = lo; c < hi; c++) {
    start[c] = run;
    run += a.count[c];
  }
  if (threadIdx.x == kEspThreads - 1)
    start[a.ncell] = run;
  __syncthreads();
  if (blockIdx.x == 0)
    for (int c = threadIdx.x; c <= a.ncell; c += kEspThreads)
      a.start[c] = start[c];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.nsite && a.cell[i] >= 0)
    a.ids[start[a.cell[i]] + a.slot[i]] = i;
}

// each cell's sites in site order, and what the sums read of them
__global__ void __launch_bounds__(kEspThreads) k_esp_place(EspArgs a)
{
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.start[a.ncell])
    return;
  const int i = a.ids[p], c = a.cell[i];
  const int b = a.start[c], e = a.start[c + 1];
  int pos = b;
  for (int k = b; k < e; k++)
    pos += a.ids[k] < i;
  const double x = a.r[3 * i], y = a.r[3 * i + 1], z = a.r[3 * i + 2];
  float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
  esp_cell(a, 0, x, w.x);
  esp_cell(a, 1, y, w.y);
  esp_cell(a, 2, z, w.z);
  a.near[pos] = w;
  a.site[pos] = make_double4(x, y, z, a.q[i]);
  a.screen[pos] = a.rscreen[i];
}

// distance along one axis between wrapped coordinates, minimum image
__device__ __forceinline__ float near_dist(float d, float L)
{
  d = fabsf(d);
  return fminf(d, L - d);
}

// potential of sorted site k at a point
__device__ __forceinline__ double esp_site(const EspArgs &a, int k, double gx, double gy, double gz)
{
  const double4 s = a.site[k];
  // site minus point, then the displacement to the central box
  double x = __dsub_rn(s.x, gx), y = __dsub_rn(s.y, gy), z = __dsub_rn(s.z, gz);
  min_image_ref(a.box, x, y, z);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
  if (r2 > a.rhi2)
    return 0.0;
  double b0 = esp_b0(a, r2);
  const double rs = a.screen[k];
  if (r2 < rs * rs) {
    const double invr = 1.0 / sqrt(r2);
    b0 += (-0.5 * r2 * (1.0 / (rs * rs * rs)) + 1.5 / rs) - invr;
  }
  if (r2 > a.rlo2) {
    const double zz = (r2 - a.rlo2) * a.inv_sw;
    b0 *= ((-6 * zz + 15) * zz - 10) * zz * zz * zz + 1;
  }
  return s.w * b0;
}

// of all sites, by a warp (a call, so that it costs the other points no registers:
// tested for before their walk, the points call took 160 us instead of 154)
__device__ __noinline__ double esp_all(const EspArgs &a, double gx, double gy, double gz, int lane)
{
  double p = 0;
  for (int k = lane; k < a.start[a.ncell]; k += 32)
    p += esp_site(a, k, gx, gy, gz);
  for (int o = 16; o > 0; o >>= 1)
    p += __shfl_xor_sync(0xffffffffu, p, o);
  return p;
}

__global__ void __launch_bounds__(kEspThreads) k_esp_rspace(const __grid_constant__ EspArgs a)
{
  __shared__ int queue[kEspWarps][2][64];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * kEspWarps + w;
  if (j >= a.npoint)
    return;  // the whole warp
  const unsigned below = (1u << lane) - 1;
  // [0]: sites the table's cubic covers; [1]: those near its lower end, which may
  // take erfc (a handful a point: together, not one or two lanes of every batch)
  int(*const wq)[64] = queue[w];
  const double gx = a.pts[3 * (size_t) j], gy = a.pts[3 * (size_t) j + 1], gz = a.pts[3 * (size_t) j + 2];
  double p = 0;
  auto eval = [&](int k) { p += esp_site(a, k, gx, gy, gz); };
  float px, py, pz;
  const int cx = esp_cell(a, 0, gx, px), cy = esp_cell(a, 1, gy, py);
  esp_cell(a, 2, gz, pz);
  int qn[2] = {0, 0};
  const int nx = a.n[0], ny = a.n[1], nz = a.n[2];
  const int sx = min(2 * a.reach[0] + 1, nx), sy = min(2 * a.reach[1] + 1, ny);
  // offsets -reach..reach, or every cell of a short axis
  const int x0 = sx == nx ? 0 : cx - a.reach[0], y0 = sy == ny ? 0 : cy - a.reach[1];
  for (int c0 = 0; c0 < sx * sy; c0 += 32) {
    // a lane's column: its sites within reach, up to two ranges [b1, b1 + l1) and
    // [b2, ...) where they wrap around the box
    int b1 = 0, l1 = 0, b2 = 0, len = 0;
    if (c0 + lane < sx * sy) {
      const int u = (c0 + lane) / sy, v = c0 + lane - u * sy;
      int ix = x0 + u, iy = y0 + v;
      ix += ix < 0 ? nx : 0;
      ix -= ix >= nx ? nx : 0;
      iy += iy < 0 ? ny : 0;
      iy -= iy >= ny ? ny : 0;
      const float ex = fmaxf(near_dist(px - (ix + 0.5f) * a.edge[0], a.Lf[0]) - 0.5f * a.edge[0], 0.f);
      const float ey = fmaxf(near_dist(py - (iy + 0.5f) * a.edge[1], a.Lf[1]) - 0.5f * a.edge[1], 0.f);
      const float h2 = a.reach2 - ex * ex - ey * ey;  // half the chord of the column, squared
      if (h2 >= 0) {
        const float h = sqrtf(h2);
        int lo = (int) floorf((pz - h) / a.edge[2]), hi = (int) floorf((pz + h) / a.edge[2]);
        const int *st = a.start + (ix * ny + iy) * nz;
        int lo2 = 0, hi2 = -1;
        if (hi - lo >= nz - 1) {
          lo = 0;
          hi = nz - 1;
        } else if (lo < 0) {
          lo2 = 0;
          hi2 = hi;
          lo += nz;
          hi = nz - 1;
        } else if (hi >= nz) {
          hi2 = hi - nz;
          hi = nz - 1;
        }
        b1 = st[lo];
        l1 = st[hi + 1] - b1;
        b2 = st[lo2];
        len = l1 + st[hi2 + 1] - b2;
      }
    }
    int incl = len;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o)
        incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    // the columns' sites as one sequence: the t-th
    auto site_at = [&](int t) {
      int o = 0;  // the lane whose column holds it
#pragma unroll
      for (int h = 16; h > 0; h >>= 1)
        if (__shfl_sync(0xffffffffu, incl, o + h - 1) <= t)
          o += h;
      const int off = t - (__shfl_sync(0xffffffffu, incl, o) - __shfl_sync(0xffffffffu, len, o));
      const int f = __shfl_sync(0xffffffffu, l1, o);
      const int p1 = __shfl_sync(0xffffffffu, b1, o), p2 = __shfl_sync(0xffffffffu, b2, o);
      return off < f ? p1 + off : p2 + (off - f);
    };
    int k = site_at(min(lane, max(total - 1, 0)));
    float4 s = total > 0 ? a.near[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int base = 0; base < total; base += 32) {
      // the next 32 are on their way while these are tested
      const int kn = site_at(min(base + 32 + lane, total - 1));
      const float4 sn = a.near[kn];
      const float x = near_dist(s.x - px, a.Lf[0]), y = near_dist(s.y - py, a.Lf[1]), z = near_dist(s.z - pz, a.Lf[2]);
      const float f2 = x * x + y * y + z * z;
      const bool take = base + lane < total && f2 <= a.reach2, low = f2 < a.low2;
#pragma unroll
      for (int g = 0; g < 2; g++) {
        const bool mine = take && low == (g == 1);
        const unsigned bal = __ballot_sync(0xffffffffu, mine);
        if (mine)
          wq[g][qn[g] + __popc(bal & below)] = k;
        qn[g] += __popc(bal);
        __syncwarp();
        if (qn[g] >= 32) {
          qn[g] -= 32;
          eval(wq[g][qn[g] + lane]);
          __syncwarp();
        }
      }
      k = kn;
      s = sn;
    }
  }
  for (int g = 0; g < 2; g++)
    if (lane < qn[g])
      eval(wq[g][lane]);
  for (int o = 16; o > 0; o >>= 1)
    p += __shfl_xor_sync(0xffffffffu, p, o);
  if (*a.far || !esp_near(a, gx, gy, gz))
    p = esp_all(a, gx, gy, gz, lane);
  if (lane == 0)
    a.phi[j] = p;
}

}  // namespace mmnb

using namespace mmnb;

static int esp_fail(mmnb_handle *h, int code, const std::string &msg)
{
  if (h)
    h->err = msg;
  return code;
}

extern "C" int mmnb_phi_at_points(mmnb_handle *h, const double *r, int npoint, const double *points, double *phi)
{
  if (!h || !r || (npoint > 0 && (!points || !phi)) || npoint < 0)
    return esp_fail(h, MMNB_ERR_ARG, "null handle, positions, points or output, or a negative point count");
  if (npoint > (1 << 30) / 3)
    return esp_fail(h, MMNB_ERR_ARG, "at most 357,913,941 points per call (32-bit point indices)");
  if (!h->params_set)
    return esp_fail(h, MMNB_ERR_STATE, "mmnb_set_params has not been called");
  if (npoint == 0)
    return MMNB_OK;
  const mmnb_config &c = h->cfg;
  cudaError_t e = cudaSuccess;
  // wave vectors of kspace_new(kspace_cutoff, .) (src/kspace.c:35-71): the
  // handle's, or with P3M made here once
  if (c.include_kspace && !h->ew.made && (e = ewald_make(h, h->ew)) != cudaSuccess) {
    if (e == cudaErrorInvalidValue)
      return esp_fail(h, MMNB_ERR_ARG, "kspace_cutoff is too large");
    return esp_fail(h, MMNB_ERR_CUDA, std::string("potential at points: ") + cudaGetErrorString(e));
  }
  const int nk = c.include_kspace ? h->ew.nk : 0;
  EspArgs a{};
  a.nsite = h->nsite;
  a.npoint = npoint;
  a.box = h->box;
  a.rlo2 = h->rlo2;
  a.rhi2 = h->rhi2;
  a.inv_sw = h->inv_sw;
  a.eta = h->eta;
  a.cheb_min = h->cheb_min;
  a.cheb_max = h->cheb_max;
  a.cheb_inv_dx = h->cheb_inv_dx;
  a.t0 = reinterpret_cast<const double2 *>(h->d_cheb_w);
  a.t1 = a.t0 + h->cheb_w_nseg;
  a.q = h->d_q;
  a.rscreen = h->d_rscreen;
  a.mask = h->d_mask;
  // the FP32 test's reach: the cutoff, a margin over the rounding of wrapped
  // FP32 coordinates and of the cells' bounds
  const double lmax = std::max(std::max(h->box.L[0], h->box.L[1]), h->box.L[2]);
  const double reach = h->rc + 0.01 + 16 * lmax * std::ldexp(1.0, -23);
  a.reach2 = (float) (reach * reach);
  a.low2 = (float) ((sqrt(h->cheb_min) + (reach - h->rc)) * (sqrt(h->cheb_min) + (reach - h->rc)));
  // cells of at least half the reach, larger when there would be too many
  double least = 0.5 * reach;
  do {
    a.ncell = 1;
    for (int d = 0; d < 3; d++) {
      a.n[d] = std::max(1, (int) std::min(1.0 * kEspMaxCells, h->box.L[d] / least));
      a.ncell = (int) std::min(1e9, (double) a.ncell * a.n[d]);
    }
    least *= 1.1;
  } while (a.ncell > kEspMaxCells);
  for (int d = 0; d < 3; d++) {
    a.Lf[d] = (float) h->box.L[d];
    a.edge[d] = (float) (h->box.L[d] / a.n[d]);
    a.reach[d] = (int) ceil(reach / (h->box.L[d] / a.n[d]) + 1e-3);
  }
  // scratch, in doubles: positions, points, potentials, the sorted sites (6.5
  // each) and three ints a site, the cells; kept with the handle up to 64 MB
  const size_t n = h->nsite, m = npoint;
  const size_t ints = 3 * n + 2 * (size_t) a.ncell + 2;
  const size_t need = 3 * n + 4 * m + 4 * n + 2 * n + n + (ints + 1) / 2 + 8;
  double *buf = h->d_esp;
  if (h->esp_cap < need) {
    if (h->d_esp)
      cudaFree(h->d_esp);
    h->d_esp = nullptr;
    h->esp_cap = 0;
    if ((e = cudaMalloc(&buf, need * sizeof(double))) != cudaSuccess)
      return esp_fail(h, MMNB_ERR_CUDA, std::string("potential at points: ") + cudaGetErrorString(e));
    if (need * sizeof(double) <= (64u << 20)) {
      h->d_esp = buf;
      h->esp_cap = need;
    }
  }
  // the 32-byte entries first: every array then starts on a multiple of its entry
  a.site = reinterpret_cast<double4 *>(buf);
  a.near = reinterpret_cast<float4 *>(a.site + n);
  double *d_r = reinterpret_cast<double *>(a.near + n), *d_pts = d_r + 3 * n, *d_phi = d_pts + 3 * m;
  a.r = d_r;
  a.pts = d_pts;
  a.phi = d_phi;
  a.screen = d_phi + m;
  a.cell = reinterpret_cast<int *>(a.screen + n);
  a.slot = a.cell + n;
  a.ids = a.slot + n;
  a.count = a.ids + n;  // the counts and the flag behind them are cleared together
  a.far = a.count + a.ncell;
  a.start = a.far + 1;
  e = cudaMemcpyAsync(d_r, r, 3 * n * sizeof(double), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess && c.include_rspace) {
    e = cudaMemsetAsync(a.count, 0, ((size_t) a.ncell + 1) * sizeof(int), h->stream);
    const int blocks = div_up(h->nsite, kEspThreads);
    k_esp_count<<<blocks, kEspThreads, 0, h->stream>>>(a);
    k_esp_scatter<<<blocks, kEspThreads, (a.ncell + 1) * sizeof(int), h->stream>>>(a);
    k_esp_place<<<blocks, kEspThreads, 0, h->stream>>>(a);
    h->launches += 3;
    if (e == cudaSuccess)
      e = cudaGetLastError();
  }
  if (e == cudaSuccess && nk > 0)
    e = launch_ewald_structure(h, h->ew, d_r, nullptr);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_pts, points, 3 * m * sizeof(double), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess && c.include_rspace) {
    k_esp_rspace<<<div_up(npoint, kEspWarps), kEspThreads, 0, h->stream>>>(a);
    h->launches += 1;
    e = cudaGetLastError();
  } else if (e == cudaSuccess) {
    e = cudaMemsetAsync(d_phi, 0, m * sizeof(double), h->stream);
  }
  const double neutral = c.include_self ? h->neutral_b : 0.0;
  if (e == cudaSuccess && (nk > 0 || neutral != 0)) {
    EwaldSum none;
    none.made = true;
    e = launch_ewald_sum(h, nk > 0 ? h->ew : none, npoint, d_pts, neutral, d_phi, nullptr, true);
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(phi, d_phi, npoint * sizeof(double), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(h->stream);
  if (buf != h->d_esp)
    cudaFree(buf);
  if (e != cudaSuccess)
    return esp_fail(h, MMNB_ERR_CUDA, std::string("potential at points: ") + cudaGetErrorString(e));
  return MMNB_OK;
}
