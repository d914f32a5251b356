// Everything an evaluation does per site after the pair kernels and the mesh
// transforms, in one kernel: interpolation of potential and field from the P3M
// mesh (src/pppm.c:498-641), exclusion corrections and 1-4 pairs
// (src/rspace.c:219-242, 492-557), self terms, force assembly and energies
// (src/eleclj.cpp:794-805, 961-976).
//
//   * mesh: P lanes per site along z, lane c taking the points z = base + c of the
//     site's P^2 rows, so a site's lanes read consecutive mesh words (three of them work
//     out the weights of an axis each for all); the P rows of
//     one x-plane are summed with the y weights first (2 multiply-adds a point
//     where the three-weight products of a thread per site took 8).  FP64, or FP32
//     converted to fixed point per site (mixed form).  Without a mesh, two lanes per
//     site share the partners below;
//   * exclusions and 1-4 pairs: the site's partners shared out over its lanes;
//   * phi -= (2 eta / sqrt(pi)) q, plus the neutralising background -pi/(eta^2 V)
//     sum(q) when the system is charged; F = q E + F_LJ (AtomSite projection,
//     include/eleclj.hpp:68-71), by the site's first lane;
//   * energies: elec = (q . phi)/2, LJ = pair sum + tail.  Each block writes its
//     partial sums; the last block to finish (a counter taken after a fence) adds
//     them in index order, so the FP64 energies are bitwise reproducible without a
//     second launch.
//
// As three kernels (exclusions, interpolation, assembly) the sites' potential,
// field and LJ force went through memory between them and each waited for the
// last (profiled one by one, caches cold): 98,304 sites 32.5 us mixed, 59 us FP64;
// 12,288 sites 26 and 37 us.  This kernel, in a step with stage timing: 98,304 sites 26
// us mixed, 29 FP64; 12,288 sites 14 and 15.  Bound by the loads' latency: a site's lanes
// cover it where the sites alone would leave the chip idle, and repeat its weights where
// they would not.

#include "mesh.cuh"

namespace mmnb {

constexpr int kSiteThreads = 128;

enum MeshKind { kNoMesh, kMesh64, kMesh64Ik, kMesh32, kMesh32Ik };

struct SiteArgs {
  int nsite, do_self, do_excl, do14, geometric;
  int keep_fields;       // write phi, E and the LJ force back (the caller asked for the site fields)
  int assign_f;          // write the forces instead of adding them
  int have_sums;         // phi, E (and the FP64 form's LJ force) hold terms of this evaluation
  int have_ljf;
  Box box;
  double eta, self_a, neutral_b, e14, l14;
  int scale_e14, scale_l14;
  MeshArgs mesh;
  const double *r, *q, *sig, *eps, *rscreen;
  const int *mask, *excl_ptr, *excl_idx, *p14_ptr, *p14_idx;
  const double *mesh64, *egrid64;
  const float *mesh32, *egrid32;
  size_t nr;
  const long long *acc;  // mixed form: fixed-point potential, field and LJ force per site
  double *phi, *evec, *ljf, *f;
  // energy reduction
  double *part;                       // per block: q phi, LJ of 1-4 pairs, their virial, LJ of its rows
  const double *lj_row;               // per-row LJ energies [0, nrow), or null
  int nrow, any_q;
  const unsigned long long *wsum;     // mixed water kernel's fixed-point energies, or null
  unsigned long long *counter;        // finished-block counter, left at 0
  int *flags;                         // list flags: counts evaluations finished on cut rows
  double *status;                     // or null: the host call's mapped status block
                                      // (energies, flags, ready word)
  double tail;
  double *energy, *vir14;
};

// sums of N values over the block in a fixed order: lanes by a shuffle tree, then
// the warps' sums in warp order; thread 0 returns them
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], double (*sh)[N])
{
  constexpr int kWarps = kSiteThreads / 32;
#pragma unroll
  for (int k = 0; k < N; k++)
    for (int o = 16; o > 0; o >>= 1)
      v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < N; k++)
      sh[threadIdx.x >> 5][k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kWarps; w++)
#pragma unroll
      for (int k = 0; k < N; k++)
        v[k] += sh[w][k];
}

// b0 = -erf(eta r)/r of an excluded pair and b1 = -2 d b0 / d(r^2): erf's
// Maclaurin series at bond distances (kErfSeries; no division, no cancellation),
// else the functions
__device__ __forceinline__ void excluded_b(const SiteArgs &a, double r2, double &b0, double &b1)
{
  const double eta2 = a.eta * a.eta, y = eta2 * r2, cerf = a.eta * M_2_SQRTPI;
  if (y <= kErfSeriesMax * kErfSeriesMax) {
    double p, d;
    erf_series(y, p, d);
    b0 = -cerf * p;
    b1 = 2 * cerf * eta2 * d;
  } else {
    const double rm = sqrt(r2);
    b0 = -erf(a.eta * rm) / rm;
    b1 = (b0 + cerf * exp(-y)) / r2;
  }
}

// a mesh row's points of one lane, 16 bytes a load when whole rows allow it
template <typename T, int V>
struct MeshVec {
  T v[V];
};
template <int V>
__device__ __forceinline__ MeshVec<float, V> mesh_load(const float *p)
{
  MeshVec<float, V> o;
  if constexpr (V == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    o.v[0] = t.x, o.v[1] = t.y, o.v[2] = t.z, o.v[3] = t.w;
  } else {
    o.v[0] = __ldg(p);
  }
  return o;
}
template <int V>
__device__ __forceinline__ MeshVec<double, V> mesh_load(const double *p)
{
  MeshVec<double, V> o;
  if constexpr (V == 2) {
    const double2 t = __ldg(reinterpret_cast<const double2 *>(p));
    o.v[0] = t.x, o.v[1] = t.y;
  } else {
    o.v[0] = __ldg(p);
  }
  return o;
}

// Blocks an SM the register budget is cut for, a lane per site.  The sites' loads want
// many warps, a spilled order takes more from them than they give, and the best cut
// moves with the order's arrays.  32,768 waters, the step in us at 6 / 4 / 3 / 2 blocks:
//   FP64  order 3: 228 / 232 / 233 / 232    mixed  122 / 126 / 124 / -
//         order 4: 256 / 245 / 244 / 248           133 / 136 / 135 / -
//         order 5: 285 / 263 / 257 / 262           154 / 147 / 149 / 154
//         order 6: 324 / 313 / 285 / 284           181 / 169 / 171 / 176
//         order 7: 383 / 361 / 332 / 316           222 / 209 / 190 / 196
//   with ik, 5:    372 / 372 / 367 / 368           199 / 207 / 206 / -
//            7:    521 / 519 / 481 / 470           297 / 293 / 269 / 286
// (orders 5 and 7 of 66,000 sites with ik, mixed: one wave at 4 blocks, 149 us; 154 at
// 6, 163 at 3.)  One cap of 6 for all, which order 5's whole-word rows were measured
// with, spilled up to 6 KB a thread: order 7 388 us FP64 and 233 mixed on rows of 81.
constexpr int site_blocks_per_sm(int P, MeshKind kind, int V)
{
  const bool k32 = kind == kMesh32 || kind == kMesh32Ik, ik = kind == kMesh64Ik || kind == kMesh32Ik;
  if (V > 1)
    return k32 || P <= 5 ? 6 : 3;
  return P <= 3 || (k32 && P == 4) ? 6 : P == 4 || (k32 && P == 5) ? 4 : !k32 && (P == 7 || ik) ? 2 : 3;
}

// Mesh points a load of a lane per site past kSiteWordsMin sites.  16 bytes' take fewer
// requests of a row but 8 points for an order of 5: little in a box whose molecules are in
// order, more once they have diffused and a warp's sites share no lines.  32,768 waters in
// order / shuffled, us a step, point by point and by 16 bytes: order 5 mixed 147 / 161 and
// 147 / 150; with ik, mixed 4 180 / 226 and 189 / 205, 5 207 / 272 and 205 / 231; FP64 4
// 348 / 375 and 347 / 366, 5 368 / 417 and 369 / 404, 7 470 / 612 and 472 / 565.  The others
// point by point: order 7 mixed 192 / 217 and 198 / 211, with ik 269 / 395 and 294 / 367,
// 3 with ik 160 / 183 and 168 / 179, FP64 6 288 / 306 and 290 / 300.
constexpr int site_words(int P, MeshKind kind)
{
  if (kind == kMesh64Ik)
    return P >= 4 ? 2 : 1;
  return (kind == kMesh32 && P == 5) || (kind == kMesh32Ik && (P == 4 || P == 5)) ? 4 : 1;
}

// P: assignment order, or 0 without a mesh; L: lanes per site (P or one with a mesh);
// V: mesh points per load (one lane per site and rows of whole 16-byte words; else 1)
template <int P, MeshKind KIND, int L, int V>
__global__ void __launch_bounds__(kSiteThreads, L == 1 ? site_blocks_per_sm(P, KIND, V) : 1) k_sites(SiteArgs a)
{
  constexpr int S = 32 / L;
  constexpr bool k32 = KIND == kMesh32 || KIND == kMesh32Ik, kIk = KIND == kMesh64Ik || KIND == kMesh32Ik;
  __shared__ double sh[kSiteThreads / 32][4];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, c = lane % L;
  const int i = (int) ((blockIdx.x * kSiteThreads + threadIdx.x) >> 5) * S + lane / L;
  const bool live = lane < S * L && i < a.nsite;
  cudaTriggerProgrammaticLaunchCompletion();
  // exclusion and 1-4 terms of this lane's partners; FP64 mesh terms join them
  double v[4] = {0, 0, 0, 0}, lf[3] = {0, 0, 0}, elj = 0, vir = 0;
  float v32[4] = {0.f, 0.f, 0.f, 0.f};
  int mi = 0, x0 = 0, x1 = 0, jx = 0;
  double qi = 0;
  typedef typename std::conditional<k32, float, double>::type T;
  constexpr int NZ = L == 1 ? P : 1;  // points along z of this lane
  constexpr bool kShared = KIND != kNoMesh && L >= 3;
  MeshRows<P ? P : 1, P ? NZ : 1, T> o;
  if constexpr (kShared)
    mesh_rows_lanes<P, T>(a.mesh, a.r + 3 * (size_t) (live ? i : 0), lane - c, c, o);
  if (live) {
    // first what the later parts' loads depend on
    mi = a.mask[i];
    qi = a.q[i];
    if (a.do_excl) {
      x0 = a.excl_ptr[i] + c;
      x1 = a.excl_ptr[i + 1];
      if (x0 < x1)
        jx = a.excl_idx[x0];
    }
    if constexpr (KIND != kNoMesh) {
      constexpr int NV = V == 1 ? NZ : (V - 1 + P + V - 1) / V;  // loads a row
      if constexpr (!kShared)
        mesh_rows<P, NZ, T>(a.mesh, a.r + 3 * (size_t) i, c, o);
      const T *const mesh = k32 ? (const T *) a.mesh32 : (const T *) a.mesh64;
      const T *const eg = k32 ? (const T *) a.egrid32 : (const T *) a.egrid64;
      // the row's words and the weights of their points: with whole words the P points
      // start at point `sh0` of the first, the others weigh nothing
      T wz[NV * V], dz[NV * V];
      int iz[NV];
      if constexpr (V > 1) {
        const int sh0 = o.iz[0] % V;
        int k = o.iz[0] - sh0;
#pragma unroll
        for (int z = 0; z < NV; z++) {
          iz[z] = k;
          k = k + V == a.mesh.n[2] ? 0 : k + V;
        }
#pragma unroll
        for (int z = 0; z < NV * V; z++)
          wz[z] = dz[z] = 0;
#pragma unroll
        for (int s = 0; s < V; s++)
#pragma unroll
          for (int z = 0; z < P; z++)
            if (s == sh0) {
              wz[s + z] = o.wz[z];
              dz[s + z] = o.dz[z];
            }
      } else {
#pragma unroll
        for (int z = 0; z < NV; z++) {
          wz[z] = o.wz[z];
          dz[z] = o.dz[z];
          iz[z] = o.iz[z];
        }
      }
      // sums of the potential (s0: weights; s1, s2, s3: the derivative along x, y, z)
      // or, with ik, of the potential and the three field meshes
      T s0 = 0, s1 = 0, s2 = 0, s3 = 0;
#pragma unroll
      for (int x = 0; x < P; x++) {
        T t0 = 0, t1 = 0, t2 = 0, t3 = 0;
        const size_t plane = (size_t) o.ix[x] * (a.mesh.n[1] * a.mesh.n[2]);
        const T *const mp = mesh + plane, *const ep = eg + plane;
#pragma unroll
        for (int y = 0; y < P; y++) {
          const int row = o.iy[y] * a.mesh.n[2];
          T u0 = 0, u1 = 0, u2 = 0, u3 = 0;
#pragma unroll
          for (int z = 0; z < NV; z++) {
            const int k = row + iz[z];
            const MeshVec<T, V> u = mesh_load<V>(mp + k);
            MeshVec<T, V> e1, e2, e3;
            if constexpr (kIk) {
              e1 = mesh_load<V>(ep + k);
              e2 = mesh_load<V>(ep + a.nr + k);
              e3 = mesh_load<V>(ep + 2 * a.nr + k);
            }
#pragma unroll
            for (int s = 0; s < V; s++) {
              const T w = wz[z * V + s];
              u0 += w * u.v[s];
              if constexpr (kIk) {
                u1 += w * e1.v[s];
                u2 += w * e2.v[s];
                u3 += w * e3.v[s];
              } else {
                u3 += dz[z * V + s] * u.v[s];
              }
            }
          }
          t0 += o.wy[y] * u0;
          t1 += kIk ? o.wy[y] * u1 : o.dy[y] * u0;
          if (kIk)
            t2 += o.wy[y] * u2;
          t3 += o.wy[y] * u3;
        }
        s0 += o.wx[x] * t0;
        s1 += kIk ? o.wx[x] * t1 : o.dx[x] * t0;
        s2 += o.wx[x] * (kIk ? t2 : t1);
        s3 += o.wx[x] * t3;
      }
      T m[4];
      // with ik the field meshes hold the Cartesian field; otherwise
      // E = A^T (-grad_s phi) (left_operate, include/cart.h:28-36), A diagonal
      m[0] = s0;
      m[1] = kIk ? s1 : s1 * (T) a.mesh.A[0];
      m[2] = kIk ? s2 : s2 * (T) a.mesh.A[4];
      m[3] = kIk ? s3 : s3 * (T) a.mesh.A[8];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (k32)
          v32[k] = (float) m[k];
        else
          v[k] = m[k];
      }
    }
    if (a.do_excl) {
      const double xi = a.r[3 * i], yi = a.r[3 * i + 1], zi = a.r[3 * i + 2];
      if (mi & MMNB_SITE_HAS_Q) {
        for (int n = x0; n < x1; n += L) {
          const int j = jx;
          if (n + L < x1)
            jx = a.excl_idx[n + L];
          if (!(a.mask[j] & MMNB_SITE_HAS_Q))
            continue;
          double x = xi - a.r[3 * j], y = yi - a.r[3 * j + 1], z = zi - a.r[3 * j + 2];
          min_image_ref(a.box, x, y, z);
          double b0, b1;
          excluded_b(a, x * x + y * y + z * z, b0, b1);
          const double qj = a.q[j];
          v[0] += qj * b0;
          v[1] += qj * b1 * x;
          v[2] += qj * b1 * y;
          v[3] += qj * b1 * z;
        }
      }
      if (a.do14) {
        const int end = a.p14_ptr[i + 1];
        for (int n = a.p14_ptr[i] + c; n < end; n += L) {
          const int j = a.p14_idx[n];
          const int m = mi & a.mask[j];
          double x = xi - a.r[3 * j], y = yi - a.r[3 * j + 1], z = zi - a.r[3 * j + 2];
          min_image_ref(a.box, x, y, z);
          const double r2 = x * x + y * y + z * z;
          if (m & MMNB_SITE_HAS_Q) {
            const double rs = a.rscreen[i] + a.rscreen[j];
            double b0, b1;
            if (r2 < rs * rs) {
              b1 = 1.0 / (rs * rs * rs);
              b0 = -0.5 * r2 * b1 + 1.5 / rs;
            } else {
              const double invr = 1.0 / sqrt(r2);
              b0 = invr;
              b1 = invr * invr * invr;
            }
            if (a.scale_e14) {
              b0 *= a.e14;
              b1 *= a.e14;
            }
            const double qj = a.q[j];
            v[0] += qj * b0;
            v[1] += qj * b1 * x;
            v[2] += qj * b1 * y;
            v[3] += qj * b1 * z;
          }
          if (m & MMNB_SITE_HAS_LJ) {
            const double sg = a.geometric ? a.sig[i] * a.sig[j]
                                          : (0.5 * (a.sig[i] + a.sig[j])) * (0.5 * (a.sig[i] + a.sig[j]));
            const double s6 = sg * sg * sg;
            const double b = 4 * sqrt(a.eps[i] * a.eps[j]) * s6;
            const double aa = b * s6;
            const double invr2 = 1.0 / r2;
            const double invr6 = invr2 * invr2 * invr2;
            double du = 12 * aa * invr6 * invr6 * invr2 - 6 * b * invr6 * invr2;
            double u = aa * invr6 * invr6 - b * invr6;
            if (a.scale_l14) {
              u *= a.l14;
              du *= a.l14;
            }
            elj += 0.5 * u;
            vir += 0.5 * du * r2;
            lf[0] += du * x;
            lf[1] += du * y;
            lf[2] += du * z;
          }
        }
      }
    }
  }
  // the site's terms into its first lane
  if (L > 1 && (KIND == kMesh64 || KIND == kMesh64Ik || a.do_excl))
#pragma unroll
    for (int k = 0; k < 4; k++)
      v[k] = lanes_sum<L>(v[k], c);
  if (a.do14)
#pragma unroll
    for (int k = 0; k < 3; k++)
      lf[k] = lanes_sum<L>(lf[k], c);
  if constexpr (k32) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      v32[k] = lanes_sum<L>(v32[k], c);
  }
  double e = 0;
  if (live && c == 0) {
    double p = v[0], ev[3] = {v[1], v[2], v[3]};
    if (a.have_sums) {
      p += a.phi[i];
      for (int d = 0; d < 3; d++)
        ev[d] += a.evec[3 * i + d];
    }
    if (a.have_ljf)
      for (int d = 0; d < 3; d++)
        lf[d] += a.ljf[3 * i + d];
    if (a.acc) {
      // fold the fixed-point sums into the FP64 site values (one site's words
      // are 64 contiguous bytes: four 16-byte loads)
      const longlong2 *o2 = reinterpret_cast<const longlong2 *>(a.acc + (size_t) i * 8);
      const longlong2 w01 = o2[0], w23 = o2[1], w45 = o2[2], w67 = o2[3];
      const long long o[7] = {w01.x, w01.y, w23.x, w23.y, w45.x, w45.y, w67.x};
      long long k[4] = {0, 0, 0, 0};
      if (k32)
        for (int d = 0; d < 4; d++)
          k[d] = __float2ll_rn(v32[d] * 4294967296.0f);
      p += (double) (o[0] + k[0]) * kFxInv;
      for (int d = 0; d < 3; d++) {
        ev[d] += (double) (o[1 + d] + k[1 + d]) * kFxInv;
        lf[d] += (double) o[4 + d] * kFxInv;
      }
    }
    if (a.do_self) {
      p -= a.self_a * qi;
      p += a.neutral_b;
    }
    e = qi * p;
    if (a.keep_fields) {
      a.phi[i] = p;
      for (int d = 0; d < 3; d++) {
        a.evec[3 * i + d] = ev[d];
        a.ljf[3 * i + d] = lf[d];
      }
    }
    if (a.f) {
      for (int d = 0; d < 3; d++) {
        const double f = qi * ev[d] + lf[d];
        a.f[3 * i + d] = a.assign_f ? f : a.f[3 * i + d] + f;
      }
    }
  }
  double rs = 0;
  if (a.lj_row) {
    // this block's slice of the per-row LJ energies (fixed slices, fixed order)
    const int per = (a.nrow + gridDim.x - 1) / gridDim.x;
    const int lo = min(a.nrow, (int) blockIdx.x * per), hi = min(a.nrow, lo + per);
    for (int k = lo + threadIdx.x; k < hi; k += blockDim.x)
      rs += a.lj_row[k];
  }
  double t[4] = {e, elj, vir, rs};
  block_sums<4>(t, sh);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 4; k++)
      a.part[4 * (size_t) blockIdx.x + k] = t[k];
    __threadfence();
    last = atomicAdd(a.counter, 1ull) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last)
    return;
  __threadfence();
  double s[4] = {0, 0, 0, 0};
  for (int b = threadIdx.x; b < (int) gridDim.x; b += kSiteThreads)
#pragma unroll
    for (int k = 0; k < 4; k++)
      s[k] += a.part[4 * (size_t) b + k];
  block_sums<4>(s, sh);
  if (threadIdx.x == 0) {
    double el = s[0], lj = s[1] + s[3];
    if (a.wsum) {
      // the water kernel's real-space Coulomb energy is a pair sum (not in phi)
      el += 2 * ((double) (long long) a.wsum[0] * kFxInv);
      lj += (double) (long long) a.wsum[1] * kFxInv;
    }
    const double elec = a.any_q ? el / 2 : 0;
    const double ljt = lj + a.tail;
    a.energy[0] = elec;
    a.energy[1] = ljt;
    a.energy[2] = a.tail;
    a.energy[3] = elec + ljt;
    *a.vir14 = s[2];
    *a.counter = 0ull;
    if (a.flags[kFlagListTrunc])
      a.flags[kFlagTruncEvals] += 1;
    if (a.status) {
      // over the bus to the waiting host: the block first, the ready word last
      volatile double *st = a.status;
      st[0] = elec;
      st[1] = ljt;
      st[2] = a.tail;
      st[3] = elec + ljt;
      volatile int *fl = reinterpret_cast<volatile int *>(a.status + 4);
      for (int k = 0; k < kFlagCount; k++)
        fl[k] = a.flags[k];
      __threadfence_system();
      reinterpret_cast<volatile unsigned long long *>(a.status)[mmnb_handle::kStatusReady] = 1ull;
    }
  }
}

// blocks of the site kernel for L lanes per site
static int site_grid(int nsite, int L) { return div_up((long) div_up(nsite, 32 / L) * 32, kSiteThreads); }

int site_blocks(const mmnb_handle *h) { return site_grid(h->nsite, kMaxOrder); }

// A lane per mesh plane up to this many sites, where a lane per site leaves much of the
// chip idle.  Shuffled boxes, the step in us, lanes per plane against per site: with ik
// 40,000, mixed order 4 12,288 sites 49.5 and 52.8, 36,000 82.9 and 86.8, order 7 68.8 and
// 83.3, 139.8 and 155.6, FP64 order 5 76.2 and 84.2, 162.7 and 160.6, order 7 93 and 118,
// 209 and 233; without, 14,000, FP64 order 5 10,500 sites 61.8 and 64.5, 15,000 80.1 and
// 79.5, 36,000 129.7 and 125.1, mixed order 7 12,288 56.9 and 59.4, 36,000 102 and 98.
// Mixed orders up to 5 without ik, where the lanes gain least (650 sites 28.0 and 29.9,
// 3,000 32.8 and 34.9, 12,288 45.4 and 47.4, 24,000 63.1 and 62.2), take a lane per site
// from 2,500 sites on: replicas that fill the chip together pay for the lanes' work (64 of
// 258 to 3,933 waters, 1,000 steps: 760 ms with 10,000 here, 731 with 2,500).
constexpr int site_lanes_max(int P, MeshKind kind)
{
  return kind == kMesh32Ik || kind == kMesh64Ik ? 40000 : kind == kMesh32 && P <= 5 ? 2500 : 14000;
}
// (site_words' loads, at 6 blocks an SM, want the chip filled: order 5 mixed, shuffled, point
// by point against them: 18,000 sites 58.0 and 60.8, 36,000 74.7 and 75.1, 98,304 161 and 150)
constexpr int kSiteWordsMin = 40000;

template <int P, MeshKind KIND>
static void launch_sites_p(mmnb_handle *h, const SiteArgs &a)
{
  constexpr int V = site_words(P, KIND);
  if (h->nsite <= site_lanes_max(P, KIND))
    k_sites<P, KIND, P, 1><<<site_grid(h->nsite, P), kSiteThreads, 0, h->stream>>>(a);
  else if (h->nsite > kSiteWordsMin && h->mesh[2] % V == 0)
    k_sites<P, KIND, 1, V><<<site_grid(h->nsite, 1), kSiteThreads, 0, h->stream>>>(a);
  else
    k_sites<P, KIND, 1, 1><<<site_grid(h->nsite, 1), kSiteThreads, 0, h->stream>>>(a);
}

template <MeshKind KIND>
static cudaError_t launch_sites_kind(mmnb_handle *h, const SiteArgs &a)
{
  switch (h->cfg.p3m_assignment_order) {
  case 2: launch_sites_p<2, KIND>(h, a); break;
  case 3: launch_sites_p<3, KIND>(h, a); break;
  case 4: launch_sites_p<4, KIND>(h, a); break;
  case 5: launch_sites_p<5, KIND>(h, a); break;
  case 6: launch_sites_p<6, KIND>(h, a); break;
  case 7: launch_sites_p<7, KIND>(h, a); break;
  default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_sites(mmnb_handle *h, const double *d_r, double *d_f, double *d_energy)
{
  const bool mixed = h->cfg.precision == MMNB_MIXED;
  const bool p3m = h->any_q && h->cfg.include_kspace && h->p3m;
  SiteArgs a{};
  a.nsite = h->nsite;
  a.do_self = (h->any_q && h->cfg.include_self) ? 1 : 0;
  a.do_excl = h->cfg.include_rspace ? 1 : 0;
  a.do14 = h->cfg.include_rspace && h->use_14 ? 1 : 0;
  a.geometric = h->cfg.geometric_combining_for_sigma;
  a.keep_fields = h->want_fields ? 1 : 0;
  a.assign_f = h->assign_forces ? 1 : 0;
  // what the site arrays hold: the FP64 pair kernels' sums, the k-sum's
  a.have_sums = (!mixed && h->cfg.include_rspace) || h->used_ksum ? 1 : 0;
  a.have_ljf = !mixed && h->cfg.include_rspace ? 1 : 0;
  a.box = h->box;
  a.eta = h->eta;
  a.self_a = h->eta * M_2_SQRTPI;
  // neutralising background for a charged system (src/eleclj.cpp:965-975)
  a.neutral_b = h->neutral_b;
  a.e14 = h->cfg.elec_1_4_scale_factor - 1;
  a.l14 = h->cfg.lj_1_4_scale_factor - 1;
  a.scale_e14 = fabs(h->cfg.elec_1_4_scale_factor - 1) > 1e-10;
  a.scale_l14 = fabs(h->cfg.lj_1_4_scale_factor - 1) > 1e-10;
  a.r = d_r;
  a.q = h->d_q;
  a.sig = h->d_sig;
  a.eps = h->d_eps;
  a.rscreen = h->d_rscreen;
  a.mask = h->d_mask;
  a.excl_ptr = h->d_excl_ptr;
  a.excl_idx = h->d_excl_idx;
  a.p14_ptr = h->d_p14_ptr;
  a.p14_idx = h->d_p14_idx;
  if (p3m) {
    a.mesh = mesh_args(h);
    a.mesh64 = h->d_mesh;
    a.egrid64 = h->d_egrid;
    a.mesh32 = h->d_mesh32;
    a.egrid32 = h->d_egrid32;
    a.nr = (size_t) h->mesh[0] * h->mesh[1] * h->mesh[2];
  }
  a.acc = mixed ? h->mx.acc : nullptr;
  a.phi = h->d_phi;
  a.evec = h->d_evec;
  a.ljf = h->d_ljf;
  a.f = d_f;
  a.part = h->d_site_part;
  a.lj_row = h->used_rows ? h->d_lj_row : nullptr;
  a.nrow = h->ngroup;
  a.any_q = h->any_q ? 1 : 0;
  a.wsum = h->used_fx ? h->d_wsum : nullptr;
  a.counter = h->d_wsum + 2;
  a.flags = h->d_flags;
  a.tail = h->cfg.include_lj_correction ? h->lj_correction : 0.0;
  a.energy = d_energy;
  a.vir14 = h->d_energy + 8;
  a.status = h->want_status ? h->d_status : nullptr;
  h->launches += 1;
  if (!p3m) {
    k_sites<0, kNoMesh, 2, 1><<<site_grid(h->nsite, 2), kSiteThreads, 0, h->stream>>>(a);
    return cudaGetLastError();
  }
  const bool ik = h->cfg.p3m_ik_differentiate != 0;
  if (mixed)
    return ik ? launch_sites_kind<kMesh32Ik>(h, a) : launch_sites_kind<kMesh32>(h, a);
  return ik ? launch_sites_kind<kMesh64Ik>(h, a) : launch_sites_kind<kMesh64>(h, a);
}

}  // namespace mmnb
