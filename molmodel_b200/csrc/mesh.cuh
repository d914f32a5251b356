// B-splines on the P3M mesh: what charge assignment and interpolation share.
#pragma once

#include "mmnb_internal.cuh"

namespace mmnb {

struct MeshArgs {
  int n[3];
  double A[9];      // mesh-scaled inverse lattice, tensor_t layout: s = A r
  int nsite;
};

// Nearest mesh point and offset of a particle at mesh coordinate s
// (src/pppm.c:533-548): returns the first of the P assigned points and
// w = delta + 1/2 in [0, 1].
template <int P>
__device__ __forceinline__ int bspline_base(double s, double &w)
{
  int j;
  double delta;
  if (P % 2) {
    j = (int) floor(s + 0.5);
    delta = s - j;
  } else {
    j = (int) floor(s);
    delta = s - (j + 0.5);
  }
  w = delta + 0.5;
  return j - ((P + 1) / 2 - 1);
}

// Weights W[p] and negated derivatives ND[p] of the points base + p.
template <int P, typename T>
__device__ __forceinline__ void bspline_eval(T w, T *W, T *ND)
{
  T m[P], prev[P];
  m[0] = T(1);
#pragma unroll
  for (int k = 2; k <= P; k++) {
    const T inv = T(1) / T(k - 1);
#pragma unroll
    for (int i = 0; i < k - 1; i++)
      prev[i] = m[i];
#pragma unroll
    for (int i = 0; i < k; i++) {
      const T a = i < k - 1 ? prev[i] : T(0);
      const T b = i > 0 ? prev[i - 1] : T(0);
      m[i] = ((w + T(i)) * a + (T(k) - w - T(i)) * b) * inv;
    }
  }
#pragma unroll
  for (int p = 0; p < P; p++) {
    const int i = P - 1 - p;
    W[p] = m[i];
    const T a = i < P - 1 ? prev[i] : T(0);
    const T b = i > 0 ? prev[i - 1] : T(0);
    ND[p] = b - a;
  }
}

__device__ __forceinline__ int wrap_idx(int i, int n)
{
  i %= n;
  return i < 0 ? i + n : i;
}

// A particle's mesh points: weights, negated derivatives and wrapped points along x
// and y, and along z those of NZ points from `first` on (all P of them, or the one
// of a lane).  Arithmetic in T from the FP64 mesh coordinates.
template <int P, int NZ, typename T>
struct MeshRows {
  T wx[P], dx[P], wy[P], dy[P], wz[NZ], dz[NZ];
  int ix[P], iy[P], iz[NZ];
};

template <int P, int NZ, typename T>
__device__ __forceinline__ void mesh_rows(const MeshArgs &m, const double *__restrict__ r, int first,
                                          MeshRows<P, NZ, T> &o)
{
  const double x = r[0], y = r[1], z = r[2];
  T wz[P], dz[P];
  double w;
  const int b0 = bspline_base<P>(m.A[0] * x + m.A[3] * y + m.A[6] * z, w);
  bspline_eval<P, T>((T) w, o.wx, o.dx);
  const int b1 = bspline_base<P>(m.A[1] * x + m.A[4] * y + m.A[7] * z, w);
  bspline_eval<P, T>((T) w, o.wy, o.dy);
  const int b2 = bspline_base<P>(m.A[2] * x + m.A[5] * y + m.A[8] * z, w);
  bspline_eval<P, T>((T) w, wz, dz);
  int jx = wrap_idx(b0, m.n[0]), jy = wrap_idx(b1, m.n[1]), jz = wrap_idx(b2, m.n[2]);
#pragma unroll
  for (int p = 0; p < P; p++) {
    o.ix[p] = jx;
    o.iy[p] = jy;
    jx = jx + 1 == m.n[0] ? 0 : jx + 1;
    jy = jy + 1 == m.n[1] ? 0 : jy + 1;
    if (NZ == P || p == first) {
      o.wz[NZ == P ? p : 0] = wz[p];
      o.dz[NZ == P ? p : 0] = dz[p];
      o.iz[NZ == P ? p : 0] = jz;
    }
    jz = jz + 1 == m.n[2] ? 0 : jz + 1;
  }
}

// The same for a particle's P lanes from lane `first` of the warp on, lane c taking the
// point z = base + c: three of them work out an axis each and hand it to the others
// (every lane of the warp calls).
template <int P, typename T>
__device__ __forceinline__ void mesh_rows_lanes(const MeshArgs &m, const double *__restrict__ r, int first, int c,
                                                MeshRows<P, 1, T> &o)
{
  const int d = c < 2 ? c : 2;
  T W[P], D[P];
  double w;
  const int b = bspline_base<P>(m.A[d] * r[0] + m.A[3 + d] * r[1] + m.A[6 + d] * r[2], w);
  bspline_eval<P, T>((T) w, W, D);
  const int j = wrap_idx(b, m.n[d]);
  const unsigned all = 0xffffffffu;
  int jx = __shfl_sync(all, j, first), jy = __shfl_sync(all, j, first + 1), jz = __shfl_sync(all, j, first + 2);
#pragma unroll
  for (int p = 0; p < P; p++) {
    o.ix[p] = jx;
    o.iy[p] = jy;
    jx = jx + 1 == m.n[0] ? 0 : jx + 1;
    jy = jy + 1 == m.n[1] ? 0 : jy + 1;
    o.wx[p] = __shfl_sync(all, W[p], first);
    o.dx[p] = __shfl_sync(all, D[p], first);
    o.wy[p] = __shfl_sync(all, W[p], first + 1);
    o.dy[p] = __shfl_sync(all, D[p], first + 1);
    const T wz = __shfl_sync(all, W[p], first + 2), dz = __shfl_sync(all, D[p], first + 2);
    if (p == c) {
      o.wz[0] = wz;
      o.dz[0] = dz;
      o.iz[0] = jz;
    }
    jz = jz + 1 == m.n[2] ? 0 : jz + 1;
  }
}

// sum of v over the L lanes [first, first + L) of a particle, into its first lane
// (c: the lane's place among them; every lane of the warp calls)
template <int L, typename T>
__device__ __forceinline__ T lanes_sum(T v, int c)
{
#pragma unroll
  for (int off = 4; off >= 1; off >>= 1) {
    if (off >= L)  // (one lane: nothing to add)
      continue;
    const T t = __shfl_down_sync(0xffffffffu, v, off);
    if (c + off < (2 * off < L ? 2 * off : L))
      v += t;
  }
  return v;
}

inline MeshArgs mesh_args(const mmnb_handle *h)
{
  MeshArgs m;
  for (int d = 0; d < 3; d++)
    m.n[d] = h->mesh[d];
  for (int i = 0; i < 9; i++)
    m.A[i] = 0;
  // inverse of the diagonal lattice as the reference's inverse() computes it,
  // rows scaled by the mesh size (src/pppm.c:428, 523-525)
  const double xx = h->box.L[0], yy = h->box.L[1], zz = h->box.L[2];
  const double det = xx * yy * zz;
  const double id = 1.0 / det;
  m.A[0] = id * (yy * zz) * h->mesh[0];
  m.A[4] = id * (xx * zz) * h->mesh[1];
  m.A[8] = id * (xx * yy) * h->mesh[2];
  m.nsite = h->nsite;
  return m;
}

}  // namespace mmnb
