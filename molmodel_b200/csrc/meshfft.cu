// The P3M mesh solve in three kernels: real mesh -> spectrum -> times the influence
// function -> real mesh (p3m_field's two transforms, src/pppm.c:551-608).
//
//   * k_fft_planes: a block per x-plane.  Two real rows make one complex line along
//     z; the rows' half spectra are separated where the transform along y reads them.
//     The mixed form's fixed-point mesh is converted as it is read, and cleared;
//   * k_fft_lines: a block per tile of adjacent columns, along x forwards, times the
//     influence function (with ik also times -ik per component), and back;
//   * k_fft_planes_inv: y backwards, then z with two half spectra per complex line.
//
// A length is split as n = r1 r2, radices up to 12: X[k1 + r1 k2] = sum_b W_r2^(b k2)
// W_n^(b k1) sum_a W_r1^(a k1) x[b + r2 a] (Cooley and Tukey's), so a line is two
// passes, each with one DFT of its radix in a thread's registers.  The second pass
// forwards along x holds just the elements of the first pass backwards: the influence
// function is applied between them without a trip to shared memory.
//
// The library's transforms make four launches each way, and the fixed-point
// conversion and the product two more.  Profiled one by one with cold caches, mixed
// form: 96^3 points 48 -> 32 us, 48^3 35 -> 23 us; FP64: 56 -> 37 and 33 -> 24 us.  In
// a running program a third less: cold, the kernels wait for their instructions (11 of
// a warp's 18 cycles between two; a pass is straight code run once).  FP32
// reciprocal forces against FP64, nine lengths 20 to 108, six boxes of 512 waters each:
// 0.9-2.0e-6 before, 0.8-1.3e-6 now, lower at each.

#include "meshfft.cuh"

#include <cmath>
#include <vector>

namespace mmnb {

// ---- DFTs in registers -------------------------------------------------------

template <typename T>
struct alignas(2 * sizeof(T)) Cx {
  T x, y;
};

template <typename T>
__device__ __forceinline__ Cx<T> operator+(Cx<T> a, Cx<T> b) { return {a.x + b.x, a.y + b.y}; }
template <typename T>
__device__ __forceinline__ Cx<T> operator-(Cx<T> a, Cx<T> b) { return {a.x - b.x, a.y - b.y}; }
// a times (b.x + i S b.y): a twiddle factor of the forward table, or its conjugate
template <int S, typename T>
__device__ __forceinline__ Cx<T> twiddle(Cx<T> a, Cx<T> b)
{
  return S < 0 ? Cx<T>{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}
               : Cx<T>{a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y};
}

// cos and sin of 2 pi j / N
template <int N>
__device__ constexpr double unit_cos(int j)
{
  constexpr double c5[3] = {1, 0.30901699437494742410, -0.80901699437494742410};
  constexpr double c7[4] = {1, 0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
  constexpr double c8[5] = {1, 0.70710678118654752440, 0, -0.70710678118654752440, -1};
  constexpr double c9[5] = {1, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405};
  const int k = j > N / 2 ? N - j : j;
  return N == 5 ? c5[k % 3] : N == 7 ? c7[k % 4] : N == 8 ? c8[k % 5] : c9[k % 5];
}
template <int N>
__device__ constexpr double unit_sin(int j)
{
  constexpr double s5[3] = {0, 0.95105651629515357212, 0.58778525229247312917};
  constexpr double s7[4] = {0, 0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
  constexpr double s8[5] = {0, 0.70710678118654752440, 1, 0.70710678118654752440, 0};
  constexpr double s9[5] = {0, 0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676,
                            0.34202014332566873304};
  const int k = j > N / 2 ? N - j : j;
  const double s = N == 5 ? s5[k % 3] : N == 7 ? s7[k % 4] : N == 8 ? s8[k % 5] : s9[k % 5];
  return j > N / 2 ? -s : s;
}

// v -> its DFT of length R with exp(S 2 pi i jk / R), in place
template <int R, int S>
struct Dft;

template <int S>
struct Dft<2, S> {
  template <typename T>
  static __device__ __forceinline__ void run(Cx<T> (&v)[2])
  {
    const Cx<T> a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  }
};
template <int S>
struct Dft<3, S> {
  template <typename T>
  static __device__ __forceinline__ void run(Cx<T> (&v)[3])
  {
    const T s = T(S * 0.86602540378443864676);
    const Cx<T> t = v[1] + v[2], u = v[1] - v[2], m = {v[0].x - T(0.5) * t.x, v[0].y - T(0.5) * t.y};
    v[0] = v[0] + t;
    v[1] = {m.x - s * u.y, m.y + s * u.x};
    v[2] = {m.x + s * u.y, m.y - s * u.x};
  }
};
template <int S>
struct Dft<4, S> {
  template <typename T>
  static __device__ __forceinline__ void run(Cx<T> (&v)[4])
  {
    const Cx<T> a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3], d = v[1] - v[3];
    const Cx<T> e = {-S * d.y, S * d.x};
    v[0] = a + c;
    v[1] = b + e;
    v[2] = a - c;
    v[3] = b - e;
  }
};
// odd primes: the pairs j, R - j by their sums and differences
template <int R, int S>
struct DftPrime {
  template <typename T>
  static __device__ __forceinline__ void run(Cx<T> (&v)[R])
  {
    constexpr int H = R / 2;
    Cx<T> t[H + 1], u[H + 1], o = v[0];
#pragma unroll
    for (int j = 1; j <= H; j++) {
      t[j] = v[j] + v[R - j];
      u[j] = v[j] - v[R - j];
      o = o + t[j];
    }
#pragma unroll
    for (int k = 1; k <= H; k++) {
      Cx<T> m = v[0], n = {T(0), T(0)};
#pragma unroll
      for (int j = 1; j <= H; j++) {
        const T c = T(unit_cos<R>(j * k % R)), s = T(S * unit_sin<R>(j * k % R));
        m.x += c * t[j].x;
        m.y += c * t[j].y;
        n.x += s * u[j].x;
        n.y += s * u[j].y;
      }
      t[0] = {m.x - n.y, m.y + n.x};
      u[0] = {m.x + n.y, m.y - n.x};
      // (v[k], v[R - k] are not read again: t and u hold all of them)
      v[k] = t[0];
      v[R - k] = u[0];
    }
    v[0] = o;
  }
};
template <int S>
struct Dft<5, S> : DftPrime<5, S> {};
template <int S>
struct Dft<7, S> : DftPrime<7, S> {};
// A B with A, B coprime (Good's mapping: no twiddle factors)
template <int A, int B, int S>
struct DftCoprime {
  static __device__ constexpr int out(int k1, int k2)
  {
    int k = k1;
    while (k % B != k2)
      k += A;
    return k;
  }
  template <typename T>
  static __device__ __forceinline__ void run(Cx<T> (&v)[A * B])
  {
    Cx<T> w[A][B];
#pragma unroll
    for (int b = 0; b < B; b++) {
      Cx<T> t[A];
#pragma unroll
      for (int a = 0; a < A; a++)
        t[a] = v[(B * a + A * b) % (A * B)];
      Dft<A, S>::run(t);
#pragma unroll
      for (int a = 0; a < A; a++)
        w[a][b] = t[a];
    }
#pragma unroll
    for (int a = 0; a < A; a++) {
      Dft<B, S>::run(w[a]);
#pragma unroll
      for (int b = 0; b < B; b++)
        v[out(a, b)] = w[a][b];
    }
  }
};
template <int S>
struct Dft<6, S> : DftCoprime<2, 3, S> {};
template <int S>
struct Dft<10, S> : DftCoprime<2, 5, S> {};
template <int S>
struct Dft<12, S> : DftCoprime<3, 4, S> {};
// A B with twiddle factors W_AB^(b k1)
template <int A, int B, int S>
struct DftSplit {
  template <typename T>
  static __device__ __forceinline__ void run(Cx<T> (&v)[A * B])
  {
    constexpr int N = A * B;
    Cx<T> w[A][B];
#pragma unroll
    for (int b = 0; b < B; b++) {
      Cx<T> t[A];
#pragma unroll
      for (int a = 0; a < A; a++)
        t[a] = v[b + B * a];
      Dft<A, S>::run(t);
#pragma unroll
      for (int k = 0; k < A; k++) {
        const int j = b * k % N;
        if (j == 0)
          w[k][b] = t[k];
        else if (4 * j == N)
          w[k][b] = {-S * t[k].y, S * t[k].x};
        else
          w[k][b] = twiddle<-1>(t[k], Cx<T>{T(unit_cos<N>(j)), T(S * unit_sin<N>(j))});
      }
    }
#pragma unroll
    for (int k = 0; k < A; k++) {
      Dft<B, S>::run(w[k]);
#pragma unroll
      for (int b = 0; b < B; b++)
        v[k + A * b] = w[k][b];
    }
  }
};
template <int S>
struct Dft<8, S> : DftSplit<2, 4, S> {};
template <int S>
struct Dft<9, S> : DftSplit<3, 3, S> {};

template <int R>
struct Radix {
  static constexpr int value = R;
};
// f with the radix as a compile-time constant (the same for the whole grid)
template <typename F>
__device__ __forceinline__ void by_radix(int r, F &&f)
{
  switch (r) {
  case 2: f(Radix<2>()); break;
  case 3: f(Radix<3>()); break;
  case 4: f(Radix<4>()); break;
  case 5: f(Radix<5>()); break;
  case 6: f(Radix<6>()); break;
  case 7: f(Radix<7>()); break;
  case 8: f(Radix<8>()); break;
  case 9: f(Radix<9>()); break;
  case 10: f(Radix<10>()); break;
  case 12: f(Radix<12>()); break;
  }
}

// q = t / d and t - q d for t < 2^21 (the quotient's distance from the next integer,
// 0.5 / d, is above the rounding of the product)
struct Divider {
  int d;
  float inv;
  __device__ __forceinline__ int div(int t, int &rest) const
  {
    const int q = (int) ((t + 0.5f) * inv);
    rest = t - q * d;
    return q;
  }
};

// a length n = r1 r2 and its factors exp(-2 pi i j / n)
template <typename T>
struct Axis {
  int n, r1, r2;
  Divider d1, d2;
  const Cx<T> *w;
};

template <typename T>
struct FftArgs {
  Axis<T> x, y, z;
  int nzh, np;   // points of a half spectrum; pairs of rows of a plane
  Divider dh;    // nzh
  int sa, p2;    // complex line along z: elements, and of the r2 of a first-pass output
  int buf;       // elements of the first of the two buffers
  int tc;        // columns of a tile along x (a power of two), and its log2
  int ltc;
  int m;         // ny nzh: columns
};

__device__ __forceinline__ double mesh_value(double t) { return t; }
__device__ __forceinline__ float mesh_value(unsigned long long t) { return (float) ((double) (long long) t * kFxInv); }

// Threads of a plane's block.  FP32 at 768 leaves 80 registers and spills 268 bytes a
// thread forwards, 80 back; 640 and 512 spill less and nothing and take as long: 32,768
// waters mixed 149 us a step at 768, 149.5 at 640, 150.5 at 512 (shuffled 150.5, 151.9 and
// 152.9), 8,192 waters 66, 65 and 66.
template <typename T>
constexpr int kPlaneThreads = sizeof(T) == 8 ? 512 : 768;
constexpr int kLineThreads = 256;

template <typename T, typename In>
__global__ void __launch_bounds__(kPlaneThreads<T>) k_fft_planes(FftArgs<T> a, In *__restrict__ in,
                                                                 Cx<T> *__restrict__ out)
{
  extern __shared__ __align__(16) unsigned char fft_smem[];
  Cx<T> *const A = reinterpret_cast<Cx<T> *>(fft_smem), *const B = A + a.buf;
  const int tid = threadIdx.x, nt = blockDim.x, nz = a.z.n, nzh = a.nzh;
  in += (size_t) blockIdx.x * a.y.n * nz;
  out += (size_t) blockIdx.x * a.m;
  // z, first pass: rows 2p and 2p + 1 as one complex line
  by_radix(a.z.r1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r2 = a.z.r2;
    for (int t = tid; t < a.np * r2; t += nt) {
      int b;
      const int p = a.z.d2.div(t, b);
      const bool two = 2 * p + 1 < a.y.n;
      In *const row = in + (size_t) 2 * p * nz + b;
      Cx<T> v[R];
      {
        In u[R], w[R];
#pragma unroll
        for (int k = 0; k < R; k++) {
          u[k] = row[k * r2];
          w[k] = two ? row[nz + k * r2] : In(0);
        }
        if (sizeof(T) == 4) {
          // (the fixed-point mesh is left cleared for the next evaluation)
#pragma unroll
          for (int k = 0; k < R; k++) {
            row[k * r2] = In(0);
            if (two)
              row[nz + k * r2] = In(0);
          }
        }
#pragma unroll
        for (int k = 0; k < R; k++)
          v[k] = {mesh_value(u[k]), mesh_value(w[k])};
      }
      Dft<R, -1>::run(v);
      Cx<T> *const o = A + p * a.sa + b;
      o[0] = v[0];
#pragma unroll
      for (int k = 1; k < R; k++)
        o[k * a.p2] = twiddle<-1>(v[k], a.z.w[b * k]);
    }
  });
  __syncthreads();
  by_radix(a.z.r2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r1 = a.z.r1;
    for (int t = tid; t < a.np * r1; t += nt) {
      int k;
      const int p = a.z.d1.div(t, k);
      const Cx<T> *const i = A + p * a.sa + k * a.p2;
      Cx<T> v[R];
#pragma unroll
      for (int b = 0; b < R; b++)
        v[b] = i[b];
      Dft<R, -1>::run(v);
      Cx<T> *const o = B + p * nz + k;
#pragma unroll
      for (int b = 0; b < R; b++)
        o[b * r1] = v[b];
    }
  });
  __syncthreads();
  // y, first pass: row 2p's spectrum is (Z[k] + conj Z[n - k]) / 2, row 2p + 1's
  // (Z[k] - conj Z[n - k]) / 2i
  by_radix(a.y.r1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r2 = a.y.r2;
    for (int t = tid; t < nzh * r2; t += nt) {
      int k;
      const int b = a.dh.div(t, k), kc = k ? nz - k : 0;
      Cx<T> v[R];
#pragma unroll
      for (int j = 0; j < R; j++) {
        const int y = b + r2 * j;
        const Cx<T> *const line = B + (y >> 1) * nz;
        const Cx<T> u = line[k], w = line[kc];
        const T h = T(0.5);
        v[j] = y & 1 ? Cx<T>{h * (u.y + w.y), h * (w.x - u.x)} : Cx<T>{h * (u.x + w.x), h * (u.y - w.y)};
      }
      Dft<R, -1>::run(v);
      Cx<T> *const o = A + b * nzh + k;
      o[0] = v[0];
#pragma unroll
      for (int j = 1; j < R; j++)
        o[j * r2 * nzh] = twiddle<-1>(v[j], a.y.w[b * j]);
    }
  });
  __syncthreads();
  by_radix(a.y.r2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r1 = a.y.r1;
    for (int t = tid; t < nzh * r1; t += nt) {
      int k;
      const int k1 = a.dh.div(t, k);
      const Cx<T> *const i = A + k1 * R * nzh + k;
      Cx<T> v[R];
#pragma unroll
      for (int b = 0; b < R; b++)
        v[b] = i[b * nzh];
      Dft<R, -1>::run(v);
      Cx<T> *const o = out + (size_t) k1 * nzh + k;
#pragma unroll
      for (int b = 0; b < R; b++)
        o[(size_t) b * r1 * nzh] = v[b];
    }
  });
}

// spec: times the influence function, transformed along x both ways: in place, or with
// IK, where blockIdx.y says which, the three spectra -i k_d of it (the product
// (k im, -k re)) and the potential's own to the four parts of `field`.  (One block for
// all four in turn took 29 us on 54^3 points, 189 blocks of three warps; 13 so.)
template <typename T, bool IK>
__global__ void __launch_bounds__(kLineThreads) k_fft_lines(FftArgs<T> a, const T *__restrict__ green,
                                                            const double *__restrict__ kvec,
                                                            Cx<T> *__restrict__ spec, Cx<T> *__restrict__ field)
{
  extern __shared__ __align__(16) unsigned char fft_smem[];
  const int tc = a.tc, n = a.x.n, m = a.m;
  Cx<T> *const A = reinterpret_cast<Cx<T> *>(fft_smem), *const B = A + n * tc;
  const int c = threadIdx.x & (tc - 1), col = blockIdx.x * tc + c;
  const int step = blockDim.x >> a.ltc, first = threadIdx.x >> a.ltc;
  const bool live = col < m;
  by_radix(a.x.r1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r2 = a.x.r2;
    for (int b = first; b < r2; b += step) {
      Cx<T> v[R];
#pragma unroll
      for (int j = 0; j < R; j++)
        v[j] = live ? spec[(size_t) (b + r2 * j) * m + col] : Cx<T>{T(0), T(0)};
      Dft<R, -1>::run(v);
      Cx<T> *const o = A + b * tc + c;
      o[0] = v[0];
#pragma unroll
      for (int j = 1; j < R; j++)
        o[j * r2 * tc] = twiddle<-1>(v[j], a.x.w[b * j]);
    }
  });
  __syncthreads();
  // second pass forwards, the product, first pass backwards
  const int d = IK ? blockIdx.y : 3;
  by_radix(a.x.r2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r1 = a.x.r1;
    for (int k1 = first; k1 < r1; k1 += step) {
      const Cx<T> *const i = A + k1 * R * tc + c;
      Cx<T> v[R];
#pragma unroll
      for (int j = 0; j < R; j++)
        v[j] = i[j * tc];
      Dft<R, -1>::run(v);
#pragma unroll
      for (int j = 0; j < R; j++) {
        const size_t g = (size_t) (k1 + r1 * j) * m + col;
        const T s = live ? green[g] : T(0);
        v[j].x *= s;
        v[j].y *= s;
        if (IK && d < 3) {
          const T k = live ? (T) kvec[3 * g + d] : T(0);
          v[j] = {k * v[j].y, -k * v[j].x};
        }
      }
      Dft<R, 1>::run(v);
      Cx<T> *const o = B + k1 * tc + c;
      o[0] = v[0];
#pragma unroll
      for (int j = 1; j < R; j++)
        o[j * r1 * tc] = twiddle<1>(v[j], a.x.w[k1 * j]);
    }
  });
  __syncthreads();
  by_radix(a.x.r1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r2 = a.x.r2;
    for (int q = first; q < r2; q += step) {
      const Cx<T> *const i = B + q * R * tc + c;
      Cx<T> v[R];
#pragma unroll
      for (int j = 0; j < R; j++)
        v[j] = i[j * tc];
      Dft<R, 1>::run(v);
      Cx<T> *const o = (IK ? field + (size_t) d * n * m : spec) + col;
      if (live)
#pragma unroll
        for (int j = 0; j < R; j++)
          o[(size_t) (q + r2 * j) * m] = v[j];
    }
  });
}

// blockIdx.y: which mesh (with field spectra the three field meshes, then the potential)
template <typename T>
__global__ void __launch_bounds__(kPlaneThreads<T>) k_fft_planes_inv(FftArgs<T> a, const Cx<T> *__restrict__ spec,
                                                                     const Cx<T> *__restrict__ fspec,
                                                                     T *__restrict__ mesh, T *__restrict__ fmesh)
{
  extern __shared__ __align__(16) unsigned char fft_smem[];
  Cx<T> *const A = reinterpret_cast<Cx<T> *>(fft_smem), *const B = A + a.buf;
  const int tid = threadIdx.x, nt = blockDim.x, nz = a.z.n, ny = a.y.n, nzh = a.nzh;
  const int d = blockIdx.y;
  const Cx<T> *const in = (fspec ? fspec + (size_t) d * a.x.n * a.m : spec) + (size_t) blockIdx.x * a.m;
  T *const out = (fspec && d < 3 ? fmesh + (size_t) d * a.x.n * ny * nz : mesh) + (size_t) blockIdx.x * ny * nz;
  by_radix(a.y.r1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r2 = a.y.r2;
    for (int t = tid; t < nzh * r2; t += nt) {
      int k;
      const int b = a.dh.div(t, k);
      Cx<T> v[R];
#pragma unroll
      for (int j = 0; j < R; j++)
        v[j] = in[(size_t) (b + r2 * j) * nzh + k];
      Dft<R, 1>::run(v);
      Cx<T> *const o = A + b * nzh + k;
      o[0] = v[0];
#pragma unroll
      for (int j = 1; j < R; j++)
        o[j * r2 * nzh] = twiddle<1>(v[j], a.y.w[b * j]);
    }
  });
  __syncthreads();
  by_radix(a.y.r2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r1 = a.y.r1;
    for (int t = tid; t < nzh * r1; t += nt) {
      int k;
      const int k1 = a.dh.div(t, k);
      const Cx<T> *const i = A + k1 * R * nzh + k;
      Cx<T> v[R];
#pragma unroll
      for (int b = 0; b < R; b++)
        v[b] = i[b * nzh];
      Dft<R, 1>::run(v);
      Cx<T> *const o = B + k1 * nzh + k;
#pragma unroll
      for (int b = 0; b < R; b++)
        o[b * r1 * nzh] = v[b];
    }
  });
  __syncthreads();
  // z, first pass: Z = X + i Y of the full spectra of rows 2p and 2p + 1, whose
  // elements without a partner are real (what the half spectrum holds beside is not
  // part of a real mesh)
  by_radix(a.z.r1, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r2 = a.z.r2;
    for (int t = tid; t < a.np * r2; t += nt) {
      int b;
      const int p = a.z.d2.div(t, b);
      const bool two = 2 * p + 1 < ny;
      const Cx<T> *const row = B + 2 * p * nzh;
      Cx<T> v[R];
#pragma unroll
      for (int j = 0; j < R; j++) {
        const int q = b + r2 * j;
        const bool back = 2 * q > nz;
        const int k = back ? nz - q : q;
        Cx<T> x = row[k], y = two ? row[nzh + k] : Cx<T>{T(0), T(0)};
        if (q == 0 || 2 * q == nz)
          x.y = y.y = T(0);
        v[j] = back ? Cx<T>{x.x + y.y, y.x - x.y} : Cx<T>{x.x - y.y, x.y + y.x};
      }
      Dft<R, 1>::run(v);
      Cx<T> *const o = A + p * a.sa + b;
      o[0] = v[0];
#pragma unroll
      for (int j = 1; j < R; j++)
        o[j * a.p2] = twiddle<1>(v[j], a.z.w[b * j]);
    }
  });
  __syncthreads();
  by_radix(a.z.r2, [&](auto radix) {
    constexpr int R = decltype(radix)::value;
    const int r1 = a.z.r1;
    for (int t = tid; t < a.np * r1; t += nt) {
      int k;
      const int p = a.z.d1.div(t, k);
      const bool two = 2 * p + 1 < ny;
      const Cx<T> *const i = A + p * a.sa + k * a.p2;
      Cx<T> v[R];
#pragma unroll
      for (int b = 0; b < R; b++)
        v[b] = i[b];
      Dft<R, 1>::run(v);
      T *const o = out + (size_t) 2 * p * nz + k;
#pragma unroll
      for (int b = 0; b < R; b++) {
        o[b * r1] = v[b].x;
        if (two)
          o[nz + b * r1] = v[b].y;
      }
    }
  });
}

// ---- plans ---------------------------------------------------------------------

// n = r1 r2 with both radices available and as near each other as can be
static bool split_length(int n, int &r1, int &r2)
{
  constexpr int kRadix[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 12};
  r1 = 0;
  for (int a : kRadix)
    for (int b : kRadix)
      if (a <= b && a * b == n)
        r1 = a, r2 = b;
  return r1 > 0;
}

// shared memory of a plane's block for elements of `bytes`
static int plane_elements(const int n[3], int r1z, int r2z, int &buf)
{
  const int np = (n[1] + 1) / 2, nzh = n[2] / 2 + 1;
  buf = std::max(np * r1z * (r2z | 1), n[1] * nzh);
  return buf + std::max(np * n[2], n[1] * nzh);
}

constexpr int kPlaneSmem = 227 * 1024;

bool mesh_fft_fits(const int n[3], int bytes)
{
  int r1, r2, buf;
  for (int d = 0; d < 3; d++)
    if (!split_length(n[d], r1, r2))
      return false;
  return plane_elements(n, r1, r2, buf) * 2 * bytes <= kPlaneSmem;
}

size_t mesh_fft_table_size(const int n[3]) { return (size_t) n[0] + n[1] + n[2]; }

template <typename T>
static void fill_table(const int n[3], void *host)
{
  Cx<T> *o = static_cast<Cx<T> *>(host);
  for (int d = 0; d < 3; d++)
    for (int j = 0; j < n[d]; j++) {
      const double x = 2 * M_PI * j / n[d];
      *o++ = {(T) cos(x), (T) -sin(x)};
    }
}

void mesh_fft_table(const int n[3], int bytes, void *host)
{
  if (bytes == 8)
    fill_table<double>(n, host);
  else
    fill_table<float>(n, host);
}

static Divider divider(int d) { return {d, 1.0f / d}; }

template <typename T>
static FftArgs<T> fft_args(const int n[3], const void *table, int &plane_smem, int &plane_threads)
{
  FftArgs<T> a;
  const Cx<T> *w = static_cast<const Cx<T> *>(table);
  Axis<T> *const ax[3] = {&a.x, &a.y, &a.z};
  for (int d = 0; d < 3; d++) {
    ax[d]->n = n[d];
    split_length(n[d], ax[d]->r1, ax[d]->r2);
    ax[d]->d1 = divider(ax[d]->r1);
    ax[d]->d2 = divider(ax[d]->r2);
    ax[d]->w = w;
    w += n[d];
  }
  a.nzh = n[2] / 2 + 1;
  a.np = (n[1] + 1) / 2;
  a.dh = divider(a.nzh);
  a.p2 = a.z.r2 | 1;
  a.sa = a.z.r1 * a.p2;
  plane_smem = plane_elements(n, a.z.r1, a.z.r2, a.buf) * (int) sizeof(Cx<T>);
  a.m = n[1] * a.nzh;
  // tiles of 16 columns (whole 128-byte lines), of 8 where they leave the chip idle
  a.ltc = a.m >= 16 * 148 ? 4 : 3;
  a.tc = 1 << a.ltc;
  // a thread per DFT of the widest pass
  const int most = std::max(a.np * std::max(a.z.r1, a.z.r2), a.nzh * std::max(a.y.r1, a.y.r2));
  plane_threads = std::min(kPlaneThreads<T>, div_up(most, 32) * 32);
  return a;
}

template <typename K>
static cudaError_t launch_smem(K kernel, dim3 grid, int threads, int smem, cudaStream_t s, void **args)
{
  // (always the most any plan takes: handles of several threads launch the same kernel)
  const cudaError_t e =
      cudaFuncSetAttribute((const void *) kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPlaneSmem);
  if (e != cudaSuccess)
    return e;
  return cudaLaunchKernel((const void *) kernel, grid, dim3(threads), args, smem, s);
}

template <typename T, typename In>
static cudaError_t solve(const int n[3], const void *table, In *in, const T *green, const double *kvec, Cx<T> *spec,
                         Cx<T> *fspec, T *out, T *fout, cudaStream_t s)
{
  int smem, threads;
  FftArgs<T> a = fft_args<T>(n, table, smem, threads);
  void *p1[] = {&a, &in, &spec};
  cudaError_t e = launch_smem(k_fft_planes<T, In>, dim3(n[0]), threads, smem, s, p1);
  if (e != cudaSuccess)
    return e;
  const int lthreads = std::min(kLineThreads, div_up(a.tc * std::max(a.x.r1, a.x.r2), 32) * 32);
  const int lsmem = 2 * n[0] * a.tc * (int) sizeof(Cx<T>);
  void *p2[] = {&a, &green, &kvec, &spec, &fspec};
  e = launch_smem(fspec ? k_fft_lines<T, true> : k_fft_lines<T, false>, dim3(div_up(a.m, a.tc), fspec ? 4 : 1), lthreads, lsmem, s, p2);
  if (e != cudaSuccess)
    return e;
  const Cx<T> *cspec = spec, *cfspec = fspec;
  void *p3[] = {&a, &cspec, &cfspec, &out, &fout};
  return launch_smem(k_fft_planes_inv<T>, dim3(n[0], fspec ? 4 : 1), threads, smem, s, p3);
}

cudaError_t mesh_solve(const MeshSolve<double> &m, double *in, cudaStream_t s)
{
  return solve<double, double>(m.n, m.table, in, m.green, m.kvec, reinterpret_cast<Cx<double> *>(m.spec),
                               reinterpret_cast<Cx<double> *>(m.fspec), m.out, m.fout, s);
}

cudaError_t mesh_solve(const MeshSolve<float> &m, unsigned long long *in, cudaStream_t s)
{
  return solve<float, unsigned long long>(m.n, m.table, in, m.green, m.kvec, reinterpret_cast<Cx<float> *>(m.spec),
                                          reinterpret_cast<Cx<float> *>(m.fspec), m.out, m.fout, s);
}

}  // namespace mmnb
