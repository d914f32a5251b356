// The P3M mesh solve's interface (meshfft.cu).
#pragma once

#include "mmnb_internal.cuh"

namespace mmnb {

template <typename T>
struct MeshSolve {
  int n[3];
  const void *table;     // mesh_fft_table's, on the device
  const T *green;
  const double *kvec;    // per half-spectrum point, for the field spectra
  void *spec, *fspec;    // half spectrum; null, or room for four (ik differentiation)
  T *out, *fout;         // potential mesh; the three field meshes
};

// whether the solve takes this mesh with elements of `bytes` (4 or 8)
bool mesh_fft_fits(const int n[3], int bytes);
// twiddle factors: complex elements, and their values
size_t mesh_fft_table_size(const int n[3]);
void mesh_fft_table(const int n[3], int bytes, void *host);
// charges -> potential (and field) meshes; `in` may be `out` in the FP64 form
cudaError_t mesh_solve(const MeshSolve<double> &m, double *in, cudaStream_t s);
cudaError_t mesh_solve(const MeshSolve<float> &m, unsigned long long *in, cudaStream_t s);

}  // namespace mmnb
