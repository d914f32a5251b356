// Internal declarations of libmmnb (sm_100a).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <cufft.h>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/mmnb.h"

namespace mmnb {

constexpr int kCheb = 512;          // Chebyshev segments (include/cheby.h:10)
constexpr int kChebWMax = 2048;     // segments of the rigid-water FP64 kernel's continued table
constexpr int kMaxGroup = 8;        // sites per group handled by the pair kernels
constexpr int kTailMax = 512;       // segments of the general kernel's continuation
constexpr int kMaxOrder = 7;        // P3M assignment order (src/pppm.c:61)
constexpr int kWarp = 32;

// flag words shared by the list-build kernels (device memory)
enum FlagIndex {
  kFlagRebuild = 0,    // 1 when this evaluation rebuilds the list
  kFlagOverflow = 1,   // largest row length seen when a row overflowed
  kFlagError = 2,      // MMNB_ERR_DEVICE when a device-side check failed
  kFlagMaxRow = 3,     // largest row length of the last build
  // 4: evaluations, 5: rebuilds, 6: the list check's block counter
  kFlagPruneFull = 7,  // 1: the water kernel reads the full rows and writes the pruned ones
  kFlagPruneValid = 8, // 1 while the pruned rows belong to the current build
  kFlagListTrunc = 9,  // 1 while the current list has rows cut at their capacity
  kFlagTruncEvals = 10,// evaluations finished on such a list since the last mmnb_check
  kFlagForceRebuild = 11, // 1: the next list check rebuilds (set by the host, cleared by the check)
  kFlagCount = 12
};

// Box in the form the kernels use (cubic and orthorhombic).
struct Box {
  double L[3];      // edge lengths
  double invL[3];   // 1 / L, as the reference computes it (src/rspace.c:399-404)
};

// Cell-list geometry (src/nbrlist.cpp:9-17, 84-123).
struct CellGeom {
  int n;            // cells per dimension
  double lc[3];     // cell edge = L * (1.0 / n)
  double c2;        // (cutoff + width)^2
};

// Fixed-point scale of the mixed form's accumulators: 2^32 units per unit of
// potential, field or force (range +-2^31, resolution 2.3e-10).
constexpr double kFxScale = 4294967296.0;
constexpr double kFxInv = 1.0 / 4294967296.0;
constexpr int kAccStride = 8;  // phi, Ex, Ey, Ez, Lx, Ly, Lz, (pad) per site

// Launch choices that do not change any result (mmnb_autotune times them).
struct Tuning {
  int water_minb = 5;      // rigid-water pair kernel: 4 or 5 resident warps per SM / 4 (128 or 96 registers)
  int spread_planes = 2;   // mixed P3M spread: 0 one thread per site, 1 P threads per site (x planes),
                           // 2 P lanes per site along z (coalesced reductions)
  int p3m_side = 1;        // P3M mesh work on the side stream (1) or in line (0)
  int water64_warps = 12;  // FP64 rigid-water kernel: warps per block (12, 10 or 8; fewer when the
                           // rings and the table do not fit in shared memory)
};

// Device buffers of the mixed-precision form.
struct MixedBufs {
  float4 *site = nullptr;        // sorted, padded slots: offset from the anchor (xyz), charge (w); or,
                                 // for the rigid-water kernel, three packed slots per group
  float4 *par = nullptr;         // sorted, padded slots: sigma, sqrt(epsilon), rscreen, mask bits
  double4 *anchor = nullptr;     // sorted groups: anchor position (FP64)
  float4 *anc32 = nullptr;       // rigid-water kernel, sorted groups: the anchor's offset from the corner
                                 // of its list cell (FP32) and the cell's coordinates (10 bits each, in w)
  long long *acc = nullptr;      // per site (original order), kAccStride fixed-point values
};

// Wave vectors and sums of the ordinary Ewald reciprocal space (kspace.cu)
struct EwaldSum {
  bool made = false;
  int nk = 0, nrow = 0, nmax = 0;
  double rec[3] = {0, 0, 0};
  int4 *row = nullptr;      // rows of consecutive n_z: (n_x, n_y, first n_z, its index)
  short4 *kint = nullptr;   // integer n of each wave vector
  double *ak2 = nullptr;    // 2 a_k
  double2 *sk = nullptr;    // 2 a_k S(k)
  double2 *part = nullptr;  // partial S(k) of the structure factor's blocks
};

// Stage timing with CUDA events recorded on the handle's stream.  Each
// evaluation starts with a "start" mark; a stage's time is the interval from
// the previous mark to its own.
struct Timing {
  bool on = false;
  std::vector<cudaEvent_t> pool;   // reused between resets
  std::vector<std::string> names;  // one per recorded mark
  size_t used = 0;
};

}  // namespace mmnb

struct mmnb_handle {
  mmnb_config cfg{};
  int nsite = 0, ngroup = 0, maxgs = 1, G = 1;   // G: padded sites per group slot
  int dev = 0;
  cudaStream_t stream = nullptr;       // stream every launch goes to
  cudaStream_t own_stream = nullptr;   // created by mmnb_create, destroyed by mmnb_destroy
  // P3M charge assignment and FFTs run on `side`, forked from and joined back
  // into `stream`, concurrently with the list and pair kernels
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  std::string err;

  // derived settings
  double rc = 0, nlw = 0, eta = 0, rlo2 = 0, rhi2 = 0, inv_sw = 0;  // inv_sw = 1/(rhi2 - rlo2)
  mmnb::Box box{};
  double volume = 0, min_diameter = 0;
  bool params_set = false, any_q = false, any_lj = false, has_rscreen = false;
  bool any_gexcl = false, use_14 = false;
  bool water = false;                // every group is [O(q, LJ), H(q), H(q)] with no screening or group exclusions
  // ... and every O has the same charge, sigma and epsilon and every H the
  // same charge (the rigid-water kernel then copies only the H offsets)
  bool water_uni = false;
  float uni_qO = 0, uni_qH = 0, uni_sig = 0, uni_seps = 0;
  double uni64[4] = {0, 0, 0, 0};    // the same in FP64
  bool want_fields = false;          // this evaluation must produce per-site potential and field
  bool want_virial = false;          // this evaluation's pair kernels also sum the virial's pair term
  bool used_fx = false;              // the last evaluation ran the mixed water kernel: fixed-point energies
  bool used_rows = false;            // the last evaluation ran another pair kernel: energies per row
  double totA = 0, totB = 0, lj_correction = 0, neutral_b = 0;

  // host topology
  std::vector<int> group;            // 2*ngroup
  std::vector<int> group_of_site;
  std::vector<int> excl_ptr, excl_idx;   // per-site excluded partners, both directions, sorted
  std::vector<int> p14_ptr, p14_idx;     // per-site 1-4 partners, both directions, sorted
  std::vector<int> gexcl_ptr, gexcl_idx; // per-group group-excluded partners, sorted

  // device topology and parameters (original site order)
  int *d_group = nullptr;
  int *d_excl_ptr = nullptr, *d_excl_idx = nullptr;
  int *d_p14_ptr = nullptr, *d_p14_idx = nullptr;
  int *d_gexcl_ptr = nullptr, *d_gexcl_idx = nullptr;
  int *d_mask = nullptr;
  double *d_q = nullptr, *d_sig = nullptr, *d_eps = nullptr, *d_rscreen = nullptr;
  double cheb_min = 0, cheb_max = 0, cheb_inv_dx = 0;
  // the rigid-water FP64 kernel's table: cheb_w_nseg x (c0, c1), then x (c2, c3); then
  // the general one's continuation from cheb_max on, tail_nseg x 8 coefficients
  double *d_cheb_w = nullptr;
  int cheb_w_nseg = 0, tail_nseg = 0;
  double tail_inv = 0;               // 1 / width of a tail segment
  // 512 x 4: the cubics of -eta d/d(eta) of the table (mmnb_virial)
  double *d_cheb_d = nullptr;

  // neighbour list
  mmnb::CellGeom cg{};
  int ncell3 = 0;
  int nstencil = 0;                  // offsets incl. (0,0,0) first
  int *d_stencil = nullptr;          // 3 ints per offset
  int *d_cell_rank = nullptr;        // reference cell index -> Morton rank
  int *d_cell_of_rank = nullptr;     // Morton rank -> reference cell index
  int *d_cell_of_group = nullptr;    // per group, reference numbering
  int *d_cell_count = nullptr;       // per rank, then per chunk of ranks (cell_words)
  int *d_cell_start = nullptr;       // per rank, ncell3+1
  int *d_cell_head = nullptr;        // per rank, the cell's last group to arrive
  int *d_slot = nullptr;             // per group, the group that arrived in its cell before
  int *d_sorted = nullptr;           // sorted position -> group
  int *d_rank = nullptr;             // group -> sorted position
  double *d_anchor = nullptr;        // 3*ngroup current anchors (original order)
  double *d_last = nullptr;          // 3*ngroup anchors at the last rebuild
  double *d_anchor_sorted = nullptr; // 3*ngroup anchors at the last rebuild, sorted order
  float4 *d_anchor32 = nullptr;      // the same, wrapped into the box, FP32 (list pre-test)
  double *d_top2 = nullptr;          // per-block top-2 displacements
  int top2_blocks = 0;
  int rowcap = 0;
  int *d_nbr = nullptr;              // ngroup * rowcap, sorted positions
  int *d_nbr_count = nullptr;        // ngroup
  // rows pruned to rc + prune_margin for the rigid-water kernel (same rowcap),
  // and the sorted anchors at the last prune
  int *d_pnbr = nullptr, *d_pcount = nullptr;
  double *d_plast = nullptr;
  double prune_margin = 0;           // 0: no pruning
  int *d_flags = nullptr;            // mmnb::kFlagCount ints
  // bumped by every (re)allocation of a device buffer: a captured graph holds
  // the addresses of its launch, so it is replayed only while this is unchanged
  long buf_gen = 0;
  long graph_gen = -1;               // buf_gen when mmnb_graph_capture ran
  int *h_flags = nullptr;            // pinned mirror
  long rebuilds = 0, evals = 0;
  long launches = 0;                 // kernels of this library launched so far
  long launch_per_eval = 0;          // kernels in the captured evaluation
  bool first = true;
  int force_rebuild_next = 0;

  // sorted, padded site data (FP64 form)
  double4 *d_sr = nullptr;           // ngroup*G sites: offset from the anchor, q
  double4 *d_sp = nullptr;           // sig, sqrt(eps), rscreen, -
  double4 *d_sanchor = nullptr;      // sorted groups: anchor, first site and site masks
  int *d_site_of_slot = nullptr;     // ngroup*G -> original site (or -1)

  // outputs (original order)
  double *d_phi = nullptr, *d_evec = nullptr, *d_ljf = nullptr;
  double *d_lj_row = nullptr;        // pair kernels but the mixed water one: LJ energy of each row (sorted order)
  double *d_site_part = nullptr;     // site kernel: per block, its four partial sums
  // mmnb_virial: the same kernels' virial term per row, molecule ranges,
  // masses and per-molecule sums (allocated on first use)
  double *d_vir_row = nullptr;
  int *d_vir_mol = nullptr;
  double *d_vir_molw = nullptr, *d_vir_mass = nullptr;
  int vir_mol_cap = 0;
  // [0], [1]: fixed-point Coulomb and LJ pair energies of the mixed water kernel;
  // [2]: block counter of the site kernel's last-block reduction;
  // [3]: row counter of the FP64 pair kernels; [4]: the mixed water kernel's
  // fixed-point virial term
  unsigned long long *d_wsum = nullptr;
  // parameter gradients (allocated on first use): six per-site outputs, dL/dF
  double *d_bwd = nullptr;
  size_t bwd_cap = 0;
  double *h_bwd = nullptr;  // pinned: the gradient slots come back in one copy
  // potential at points: scratch kept from call to call (at most 64 MB)
  double *d_esp = nullptr;
  size_t esp_cap = 0;
  bool grad_ready = false;           // the last evaluation was mmnb_forward's and nothing changed since
  // FP64 dipole solve for a mixed-form handle, which has no FP64 meshes or plans
  double *d_gmesh = nullptr;
  cufftDoubleComplex *d_gmeshk = nullptr;
  cufftHandle gplan_r2c = 0, gplan_c2r = 0;
  // host copies of the site parameters, and the LJ classes of the tail:
  // distinct (sigma, epsilon) as printed with %12.6g, their site counts, and
  // each site's class (-1 without LJ)
  std::vector<double> hpar;          // as copied to the device: q, sigma, epsilon, r_screen, masks
  std::vector<double> cls_sig, cls_eps;
  std::vector<long> cls_n;
  std::vector<int> site_cls;
  double *d_energy = nullptr;        // 4 doubles; [8]: the 1-4 pairs' virial term
  // host path staging
  double *d_r = nullptr, *d_f = nullptr;
  double *h_r = nullptr, *h_f = nullptr, *h_out = nullptr;  // pinned

  // P3M
  bool p3m = false;
  int mesh[3] = {0, 0, 0};
  // the mesh solve's own transforms (meshfft.cu) where they take the mesh: twiddle
  // factors of the FP32 and FP64 forms (null: the plans below)
  void *d_fft32 = nullptr, *d_fft64 = nullptr;
  cufftHandle plan_r2c = 0, plan_c2r = 0;
  double *d_mesh = nullptr;
  cufftDoubleComplex *d_meshk = nullptr;
  double *d_green = nullptr;         // nx*ny*(nz/2+1)
  double *d_kvec = nullptr;          // 3 per k-point (ik differentiation)
  double *d_egrid = nullptr;         // 3 real meshes (ik)
  cufftDoubleComplex *d_egridk = nullptr;
  double *d_chi_part = nullptr;      // per-block partials of the mesh error sum
  double p3m_chi = 0;                // the mesh's dimensionless RMS force error estimate
  bool eta_optimised = false;        // eta chosen by p3m_optimize's criterion
  // mixed-precision P3M
  cufftHandle plan_r2c32 = 0, plan_c2r32 = 0;
  float *d_mesh32 = nullptr;
  cufftComplex *d_meshk32 = nullptr;
  float *d_green32 = nullptr;
  float *d_egrid32 = nullptr;        // ik differentiation: three FP32 field meshes
  cufftComplex *d_egridk32 = nullptr;
  unsigned long long *d_mesh_fx = nullptr;

  // ordinary Ewald
  bool kspace = false;
  mmnb::EwaldSum ew;                 // made with the handle, or on the first potential at points

  // mixed form
  mmnb::MixedBufs mx;

  mmnb::Timing timing;
  mmnb::Tuning tune;

  // one captured evaluation (mmnb_graph_capture / mmnb_graph_launch)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
  // the host call's own graph (d_r -> d_f, d_energy), captured on first use
  // and dropped whenever rows, parameters, box or stream change
  cudaGraph_t hgraph = nullptr;
  cudaGraphExec_t hgraph_exec = nullptr;
  long host_launch_per_eval = 0;
  // the host call copies the forces back in chunks and adds each as it lands
  static constexpr int kChunks = 2;
  cudaEvent_t ev_chunk[kChunks] = {};
  cudaEvent_t ev_eval = nullptr;  // the host call's evaluation has ended (or failed)
  // ... and, replaying its graph, copies the positions in kInChunks pieces on
  // a stream of its own: the graph's mesh branch assigns the charges of each
  // piece as it lands (mixed form), everything else waits for the last piece
  static constexpr int kInChunks = 2;
  cudaStream_t copy_in = nullptr;
  cudaEvent_t ev_in[kInChunks] = {};
  cudaEvent_t ev_free = nullptr;  // the handle's stream has let go of d_r
  bool in_chunks = false;         // set while that graph is captured
  // the host call's status block in mapped pinned memory: k_sites writes
  // the energies [0, 4), the flags (ints, from double 4 on) and then, after a
  // system-wide fence, the ready word; the host spins on that word instead of
  // copying the block back after the evaluation
  static constexpr int kStatusDoubles = 16;
  static constexpr int kStatusReady = 15;  // double slot of the ready word
  double *h_status = nullptr;
  double *d_status = nullptr;  // its device alias
  bool assign_forces = false;  // this evaluation writes d_f instead of adding to it
  bool used_ksum = false;      // the last evaluation ran the k-sum
  bool want_status = false;    // set while the host call records its evaluation: no
                               // other evaluation writes the block
  bool capturing = false;
  bool crowded = false;  // set while a batch of many replicas records this one's step
};

namespace mmnb {

// ---- launchers (defined in the .cu files) ----------------------------------
// drop the host call's graph (called when what it captured changes)
void drop_host_graph(mmnb_handle *h);
// LJ tail correction (src/eleclj.cpp:1247-1266) for totals A and B; linear in both
double lj_tail_ab(const mmnb_handle *h, double A, double B);
// anchors, rebuild decision; then the cells and sorted order of a rebuild (a no-op
// launch when not due); the rows are built by the site-sorting kernels (nbrlist.cuh)
cudaError_t launch_list_check(mmnb_handle *h, const double *d_r, int force);
cudaError_t launch_list_cells(mmnb_handle *h);
cudaError_t launch_sort_sites(mmnb_handle *h, const double *d_r);
cudaError_t launch_rspace_fp64(mmnb_handle *h);
cudaError_t launch_prep_mixed(mmnb_handle *h, const double *d_r);
cudaError_t launch_rspace_mixed(mmnb_handle *h);
cudaError_t launch_rspace_water(mmnb_handle *h);
cudaError_t launch_sort_water64(mmnb_handle *h, const double *d_r);
cudaError_t launch_rspace_water64(mmnb_handle *h);
cudaError_t launch_p3m_green(mmnb_handle *h, double eta, double *chi);
// charge assignment and FFT round trip
cudaError_t launch_p3m_fp64(mmnb_handle *h, const double *d_r);
// FP64 meshes and plans of the adjoint's dipole solve: spread/spreadk hold one
// mesh (three with ik differentiation); solvek/solve the summed ik spectrum
// and its transform (ik only; otherwise the solve happens in place)
struct P3mScratch {
  double *spread = nullptr, *solve = nullptr;
  cufftDoubleComplex *spreadk = nullptr, *solvek = nullptr;
  bool own = false;              // the solve is the own transforms' (no plans)
  cufftHandle r2c = 0, c2r = 0;
};
// d_psi += mesh potential of the dipoles q_j g_j (g: 3 per site), FP64
cudaError_t launch_p3m_dipole_fp64(mmnb_handle *h, const double *d_r, const double *d_g, const P3mScratch &s,
                                   double *d_psi);
// d_psi += reciprocal-sum potential of the dipoles q_j g_j
cudaError_t launch_kspace_dipole(mmnb_handle *h, const double *d_r, const double *d_g, double *d_psi);
// (assigned: the charges are on the mesh already, launch_spread_mixed_range's)
cudaError_t launch_p3m_mixed(mmnb_handle *h, const double *d_r, bool assigned);
// write back and drop [p, p + bytes) from the host cores' caches (hostmem.cpp)
void evict_host_lines(const void *p, size_t bytes);

// the mixed charge assignment of sites [lo, hi) alone (the mesh words are integer
// sums, so the pieces give the mesh of one launch over all sites, bit for bit)
cudaError_t launch_spread_mixed_range(mmnb_handle *h, const double *d_r, int lo, int hi);
cudaError_t launch_green32(mmnb_handle *h);
// wave vectors of the handle's kspace_cutoff, eta and box (drops what e held)
cudaError_t ewald_make(mmnb_handle *h, EwaldSum &e);
void ewald_free(EwaldSum &e);
// S(k) of the sites at d_r (with d_g: of the dipoles q g) into e.sk
cudaError_t launch_ewald_structure(mmnb_handle *h, const EwaldSum &e, const double *d_r, const double *d_g);
// d_phi = (add: +=) potential of e.sk at the n points, + neutral; d_evec (or null) the field
cudaError_t launch_ewald_sum(mmnb_handle *h, const EwaldSum &e, int n, const double *d_pts, double neutral,
                             double *d_phi, double *d_evec, bool add);
// interpolation, exclusions, self terms, forces and energies
cudaError_t launch_sites(mmnb_handle *h, const double *d_r, double *d_f, double *d_energy);
int site_blocks(const mmnb_handle *h);  // at most this many blocks

// helpers shared by the .cu files
void timing_mark(mmnb_handle *h, const char *name);
int set_global_error(int code, const std::string &msg);  // read back by mmnb_last_error(NULL)

#ifdef __CUDACC__
// the head of a kernel that launch_after launches
__device__ __forceinline__ void after_previous()
{
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
}

// binary search of key in CSR row `row` (sorted)
__device__ __forceinline__ bool csr_has(const int *ptr, const int *idx, int row, int key)
{
  int lo = ptr[row], hi = ptr[row + 1] - 1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    const int v = idx[mid];
    if (key < v)
      hi = mid - 1;
    else if (key > v)
      lo = mid + 1;
    else
      return true;
  }
  return false;
}

// (-1)^n / (n! (2n + 1)): erf(x) = 2 x / sqrt(pi) sum_n of these x^(2n)
static __constant__ double kErfSeries[16] = {
    1.0, -1.0 / 3, 1.0 / 10, -1.0 / 42, 1.0 / 216, -1.0 / 1320, 1.0 / 9360, -1.0 / 75600, 1.0 / 685440,
    -1.0 / 6894720, 1.0 / 76204800, -1.0 / 918086400, 1.0 / 11975040000.0, -1.0 / 168129561600.0,
    1.0 / 2528170444800.0, -1.0 / 40537905408000.0};

// b0 = erfc(eta r)/r and b1 = -2 d b0 / d(r^2) for r^2 below the table, where
// eta r <= kErfSeriesMax: b0 = 1/r - erf(eta r)/r, from erf's Maclaurin series
// (16 terms: the first one left out is below 1e-17 of the sum).  A few site pairs
// of a row take this branch and the rest of the warp waits for them: 45 FP64
// operations here, several hundred for erfc and exp (rigid-water FP64 kernel 259 ->
// 226 us on 32,768 waters).
constexpr double kErfSeriesMax = 0.85;

// p = sqrt(pi) erf(x) / (2 x) and d = dp/dy at y = x^2
__device__ __forceinline__ void erf_series(double y, double &p, double &d)
{
  p = kErfSeries[15];
  d = 0;
#pragma unroll
  for (int n = 14; n >= 0; n--) {
    d = fma(d, y, p);
    p = fma(p, y, kErfSeries[n]);
  }
}

__device__ __forceinline__ void ewald_short(double eta2, double two_eta_rsqrtpi, double r2, double &b0, double &b1)
{
  const double rinv = rsqrt(r2);
  double p, d;
  erf_series(eta2 * r2, p, d);
  b0 = fma(-two_eta_rsqrtpi, p, rinv);
  b1 = fma(2 * two_eta_rsqrtpi * eta2, d, rinv * rinv * rinv);
}

// minimum image of one site displacement, rounded as the reference rounds it
__device__ __forceinline__ void min_image_ref(const Box &b, double &x, double &y, double &z)
{
  x = __dadd_rn(x, __dmul_rn(-b.L[0], floor(__dadd_rn(__dmul_rn(x, b.invL[0]), 0.5))));
  y = __dadd_rn(y, __dmul_rn(-b.L[1], floor(__dadd_rn(__dmul_rn(y, b.invL[1]), 0.5))));
  z = __dadd_rn(z, __dmul_rn(-b.L[2], floor(__dadd_rn(__dmul_rn(z, b.invL[2]), 0.5))));
}

// anchor displacement with the reference's minimum-image rounding
__device__ __forceinline__ double anchor_disp(const Box &b, double4 ri, double4 rj, double &x, double &y, double &z,
                                              double &sx, double &sy, double &sz)
{
  x = __dsub_rn(ri.x, rj.x);
  y = __dsub_rn(ri.y, rj.y);
  z = __dsub_rn(ri.z, rj.z);
  sx = __dmul_rn(-b.L[0], floor(__dadd_rn(__dmul_rn(x, b.invL[0]), 0.5)));
  sy = __dmul_rn(-b.L[1], floor(__dadd_rn(__dmul_rn(y, b.invL[1]), 0.5)));
  sz = __dmul_rn(-b.L[2], floor(__dadd_rn(__dmul_rn(z, b.invL[2]), 0.5)));
  x = __dadd_rn(x, sx);
  y = __dadd_rn(y, sy);
  z = __dadd_rn(z, sz);
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

#endif

// Segments of the continued table the rigid-water FP64 kernel uses.  Past 1.2 rc^2 the
// reference evaluates erfc and exp; the cubics continued there are within 1.1e-10 of
// them for b0 and 1.3e-7 for b1, relatively (rc 9, eta 0.35; 3e-8 for b1 at eta rc =
// 2.3), in b1 an absolute 4e-15 to 8e-13 where the table itself, inside its range, is
// off by up to 1.5e-6.  From eta rc = 2.3 on, where erfc(eta r) has fallen below ~4e-4,
// that is below 1e-12 of the pair's terms; under it the exact functions are taken.
inline double table_segments(const mmnb_handle *h)
{
  return h->eta * h->rc >= 2.3 ? h->cheb_w_nseg : kCheb;
}

inline int div_up(long a, long b) { return (int) ((a + b - 1) / b); }

// The list's cells in chunks of 2^chunk_shift, at most kMaxChunks of them: the counts
// of the cells, padded to whole 16-byte words, then those of the chunks
constexpr int kMaxChunks = 4096;
inline int chunk_shift(int ncell3)
{
  int s = 6;
  while (div_up(ncell3, 1 << s) > kMaxChunks)
    s++;
  return s;
}
inline int chunk_at(int ncell3) { return div_up(ncell3, 4) * 4; }
inline int cell_words(int ncell3) { return chunk_at(ncell3) + div_up(ncell3, 1 << chunk_shift(ncell3)); }

#ifdef __CUDACC__
// A kernel behind another one in the handle's stream: on a box small enough its blocks
// come up while the other still runs and wait there for all of it (after_previous), so
// what a launch takes passes beside that kernel's work.  On larger boxes the waiting
// blocks hold room that the mesh work or the pair kernel's first blocks would use.
// 216 waters' k-sum 83.4 -> 80.3 us, 512 waters' loss gradient 228 -> 215, 6,000 waters
// with virial 287 -> 275.  The step in us without and with it, mixed: 2,048 waters 41.0 and
// 39.2, 8,192 66.0 and 64.2, 12,288 78.6 and 76.7, 16,384 107.1 and 107.1, 24,576 111.7 and
// 112.5; FP64 51.1 and 47.9, 103.6 and 103.1, 127.9 and 127.2, 177.5 and 177.7, 204.9 and
// 210.2; solution of 4,600 groups 84.7 and 81.3, of 9,000 124.6 and 124.4, of 18,500 207.7
// and 208.1.  A batch of replicas that are more than this together does without it (64 of
// them 766 -> 759 ms per 1,000 steps).
constexpr int kAfterGroups = 12288;

template <typename... K, typename... A>
inline cudaError_t launch_after(const mmnb_handle *h, void (*kernel)(K...), dim3 grid, int threads, size_t smem,
                                const A &...args)
{
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = h->stream;
  c.attrs = &at;
  c.numAttrs = h->ngroup <= kAfterGroups && !h->crowded ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, K(args)...);
}
#endif

}  // namespace mmnb
