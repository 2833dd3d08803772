// Internal interface between the C ABI (hst_capi.cu) and the kernels
// (hst_*.cu).  Not installed; the public interface is include/hst_gpu.h.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <unordered_set>
#include <utility>
#include <vector>

#include "../../include/hst_gpu.h"

namespace hst {

// Sizes and device pointers of one field: everything a launch needs.
struct Geometry {
  int nx, ny, nz;      // deck sizes
  int nxd, nzd;        // padded transform sizes (2 nxd physical x points, nzd z points)
  int nxB, nzT, rows;  // nx+1, 2nz+1, ny+4
  int ncol;            // nxB * nzT Fourier columns
  long nf;             // complex elements of one field (ncol * rows)
  int P, PL;           // lanes of a line-solve group: of the substep and the D0 and DY kinds, of the other kinds of hst_gpu_line_solve
  int Ty, nyT;         // rows and number of the transforms' y tiles (the last may reach beyond ny)
  int EY;              // rows of the y tile that holds the four ghost rows (Ty of a z plan, else 4)
  int mp;              // mixed precision: Z, Pp, Q and their transforms in FP32 (complex64)
  // 0, or (in the view of the four ghost rows that the edge transforms take)
  // ny: the z-inverse then reads rows -2, -1, ny, ny+1 of V
  int edge_gap;
  // members of an ensemble advanced together (1 for a single field): every
  // per-field buffer holds nmem members one after another (fields nf
  // elements a member, Z 3 nyT Ty nzd nxB, Pp 6 nyT Ty nzd nxB, Q 6 ncol ny), the
  // tables are shared, and the substep's kernels cover all members in one
  // launch each
  int nmem;
};

struct DeviceState {
  double2* F[7];        // V1 V2 V3 OLD1 OLD2 RHS1 RHS2, (iy fastest, ghost rows included)
  double2* Z;           // z-inverse of V: [3][nyT][nzd][nxB][Ty]
  double2* Pp;          // x-forward of the products: [6][nyT][nzd][nxB][Ty]
  double2* Q;           // spectral products: [6][ncol][ny] (the first five in the substep)
  double* der;          // der(0:ny-1, 0:3, -2:2)
  double* derS;         // the same, slab-major for the line-solve groups (slab_major)
  double* derL;         // the same for groups of PL lanes (D2V, ETA, POISSON of hst_gpu_line_solve)
  double* derU;         // der's distinct rows, coefficient-major (DerRows); nderU of them, 0: not used
  int* derI;            // the distinct row of each row
  int nderU;
  double* d0tab;        // the D0 matrix factored for the line-solve group (d0_factor)
  double* y;            // y(-2:ny+1)
  double* dyl;          // dyl(0:ny-1)
  double* gdamp;        // gdamp(-nz:nz, 0:nx)
  double2* twx;         // exp(-2 pi i e / (2 nxd)), then the x plan's tables (x_twiddles)
  double2* twz;         // exp(-2 pi i e / nzd), then the z plan's tables (z_twiddles)
  float2* twxf;         // the same tables in FP32 (mixed precision)
  float2* twzf;
  unsigned long long* cfl;  // running max (bits of a non-negative double)
  int* err;                 // set by a kernel whose bounded wait ran out
  // TMA maps of Z, Pp and the ghost rows' buffers (make_x_maps; the ...2 of two components at a time)
  CUtensorMap tmZ, tmPp, tmPp2, tmZg, tmPpg, tmPpg2;
  CUtensorMap tmPz, tmPgz;             // of Pp and Ppg for the z-forward kernel (make_z_maps)
  // The products of the four ghost rows (-2, -1, ny, ny+1) transformed like
  // the interior ones (null when their shear-periodic images are exact):
  // Zg [3][nzd][nxB][EY], Ppg [6][nzd][nxB][EY], Qg [6][ncol][4], in the
  // transforms' precision
  double2 *Zg, *Ppg, *Qg;
  int nsm;        // SMs of the device
  double* stats;  // outstats scratch: block partials of the moments (stats_partials() a block),
                  // of the three gradients (one a block each), then the 24 results
  // the reference-layout buffers of the per-piece path (allocated by its
  // first call): VVdz [3][ny+4][nx+1][nzd], VVdx and VVdp [3][ny+4][nzd][nxd+1]
  double2 *vvdz, *vvdx, *vvdp;
  // kernels whose shared-memory limit has been raised in this context
  // (owned by the context; null: raise it at every launch)
  std::unordered_set<const void*>* configured;
};

// Raises kernel k's dynamic shared-memory limit to `bytes`, once per context
// (the attribute belongs to the function in the current context; setting it
// at every launch costs a driver call each time).
template <typename K>
inline cudaError_t smem_limit(const DeviceState& d, K k, int bytes) {
  const void* key = reinterpret_cast<const void*>(k);
  if (d.configured && d.configured->count(key)) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && d.configured) d.configured->insert(key);
  return e;
}

// Launches kernel k with programmatic stream serialization.  No kernel triggers
// its dependents early, so k's blocks start when the last block of its
// predecessor in the stream has ended: what is hidden is the launch latency and
// the reading of the tables (96^2 x 64: 62 -> 58 us a substep; 1 % or less at the
// larger sizes).  The predecessor's writes need not be visible yet, so every
// kernel waits (wait_predecessor, hst_dev.cuh) before it touches anything that
// the substep's other kernels write or read; as every kernel of a substep does,
// the wait orders a kernel after all that come before it.
template <typename... KA, typename... A>
inline cudaError_t launch_after(void (*k)(KA...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = attr;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, KA(std::forward<A>(args))...);
}

// Scalars of one substep of the column kernel.
struct SubstepScalars {
  double ode0, ode1, ode2, deltat, lambda;
  double s2now, gsoft;
  double dgx, dgz;
  double sx_t, sz_t;  // wrap displacements at t
  double sx_n, sz_n;  // at t + dt_sub
  int damp_hard;
  int yuni;      // the y grid is uniform (ystretch 0): y(r + 32) - y(r) = ytile
  double ytile;  // 32 ly / ny
};

struct PhysScalars {
  double alfa0, beta0, ni, S;
  double rdx, rdz, factor;  // 1/dx, 1/dz, 1/(2 nxd nzd)
};

cudaError_t launch_zinv(const Geometry& g, const DeviceState& d, cudaStream_t st);
// np = 5: the products uu - vv, ww - vv, uv, vw, uw that the right-hand sides
// take, as the components 0..4 of Pp and Q; 6: uu, vv, ww, uv, vw, uw
cudaError_t launch_xprod(const Geometry& g, const DeviceState& d, const PhysScalars& ph, int want_cfl, int np,
                         cudaStream_t st);
cudaError_t launch_zfwd(const Geometry& g, const DeviceState& d, int np, cudaStream_t st);
// the right-hand sides streamed through shared memory (hst_rhs.cu)
cudaError_t launch_rhs_tiled(const Geometry& g, const DeviceState& d, const PhysScalars& ps, const SubstepScalars& sc,
                             int exact, int nonlin, cudaStream_t st);
// the same row by row from global memory (hst_kernels.cu)
cudaError_t launch_rhs_rows(const Geometry& g, const DeviceState& d, const PhysScalars& ph, const SubstepScalars& sc,
                            int exact, int nonlin, cudaStream_t st);
// the implicit half (hst_solve.cu): the exact_shift shift of RHS1/2, OLD1/2,
// and the solves in two passes (half 0, then 1) from RHS1/2 into V1..V3, whose
// factors go to Pp
cudaError_t launch_shift(const Geometry& g, const DeviceState& d, const PhysScalars& ps, const SubstepScalars& sc,
                         cudaStream_t st);
cudaError_t launch_solve_half(const Geometry& g, const DeviceState& d, const PhysScalars& ps, const SubstepScalars& sc,
                              int half, cudaStream_t st);
// lanes of a solver group for ny rows and this many columns
int line_lanes(int ny, long columns);
// of k_line_solve, whose factors lie in shared memory
int line_lanes_shared(int ny);
// whether the solvers have room for groups of P lanes; the width that
// HST_LINE_LANES asks for, where they do (0: none)
bool line_lanes_fit(int ny, int P);
int line_lanes_asked(int ny);
// der(0:ny-1, 0:3, -2:2) in the slab-major order of groups of P lanes; the
// doubles that any P takes
std::vector<double> slab_major(const std::vector<double>& der, int ny, int P);
size_t slab_der_doubles(int ny);
cudaError_t launch_line_solve(const Geometry& g, const DeviceState& d, const PhysScalars& ph, int sys, double lambda,
                              int src, int dst, double sx, double sz, cudaStream_t st);
cudaError_t launch_fill_ghosts(const Geometry& g, const DeviceState& d, const PhysScalars& ph, int field, double sx,
                               double sz, cudaStream_t st);
// the factored D0 matrix of the line-solve group (P of g) into d.d0tab,
// from d.der; d0_table_doubles: the table's size for any group of ny rows
cudaError_t launch_d0_table(const Geometry& g, const DeviceState& d, cudaStream_t st);
size_t d0_table_doubles(int ny);
// outstats (src/hst_stats.f90:136-285): block count of the moments' reduction,
// the moments and (exz not null) the column energies exz(-nz:nz, 0:nx), the
// wall-normal gradients (hst_solve.cu; *blocks: its block count), the results
int stats_blocks(const Geometry& g, int nsm);
cudaError_t launch_stats_moments(const Geometry& g, const DeviceState& d, const PhysScalars& ps, double gsoft,
                                 double* partial, double* exz, cudaStream_t st);
cudaError_t launch_dy_sums(const Geometry& g, const DeviceState& d, const PhysScalars& ps, double sx, double sz,
                           double* partial, int* blocks, cudaStream_t st);
cudaError_t launch_stats_final(const Geometry& g, const DeviceState& d, const double* pm, const double* pg, int nblk_dy,
                               double ly_w, double ni, double ly, double* out, cudaStream_t st);
// moment partials a reduction block writes
int stats_partials();
// compute_pressure (src/hst_pressure.f90:35-110): the right-hand side into
// RHS1 (after the transforms), and the (0,0) mode into dst (after the
// POISSON solve)
cudaError_t launch_pressure_rhs(const Geometry& g, const DeviceState& d, const PhysScalars& ps, double s2now,
                                double sx, double sz, cudaStream_t st);
cudaError_t launch_pressure_mean(const Geometry& g, const DeviceState& d, double ly, int dst, cudaStream_t st);
// the per-piece path (hst_pieces.cu; the line transforms in hst_transforms.cu):
// kind 0 z line, 1 c2r x line, 2 r2c x line; S the sign of the exponent
cudaError_t launch_piece_lines(const DeviceState& d, double2* base, size_t stride, int nlines, int N, int kind, int S,
                               const double2* tw, cudaStream_t st);
cudaError_t launch_assemble_vvdz(const Geometry& g, const DeviceState& d, cudaStream_t st);
cudaError_t launch_transpose(const Geometry& g, const DeviceState& d, int to_x, int m, cudaStream_t st);
cudaError_t launch_build_products(const Geometry& g, const DeviceState& d, const PhysScalars& ps, int grp,
                                  cudaStream_t st);
cudaError_t launch_vvdz_to_field(const Geometry& g, const DeviceState& d, int m, int field, cudaStream_t st);
cudaError_t launch_buildrhs_group(const Geometry& g, const DeviceState& d, const PhysScalars& ps, double ode2,
                                  int grp, cudaStream_t st);
cudaError_t launch_damping_mask(const Geometry& g, const DeviceState& d, cudaStream_t st);
cudaError_t launch_shift_default(const Geometry& g, const DeviceState& d, const PhysScalars& ps, double dgx,
                                 double dgz, cudaStream_t st);
// the ghost rows' products must be transformed themselves (not taken as the
// shear-periodic images of the interior rows): with a spanwise shift (S2) and
// nzd = 3 nz, the retained modes iz = +-nz alias product modes -+2nz, whose
// wrap phases differ
bool edge_rows_needed(const Geometry& g, bool s2_active);
// the x stage of the lengths with a compiled plan (hst_xprod.cu), the TMA maps
// of Z and Pp that it uses, its twiddle tables (at most 2 N entries into out; their number, 0 without one)
bool x_compiled(int N, bool fp32);
cudaError_t launch_x(const Geometry& g, const DeviceState& d, const PhysScalars& ps, int want_cfl, int np,
                     cudaStream_t st);
cudaError_t make_x_maps(const Geometry& g, DeviceState& d);
// cuTensorMapEncodeTiled (null: the driver has none)
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled();
// the z transforms of the lengths with a compiled plan (hst_z.cu): the rows of
// their y tile (0: no plan), the TMA maps of the forward kernel, its twiddle
// tables (at most 2 N entries into out; their number)
int z_rows(int N, bool fp32);
cudaError_t make_z_maps(const Geometry& g, DeviceState& d);
int z_twiddles(int N, double2* out);
int z_twiddles(int N, float2* out);
cudaError_t launch_z_inv(const Geometry& g, const DeviceState& d, cudaStream_t st);
cudaError_t launch_z_fwd(const Geometry& g, const DeviceState& d, int np, cudaStream_t st);
int x_twiddles(int N, double2* out);
int x_twiddles(int N, float2* out);
// a transform length of the mixed-precision form
bool mp_length_ok(int n);
// a transform length the FFT kernels support
bool fft_length_ok(int n);

}  // namespace hst
