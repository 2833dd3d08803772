// hst_gpu_line_solve_noalloc: line_solve (src/hst_linsolve.f90:147-233) on
// fields the caller holds in its own device memory, without a context and
// without allocating anything.
//
// Who needs it: a caller that already keeps V, der and its work arrays on the
// device itself -- the reference's Fortran driver, whose OpenMP target data
// region maps those arrays (src/hst.f90:76) -- and that cannot let a library
// allocate next to them.  Creating an hst_ctx reserves the whole substep
// state (seven fields plus the transform buffers, gigabytes at production
// sizes) with cudaMalloc, which such a caller has no room for, and
// cudaMalloc/cudaFree also synchronise the device in the middle of the
// caller's queued work.  This entry point runs the same solve kernel as
// hst_gpu_line_solve and keeps its one piece of working memory, the
// slab-major copy of der that the solver groups read (D0, DY: the factored
// matrix), in a fixed array in the module's static device memory.
//
// Limits and rules of use:
//   - ny <= HST_NOALLOC_MAX_NY (2048): the scratch holds 20 * 2048 doubles
//     (320 KiB per device); larger ny is rejected with HST_EARG.
//   - The scratch is one array per device.  Calls on the same device must
//     not overlap (on different streams or host threads): a later call's
//     table write races with an earlier call's solve.  Queue them on one
//     stream, or order them with events.
//   - Nothing in the scratch has to start at zero: every call first rewrites
//     each entry its solve reads.
//   - Every call looks up the scratch's device address with
//     cudaGetSymbolAddress on the current device (a table lookup, not an
//     allocation), so that the address is always the one of the context
//     current now: after cudaDeviceReset, or under another context made
//     current on the same device, the library's device code is loaded again
//     and the array may move.  The first call in a context may be the one
//     that loads that code: make it before any stream capture begins.
//   - Neither src nor der may overlap dst: the solve reads both while it
//     writes dst (HST_EARG otherwise).
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "hst_internal.h"
#include "hst_line.cuh"

#define HST_NOALLOC_MAX_NY 2048

namespace {

// der(0:ny-1, 0:3, -2:2) reordered slab-major (the order of hst::slab_major)
__device__ __align__(256) double g_line_der[20 * HST_NOALLOC_MAX_NY];

// out[((n*5 + j)*mM + i)*P + s] = der(first(s) + i, n, j - 2); the place past the
// end of a shorter slab repeats its last row
__global__ void k_slab_major(const double* __restrict__ der, double* __restrict__ out, int ny, int P) {
  const int mM = hst::slab_rows(ny, P), e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 20 * mM * P) return;
  const hst::LineGeom G = hst::line_geom(ny, P);
  const int s = e % P;
  const int i = (e / P) % mM;
  const int nj = e / (P * mM);  // n * 5 + j
  const int n = nj / 5, j = nj - 5 * n;
  out[e] = der[(size_t)(G.first(s) + min(i, G.rows(s) - 1)) + (size_t)ny * (n + 4 * j)];
}

int fail(char* msg, int len, int rc, const char* fmt, ...) {
  if (msg && len > 0) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(msg, (size_t)len, fmt, ap);
    va_end(ap);
  }
  return rc;
}

// lanes of a solver group: the rules of a context of these sizes (HST_LINE_LANES
// overrides), so the results are identical to those of such a context.  D0 and
// DY take the substep's width, which hst_gpu_autotune may change in a context;
// the two then agree up to rounding
int lanes_of(int ny, long columns, bool d0) {
  if (const int e = hst::line_lanes_asked(ny)) return e;
  return d0 ? hst::line_lanes(ny, columns) : hst::line_lanes_shared(ny);
}

}  // namespace

extern "C" int hst_gpu_line_solve_noalloc(int nx, int ny, int nz, double alfa0, double beta0, double re, int sys,
                                          double lambda, const double* der, const double* src, double* dst,
                                          double shift_x, double shift_z, void* stream, char* msg, int msg_len) {
  if (msg && msg_len > 0) msg[0] = '\0';
  if (nx < 1 || nz < 1 || ny < 8 || ny % 2 != 0)
    return fail(msg, msg_len, HST_EARG, "need nx >= 1, nz >= 1 and ny >= 8 even (got %d, %d, %d)", nx, ny, nz);
  if (ny > HST_NOALLOC_MAX_NY)
    return fail(msg, msg_len, HST_EARG, "ny = %d exceeds the static scratch of this entry point (ny <= %d)", ny,
                HST_NOALLOC_MAX_NY);
  if (sys < hst::K_D2V || sys > hst::K_DY) return fail(msg, msg_len, HST_EARG, "unknown system kind %d", sys);
  if (!der || !src || !dst) return fail(msg, msg_len, HST_EARG, "null device pointer");
  if (((uintptr_t)src & 15) || ((uintptr_t)dst & 15) || ((uintptr_t)der & 7))
    return fail(msg, msg_len, HST_EARG, "src/dst must be 16-byte aligned, der 8-byte aligned");
  {
    // the solve reads src and der while it writes dst: neither may overlap it
    const size_t bytes = (size_t)(nx + 1) * (2 * nz + 1) * (ny + 4) * 16;
    const size_t dbytes = (size_t)20 * ny * sizeof(double);
    const uintptr_t a = (uintptr_t)src, b = (uintptr_t)dst, c = (uintptr_t)der;
    if (a < b + bytes && b < a + bytes) return fail(msg, msg_len, HST_EARG, "src and dst overlap");
    if (c < b + bytes && b < c + dbytes) return fail(msg, msg_len, HST_EARG, "der and dst overlap");
  }
  const bool d0 = sys == hst::K_D0 || sys == hst::K_DY;
  const int P = lanes_of(ny, (long)(nx + 1) * (2 * nz + 1), d0);

  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(msg, msg_len, HST_ECUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
  // the scratch's address in the context current now (see the header)
  double* scratch = nullptr;
  e = cudaGetSymbolAddress((void**)&scratch, g_line_der);
  if (e != cudaSuccess) return fail(msg, msg_len, HST_ECUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));

  hst::Geometry g = {};
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  g.nxB = nx + 1;
  g.nzT = 2 * nz + 1;
  g.rows = ny + 4;
  g.ncol = g.nxB * g.nzT;
  g.nf = (long)g.ncol * g.rows;
  g.P = g.PL = P;
  hst::PhysScalars ps = {};
  ps.alfa0 = alfa0;
  ps.beta0 = beta0;
  ps.ni = 1.0 / re;
  hst::DeviceState d = {};
  d.F[0] = reinterpret_cast<double2*>(const_cast<double*>(src));
  d.F[1] = reinterpret_cast<double2*>(dst);
  d.der = const_cast<double*>(der);
  d.derS = d.derL = scratch;
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  // der slab by slab, or for the D0 matrix the factored table alone
  const int n = 20 * hst::slab_rows(ny, P) * P, T = 256;
  if ((d0 ? hst::d0_table_doubles(ny) : (size_t)n) > sizeof g_line_der / sizeof(double))
    return fail(msg, msg_len, HST_EARG, "ny = %d exceeds the static scratch", ny);
  if (d0) {
    d.d0tab = scratch;
    e = hst::launch_d0_table(g, d, st);
  } else {
    k_slab_major<<<(n + T - 1) / T, T, 0, st>>>(der, scratch, ny, P);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = hst::launch_line_solve(g, d, ps, sys, lambda, 0, 1, shift_x, shift_z, st);
  if (e != cudaSuccess) return fail(msg, msg_len, HST_ECUDA, "launch: %s", cudaGetErrorString(e));
  return HST_OK;
}
