// The row-by-row right-hand sides, for the per-piece prepare and (with
// HST_RHS_TILED=0) in place of the streamed form of hst_rhs.cu, and the ghost
// rows of a field.
//
// Only the ny interior rows are transformed.  The products in the four
// ghost rows, which the reference transforms as well
// (src/hst_transforms.f90:3-6), are the shear-periodic images of the
// interior ones: the 3/2 rule makes the retained product modes exact, so the
// image of row k is row k times the wrap phase, which the right-hand-side
// stage applies when it reads them.
#include "hst_dev.cuh"
#include "hst_internal.h"
#include "hst_rhs.cuh"

namespace hst {

struct ColumnArgs {
  Geometry g;
  PhysScalars ps;
  SubstepScalars sc;
  double2 *V1, *V2, *V3, *O1, *O2, *R1, *R2;
  const double2* Q;
  const double2* Qg;  // the ghost rows' product spectra [6][ncol][4] (null: their wrap images)
  const double* der;
  const double* y;
  const double* gdamp;
};

// a product spectrum at row q of its column, with the ghost images (or,
// with Qgc, the ghost rows' own transforms: rows -2, -1, ny, ny+1 there)
__device__ __forceinline__ cxd q_at(const double2* __restrict__ Qc, const double2* __restrict__ Qgc, int q, int ny,
                                    cxd ph) {
  if (q < 0) return Qgc ? Qgc[q + 2] : cmul(Qc[q + ny], cconj(ph));
  if (q >= ny) return Qgc ? Qgc[q - ny + 2] : cmul(Qc[q - ny], ph);
  return Qc[q];
}

// buildrhs_prepare (src/hst_equations.f90:92-141) and buildrhs (:151-213), one
// warp a column, lanes over rows, into RHS1/2 and OLD1/2
template <bool EXACT, bool NONLIN>
__global__ void __launch_bounds__(128) k_rhs_rows(ColumnArgs a) {
  const Geometry& g = a.g;
  const int cg = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (cg >= g.ncol * g.nmem) return;
  const int mem = cg / g.ncol, col = cg - mem * g.ncol, ny = g.ny;
  const SubstepScalars sc = a.sc;
  const size_t cb = (size_t)cg * g.rows + 2;  // row 0 of the column
  const double2* __restrict__ V1c = a.V1 + cb;
  const double2* __restrict__ V2c = a.V2 + cb;
  const double2* __restrict__ V3c = a.V3 + cb;
  const ColConst cc = col_const(col, g, a.ps, sc, a.gdamp);
  const double2* Qc = a.Q + ((size_t)mem * 6 * g.ncol + col) * ny;
  const size_t qs = (size_t)g.ncol * ny;
#pragma unroll 1
  for (int r = lane; r < ny; r += 32) {
    auto tv = [&](int c, int j) -> cxd { return (c == 0 ? V1c : (c == 1 ? V2c : V3c))[r + j - 2]; };
    // the components uu - vv, ww - vv, uv, vw, uw in the places of uu, ww, uv, vw,
    // uw, with vv = 0: the right-hand sides depend on the differences alone
    auto tq = [&](int pr, int j) -> cxd {
      if (pr == 1) return mkc(0, 0);
      const int p = pr > 0 ? pr - 1 : 0;
      return q_at(Qc + p * qs, a.Qg ? a.Qg + (((size_t)mem * 6 + p) * g.ncol + col) * 4 : nullptr, r + j - 2, ny, cc.ph_t);
    };
    const size_t ro = cb + r;
    cxd r1, r2, o1, o2;
    const double yr = a.y[r + 2];
    auto fsh = [&]() { return cexpi(-(cc.al * sc.dgx + cc.be * sc.dgz) * yr); };
    rhs_point<NONLIN, EXACT>(cc, sc, DerFull{a.der, ny}, ny, r, fsh, tv, tq, a.O1[ro], a.O2[ro], r1, r2, o1, o2);
    a.O1[ro] = o1;
    a.O2[ro] = o2;
    a.R1[ro] = r1;
    a.R2[ro] = r2;
  }
}

cudaError_t launch_rhs_rows(const Geometry& g, const DeviceState& d, const PhysScalars& ph, const SubstepScalars& sc,
                            int exact, int nonlin, cudaStream_t st) {
  // FP64 product spectra only (the linear right-hand sides read none)
  if (g.mp && nonlin) return cudaErrorInvalidValue;
  const ColumnArgs a = {g,      ph,     sc,     d.F[0], d.F[1], d.F[2], d.F[3], d.F[4],
                        d.F[5], d.F[6], d.Q,    d.Qg,   d.der,  d.y,    d.gdamp};
  const int blocks = (g.ncol * g.nmem + 3) / 4;
  if (exact) {
    if (nonlin) k_rhs_rows<true, true><<<blocks, 128, 0, st>>>(a);
    else k_rhs_rows<true, false><<<blocks, 128, 0, st>>>(a);
  } else {
    if (nonlin) k_rhs_rows<false, true><<<blocks, 128, 0, st>>>(a);
    else k_rhs_rows<false, false><<<blocks, 128, 0, st>>>(a);
  }
  return cudaGetLastError();
}

// -------------------------------------------------------- k_fill_ghosts ----
__global__ void k_fill_ghosts(Geometry g, PhysScalars ps, double2* __restrict__ f, double sx, double sz) {
  int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= g.ncol) return;
  const int ix = col / g.nzT, iz = col - ix * g.nzT - g.nz;
  const cxd ph = cexpi(-(ps.alfa0 * ix * sx + ps.beta0 * iz * sz));
  double2* c = f + (size_t)col * g.rows + 2;
  const int ny = g.ny;
  c[ny] = cmul(c[0], ph);
  c[ny + 1] = cmul(c[1], ph);
  c[-1] = cmul(c[ny - 1], cconj(ph));
  c[-2] = cmul(c[ny - 2], cconj(ph));
}

cudaError_t launch_fill_ghosts(const Geometry& g, const DeviceState& d, const PhysScalars& ph, int field, double sx,
                               double sz, cudaStream_t st) {
  int T = 128;
  k_fill_ghosts<<<(g.ncol + T - 1) / T, T, 0, st>>>(g, ph, d.F[field], sx, sz);
  return cudaGetLastError();
}

}  // namespace hst
