// The implicit half of the substep, one Fourier column a group of P lanes
// (hst_line.cuh), the line in shared memory:
//
//   k_shift       the exact_shift shear shift (shift_unweighted,
//                 src/hst_equations.f90:263-293) of rhs1, rhs2, old1, old2: D0
//                 solve with the wrap at t, node phase exp(-i gx y), D0 stencil
//                 with the ghost images at t + dt_sub
//   k_solve_half  linsolve (src/hst_equations.f90:298-326) in two passes of
//                 one line: 0 the D2V solve, V2 with its ghost rows, dv/dy (the
//                 DY solve of its D1 stencil) into the interior rows of V1,
//                 scratch until the second pass; 1 the ETA solve, u and w,
//                 V1 and V3 with their ghost rows
//   k_dy_sums     the wall-normal gradients' part of outstats
//   k_line_solve  line_solve (src/hst_linsolve.f90:147-233) of one field
//   k_d0_table    the factored D0 matrix
//
// k_shift and k_solve_half run on a persistent grid of one block an SM whose
// warps share the tables in shared memory; the factors of the D2V and ETA
// solves go to a slice of global scratch a group, rewritten column after
// column (so that it stays in L2): without them in shared memory sixteen
// warps' lines fit an SM.  The scratch is the product buffer Pp, whose contents
// are dead from the z-forward transform to the next x stage: a group's slice is
// that of its first column, at most 32 bytes a row and column, where Pp has at
// least 48 (in FP32 48 nzd for the 2 nz + 1 columns of an x mode, nzd >= 3 nz).
//
// What bounds them: the dependent operations of a row's elimination and the
// shared-memory pipe (512 rows: 69 % busy in k_shift, 54-64 % in the halves,
// DRAM a third), so a line is cut into uneven slabs without padding rows, the
// factors are kept with unit diagonals (a multiplication less a row each
// way) and the D0 stencil and node phase are taken inside the back
// substitution: 768^2 x 512 halves 3.57 -> 3.15 ms, shift 3.17 -> 2.92; 384^2 x 256
// 0.535 -> 0.358; 1536^2 x 128 (a generic form before) 11.1 -> 2.53,
// 15251 columns of 150 rows 0.399 -> 0.115.
#include <algorithm>
#include <cstdlib>

#include "hst_internal.h"
#include "hst_line.cuh"

namespace hst {

struct SolveArgs {
  Geometry g;
  PhysScalars ps;
  SubstepScalars sc;
  double2 *V1, *V2, *V3, *O1, *O2, *R1, *R2;
  const double* derS;
  const double* d0tab;
  const double* y;
  double2* fac;  // factor scratch, facn double2 a group: the product buffer Pp, which is free between the transforms
  int facn;
};

// a group's lanes within its warp
template <int P>
__device__ __forceinline__ unsigned group_mask() {
  if (P == 32) return 0xffffffffu;
  return ((1u << (P & 31)) - 1u) << ((threadIdx.x & 31) / P * P);
}

// a column's place and wave numbers
struct Column {
  double al, be, kk;
  bool c00;
  size_t cb;  // row 0 of the column
};
__device__ __forceinline__ Column column_of(const Geometry& g, const PhysScalars& ps, int cg) {
  Column c;
  const int col = g.nmem > 1 ? cg % g.ncol : cg;
  const int ix = col / g.nzT, iz = col - ix * g.nzT - g.nz;
  c.c00 = ix == 0 && iz == 0;
  c.al = ps.alfa0 * ix;
  c.be = ps.beta0 * iz;
  c.kk = c.al * c.al + c.be * c.be;
  c.cb = (size_t)cg * g.rows + 2;
  return c;
}

// The column that this group of a persistent grid takes first; the others
// follow gridDim.x blocks' groups apart.  Consecutive warps' columns go to
// consecutive blocks, so that the last round falls on all SMs alike (both
// halves of 9664 columns of 64 rows 55 -> 42 us, of 5151 of 256 rows 102 -> 83; a
// full last round, 32896 of 256 rows, 357 and 355).
template <int P>
__device__ __forceinline__ int first_column() {
  constexpr int G = 32 / P;  // groups a warp
  const int warp = threadIdx.x >> 5;
  return (warp * gridDim.x + blockIdx.x) * G + (threadIdx.x & 31) / P;
}

// (eight loads issued before the first use: the stores to shared memory may
// alias them for all the compiler knows)
template <int P>
__device__ __forceinline__ void load_line(const double2* src, cxd* buf, const LineGeom& G, int s) {
  for (int r0 = s; r0 < G.n; r0 += 8 * P) {
    cxd v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = r0 + k * P < G.n ? load_field(src + r0 + k * P) : mkc(0, 0);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (r0 + k * P < G.n) buf[G.at(r0 + k * P)] = v[k];
  }
}
template <int P>
__device__ __forceinline__ void store_line(double2* dst, const cxd* buf, const LineGeom& G, int s) {
#pragma unroll 4
  for (int r = s; r < G.n; r += P) dst[r] = buf[G.at(r)];
}
// the four ghost rows of a column (row 0 at dst) from its line (wrap_rows,
// src/hst_mpi.f90:340-355)
template <int P>
__device__ __forceinline__ void store_ghosts(double2* dst, const cxd* buf, const LineGeom& G, cxd ph, int s) {
  for (int k = s; k < 4; k += P) {
    // k = 0: row ny (row 0 ph), 1: row ny+1 (row 1 ph), 2: row -1 (row ny-1 conj), 3: row -2
    const int srow = k < 2 ? k : G.n + 1 - k, drow = k < 2 ? G.n + k : 1 - k;
    dst[drow] = cmul(buf[G.at(srow)], k < 2 ? ph : cconj(ph));
  }
}

// A table into shared memory, eight 16-byte loads of a thread in flight (n
// even, both 16-byte aligned).  Where the columns leave a block few warps, one
// load at a time took longer than the solves: both halves of 136 columns of 512
// rows 123 us, with this 39; of 256 rows 67 and 25; of 14661 columns of 512
// rows 421 and 408.
__device__ __forceinline__ void copy_table(double* dst, const double* __restrict__ src, int n) {
  const double2* const s2 = reinterpret_cast<const double2*>(src);
  double2* const d2 = reinterpret_cast<double2*>(dst);
  const int T = blockDim.x;
  for (int i0 = threadIdx.x; i0 < n / 2; i0 += 8 * T) {
    double2 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (i0 + k * T < n / 2) v[k] = __ldg(s2 + i0 + k * T);
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (i0 + k * T < n / 2) d2[i0 + k * T] = v[k];
  }
}

// The four lines of a column one after another.  What bounds it is the
// shared-memory traffic of the tables and the lines; two lines at a time,
// sharing the table loads, leave nine warps an SM and measured slower (3.42
// against 2.92 ms at 768^2 x 512).
constexpr int SHIFT_WARPS = 16;
// SH: the tables in shared memory (the most rows have no room there)
template <int P, bool SH>
__global__ void __launch_bounds__(32 * SHIFT_WARPS, 1) k_shift(SolveArgs a) {
  extern __shared__ __align__(16) double smem_d[];
  const Geometry& g = a.g;
  const SubstepScalars& sc = a.sc;
  const LineGeom G = line_geom(g.ny, P);
  const int mM = slab_rows(g.ny, P);
  const int groups = blockDim.x / P, grp = threadIdx.x / P, s = threadIdx.x % P;
  const unsigned gmask = group_mask<P>();
  const int ntab = SH ? d0_fields(mM, P) * P : 0, nder = SH ? 5 * mM * P : 0;
  double* const d0s = smem_d;
  double* const der0s = d0s + ntab;
  copy_table(d0s, a.d0tab, ntab);
  copy_table(der0s, a.derS, nder);
  if (SH) __syncthreads();
  wait_predecessor();
  cxd* const buf = reinterpret_cast<cxd*>(der0s + nder) + (size_t)grp * P * G.MS;
  cxd* const sb = buf + s * G.MS;
  const int m = G.rows(s), r0 = G.first(s);
  const SlabDerT<SH> DS = {SH ? der0s : a.derS, mM, P};
  const D0Table<P, SH> T = {(SH ? d0s : a.d0tab) + s};
  for (int cg = first_column<P>(); cg < g.ncol * g.nmem; cg += gridDim.x * groups) {
    const Column c = column_of(g, a.ps, cg);
    const cxd pt = cexpi(-(c.al * sc.sx_t + c.be * sc.sz_t)), pn = cexpi(-(c.al * sc.sx_n + c.be * sc.sz_n));
    const double gx = c.al * sc.dgx + c.be * sc.dgz;
    // the node phase of the slab's last row; on a uniform grid the rows
    // below follow by one complex product each (dy = ly / ny apart)
    const cxd etop = sc.yuni ? cexpi(-gx * a.y[r0 + m + 1]) : mkc(1.0, 0.0);
    const cxd step = sc.yuni ? cexpi(gx * (sc.ytile / 32.0)) : mkc(1.0, 0.0);
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      double2* const f = (q == 0 ? a.O1 : (q == 1 ? a.O2 : (q == 2 ? a.R1 : a.R2))) + c.cb;
      load_line<P>(f, buf, G, s);
      __syncwarp(gmask);
      cxd e = etop;
      auto node = [&](int i) -> cxd {
        if (!sc.yuni) return cexpi(-gx * a.y[r0 + i + 2]);
        const cxd v = e;
        e = cmul(e, step);
        return v;
      };
      shift_line<P>(pt, pn, T, DS, mM, m, sb, s, gmask, node);
      __syncwarp(gmask);
      store_line<P>(f, buf, G, s);
      __syncwarp(gmask);
    }
  }
}

__host__ __device__ constexpr int half_slices(int half) { return half == 0 ? 4 : 3; }
// SH: der's slices (HALF 0: all four, 1: the first three) in shared memory
template <int P, int HALF, bool SH>
__global__ void __launch_bounds__(512, 1) k_solve_half(SolveArgs a) {
  extern __shared__ __align__(16) double smem_d[];
  const Geometry& g = a.g;
  const SubstepScalars& sc = a.sc;
  const LineGeom G = line_geom(g.ny, P);
  const int mM = slab_rows(g.ny, P), ny = g.ny;
  const int groups = blockDim.x / P, grp = threadIdx.x / P, s = threadIdx.x % P;
  const unsigned gmask = group_mask<P>();
  const int nder = SH ? half_slices(HALF) * 5 * mM * P : 0;
  if (SH) {
    copy_table(smem_d, a.derS, nder);
    __syncthreads();
  }
  wait_predecessor();
  cxd* const buf = reinterpret_cast<cxd*>(smem_d + nder) + (size_t)grp * P * G.MS;
  cxd* const sb = buf + s * G.MS;
  const int m = G.rows(s);
  const SlabDerT<SH> DS = {SH ? smem_d : a.derS, mM, P};
  const int first = first_column<P>();
  double2* const fac = a.fac + (size_t)first * a.facn + s;
  for (int cg = first; cg < g.ncol * g.nmem; cg += gridDim.x * groups) {
    const Column c = column_of(g, a.ps, cg);
    const cxd pn = cexpi(-(c.al * sc.sx_n + c.be * sc.sz_n));
    double2* const v1 = a.V1 + c.cb;
    load_line<P>((HALF == 0 ? a.R2 : a.R1) + c.cb, buf, G, s);
    __syncwarp(gmask);
    if constexpr (HALF == 0) {
      line_solve<P, 3>(band_const(K_D2V, sc.lambda, a.ps.ni, c.kk), pn, DS, m, sb, fac, s, gmask);
      if (c.c00)  // the (0,0) column's v is zero
        for (int i = 0; i < m; ++i) sb[i] = mkc(0, 0);
      __syncwarp(gmask);
      double2* const v2 = a.V2 + c.cb;
      store_line<P>(v2, buf, G, s);
      store_ghosts<P>(v2, buf, G, pn, s);
      __syncwarp(gmask);
      // D1 v, then D0 (dv/dy) = D1 v (KIND_DY)
      slab_stencil<P>(1, DS, sb, m, s, pn, gmask);
      line_solve_d0<P, false>(pn, a.d0tab, mM, m, sb, s, gmask);
      __syncwarp(gmask);
      store_line<P>(v1, buf, G, s);
    } else {
      line_solve<P, 2>(band_const(K_ETA, sc.lambda, a.ps.ni, c.kk), pn, DS, m, sb, fac, s, gmask);
      __syncwarp(gmask);
      const double rkk = c.c00 ? 0.0 : 1.0 / c.kk, ar = c.al * rkk, br = c.be * rkk;
      double2* const v3 = a.V3 + c.cb;
      // dv/dy eight rows at a time, every load issued before the first use
      for (int r0 = s; r0 < ny; r0 += 8 * P) {
        cxd dvb[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) dvb[k] = r0 + k * P < ny ? load_field(v1 + r0 + k * P) : mkc(0, 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = r0 + k * P;
          if (r >= ny) break;
          const cxd eta = buf[G.at(r)], dv = dvb[k];
          // (i alfa dv - i beta eta) / k2, (i beta dv + i alfa eta) / k2
          const cxd u = c.c00 ? mkc(eta.x, 0.0) : mkc(br * eta.y - ar * dv.y, ar * dv.x - br * eta.x);
          const cxd w = c.c00 ? mkc(eta.y, 0.0) : mkc(-br * dv.y - ar * eta.y, br * dv.x + ar * eta.x);
          v1[r] = u;
          v3[r] = w;
          if (r < 2) {
            v1[ny + r] = cmul(u, pn);
            v3[ny + r] = cmul(w, pn);
          }
          if (r >= ny - 2) {
            v1[r - ny] = cmul(u, cconj(pn));
            v3[r - ny] = cmul(w, cconj(pn));
          }
        }
      }
    }
    __syncwarp(gmask);
  }
}

// The weighted sums of |du/dy|^2, |dv/dy|^2, |dw/dy|^2 over every column and
// row (outstats, src/hst_stats.f90:136-285): D1 with the stored ghost rows, the
// DY solve, nothing written but the blocks' partials [component][block]
// SH: the tables in shared memory (the most rows have no room there)
template <int P, bool SH>
__global__ void __launch_bounds__(512, 1) k_dy_sums(SolveArgs a, double sx, double sz, const double* __restrict__ dyl,
                                                    double* __restrict__ partial) {
  extern __shared__ __align__(16) double smem_d[];
  __shared__ double part[16][3];
  const Geometry& g = a.g;
  const LineGeom G = line_geom(g.ny, P);
  const int mM = slab_rows(g.ny, P), ny = g.ny;
  const int groups = blockDim.x / P, grp = threadIdx.x / P, s = threadIdx.x % P;
  const unsigned gmask = group_mask<P>();
  const int nd1 = 5 * mM * P, ntab = SH ? d0_fields(mM, P) * P : 0, nder = SH ? nd1 : 0;
  double* const d0s = smem_d;
  double* const der1s = d0s + ntab;
  copy_table(d0s, a.d0tab, ntab);
  copy_table(der1s, a.derS + nd1, nder);
  if (SH) __syncthreads();
  cxd* const buf = reinterpret_cast<cxd*>(der1s + nder) + (size_t)grp * P * G.MS;
  cxd* const sb = buf + s * G.MS;
  const int m = G.rows(s), r0 = G.first(s);
  const SlabDerT<SH> DS = {SH ? der1s : a.derS + nd1, mM, P};
  double sum[3] = {0.0, 0.0, 0.0};
  for (int cg = blockIdx.x * groups + grp; cg < g.ncol; cg += gridDim.x * groups) {
    const Column c = column_of(g, a.ps, cg);
    const cxd ph = cexpi(-(c.al * sx + c.be * sz));
    const double wc = cg < g.nzT ? 1.0 : 2.0;  // ix > 0: the conjugate half
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const double2* const f = (q == 0 ? a.V1 : (q == 1 ? a.V2 : a.V3)) + c.cb;
      load_line<P>(f, buf, G, s);
      cxd gh[4] = {mkc(0, 0), mkc(0, 0), mkc(0, 0), mkc(0, 0)};
      if (s == 0) gh[0] = f[-2], gh[1] = f[-1];
      if (s == P - 1) gh[2] = f[ny], gh[3] = f[ny + 1];
      __syncwarp(gmask);
      slab_stencil<P>(0, DS, sb, m, s, ph, gmask, gh);
      line_solve_d0<P, SH>(ph, SH ? d0s : a.d0tab, mM, m, sb, s, gmask);
      for (int i = 0; i < m; ++i) {
        const cxd d = sb[i];
        sum[q] += wc * __ldg(dyl + r0 + i) * (d.x * d.x + d.y * d.y);
      }
      __syncwarp(gmask);
    }
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 3; ++q)
    for (int o = 16; o > 0; o >>= 1) sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], o);
  if ((threadIdx.x & 31) == 0)
    for (int q = 0; q < 3; ++q) part[threadIdx.x >> 5][q] = sum[q];
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) t += part[w][threadIdx.x];
    partial[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
  }
}

// line_solve of KIND_D2V, KIND_ETA or KIND_POISSON for every Fourier column of
// one field, the factors in shared memory (a caller's own arrays come with no
// scratch)
template <int P>
__global__ void __launch_bounds__(64) k_line_solve(Geometry g, PhysScalars ps, int sys, double lambda,
                                                   const double2* __restrict__ src, double2* __restrict__ dst, double sx,
                                                   double sz, const double* __restrict__ derL) {
  extern __shared__ __align__(16) double smem_d[];
  const LineGeom G = line_geom(g.ny, P);
  const int mM = slab_rows(g.ny, P), ny = g.ny;
  const SlabDerT<false> DS = {derL, mM, P};
  const int groups = blockDim.x / P, grp = threadIdx.x / P, s = threadIdx.x % P;
  const int col = blockIdx.x * groups + grp;
  if (col >= g.ncol) return;
  const unsigned gmask = group_mask<P>();
  double2* const buf = reinterpret_cast<double2*>(smem_d) + (size_t)grp * P * (G.MS + 2 * (mM - 2));
  double2* const fac = buf + P * G.MS + s;
  const Column c = column_of(g, ps, col);
  const double2* const sc = src + c.cb;
  double2* const dc = dst + c.cb;
  load_line<P>(sc, buf, G, s);
  __syncwarp(gmask);
  const BandConst bc = band_const(sys, lambda, ps.ni, c.kk);
  const cxd ph = cexpi(-(c.al * sx + c.be * sz));
  cxd* const sb = buf + s * G.MS;
  if (sys == K_D2V)
    line_solve<P, 3>(bc, ph, DS, G.rows(s), sb, fac, s, gmask);
  else
    line_solve<P, 2>(bc, ph, DS, G.rows(s), sb, fac, s, gmask);
  __syncwarp(gmask);
  if (c.c00 && sys == K_POISSON) return;
  if (c.c00 && sys == K_D2V)
    for (int r = s; r < ny; r += P) dc[r] = mkc(0, 0);
  else
    store_line<P>(dc, buf, G, s);
}

// line_solve of KIND_D0 or (dy) KIND_DY, whose right-hand side is D1 src, from
// the factored table
template <int P>
__global__ void __launch_bounds__(128) k_line_solve_d0(Geometry g, PhysScalars ps, int dy,
                                                       const double2* __restrict__ src, double2* __restrict__ dst,
                                                       double sx, double sz, const double* __restrict__ der,
                                                       const double* __restrict__ d0tab) {
  extern __shared__ __align__(16) double smem_d[];
  const LineGeom G = line_geom(g.ny, P);
  const int groups = blockDim.x / P, grp = threadIdx.x / P, s = threadIdx.x % P;
  const int col = blockIdx.x * groups + grp;
  if (col >= g.ncol) return;
  const unsigned gmask = group_mask<P>();
  cxd* const buf = reinterpret_cast<cxd*>(smem_d) + (size_t)grp * P * G.MS;
  const Column c = column_of(g, ps, col);
  const double2* const sc = src + c.cb;
  if (dy) {
    for (int r = s; r < G.n; r += P) {
      cxd v = mkc(0, 0);
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const double d1 = derv(der, G.n, r, 1, j - 2);
        const cxd q = sc[r + j - 2];
        v = mkc(v.x + d1 * q.x, v.y + d1 * q.y);
      }
      buf[G.at(r)] = v;
    }
  } else {
    load_line<P>(sc, buf, G, s);
  }
  __syncwarp(gmask);
  line_solve_d0<P, false>(cexpi(-(c.al * sx + c.be * sz)), d0tab, slab_rows(g.ny, P), G.rows(s), buf + s * G.MS, s, gmask);
  __syncwarp(gmask);
  store_line<P>(dst + c.cb, buf, G, s);
}

// d0_factor of the group of P lanes: one warp, lanes 0..P-1, from der itself (the
// allocation-free solve factors at every call: D0 of 528 columns of 1024 rows 43.6
// us with a slab-major copy of der made first and each row loaded when its
// turn comes, 34.2 us like this)
template <int P>
__global__ void k_d0_table(const double* __restrict__ der, int ny, double* __restrict__ tab) {
  const int s = threadIdx.x;
  if (s >= P) return;
  const LineGeom G = line_geom(ny, P);
  d0_factor<P>(SlabD0{der, ny, G.first(s)}, G.rows(s), slab_rows(ny, P), s, group_mask<P>(), tab);
}

// -------------------------------------------------------------- launchers ----
// The lanes of a solver group: as many as leave at least four rows a lane,
// then half of them while a lane has fewer than twelve rows and the columns
// exceed what sixteen warps on each of the chip's 148 SMs take at once: the
// reduction across the lanes costs as much as some ten rows, a second round of
// columns half the first or more.  Measured for both solve halves, narrower and
// wider group: 64 rows of 2080 columns 17.1 us with 8 lanes, 16.6 with 16; of 5151
// 23.0 and 32.6; of 9664 35.8 with 4, 37.5 with 8; 128 rows of 3655 columns 29.4 with
// 16, 39.4 with 32; of 32896 180 with 8, 198 with 16; 256 rows of 1281 columns 30.8
// with 16, 25.8 with 32; of 32896 350 with 16, 405 with 32; 512 rows of 14661 426 with
// 16, 334 with 32.
int line_lanes(int ny, long columns) {
  int P = 2;
  for (int c = 32; c > 2; c >>= 1)
    if (ny / c >= 4) {
      P = c;
      break;
    }
  while (P > 4 && ny / P < 12 && columns > 148L * 16 * (32 / P)) P >>= 1;
  return P;
}

// With the factors in shared memory (48 bytes a row beside the line's 16)
// fewer warps fit an SM, and shorter slabs pay: as many lanes as leave eight
// rows each (256 rows of 32896 columns: three solves 418 us with 32 lanes, 486
// with 16).
int line_lanes_shared(int ny) {
  for (int mmin : {8, 4})
    for (int c = 32; c >= 2; c >>= 1)
      if (ny / c >= mmin) return c;
  return 2;
}

// A width fits where one warp's lines (32 / P of them) have room in a block's
// shared memory beside k_dy_sums' own; every width that does also has the exact
// quotients of LineGeom::at (checked for all even ny up to 2560: two lanes lose
// them from 1512 rows on, four from 2128).
static size_t line_bytes(int ny, int P) { return (size_t)P * line_geom(ny, P).MS * sizeof(double2); }
bool line_lanes_fit(int ny, int P) { return ny / P >= 4 && line_bytes(ny, P) * (32 / P) <= 226 * 1024; }

// HST_LINE_LANES, where it divides ny and fits; 0 otherwise
int line_lanes_asked(int ny) {
  const char* env = std::getenv("HST_LINE_LANES");
  const int P = env ? std::atoi(env) : 0;
  return P >= 2 && P <= 32 && (P & (P - 1)) == 0 && ny % P == 0 && line_lanes_fit(ny, P) ? P : 0;
}

size_t slab_der_doubles(int ny) { return (size_t)20 * (ny + 32); }
size_t d0_table_doubles(int ny) {
  // d0_fields(mM, P) P, mM P < ny + P
  return (size_t)9 * (ny + 32) + 32 * (31 + 8 * 4);
}
std::vector<double> slab_major(const std::vector<double>& der, int ny, int P) {
  const int mM = slab_rows(ny, P);
  const LineGeom G = line_geom(ny, P);
  std::vector<double> o((size_t)20 * mM * P, 0.0);
  std::vector<int> first(P);
  for (int s = 0; s < P; ++s) first[s] = s * G.m + std::min(s, G.rem);
  // in the table's own order (written across it, it took as long as the rest of
  // hst_gpu_set_tables); the last place of a shorter slab stays zero
  double* q = o.data();
  for (int n = 0; n < 4; ++n)
    for (int j = 0; j < 5; ++j) {
      const double* const d = der.data() + (size_t)ny * (n + 4 * j);
      for (int i = 0; i < mM; ++i)
        for (int s = 0; s < P; ++s, ++q)
          if (i < G.m || s < G.rem) *q = d[first[s] + i];
    }
  return o;
}

// double2 of factor scratch a group
static int fac_elems(int ny, int P) { return 2 * (slab_rows(ny, P) - 2) * P; }

// warps a block (one block an SM): as many as `most` whose groups' lines fit
// beside `tabs` bytes of tables, and no more than spread the columns over the
// SMs; 0 when not even one fits
static int solve_warps(const Geometry& g, int nsm, size_t tabs, int most = 16) {
  const size_t warp = line_bytes(g.ny, g.P) * (32 / g.P);
  if (tabs + warp > 227 * 1024) return 0;
  const long groups = ((long)g.ncol * g.nmem + nsm - 1) / nsm;  // columns an SM
  const long want = (groups * g.P + 31) / 32;
  return (int)std::min<long>({most, want, (long)((227 * 1024 - tabs) / warp)});
}

// As many of W warps as give every round that W warps take the same columns: a
// nearly empty last round costs as much as half a full one, and holds the whole
// SM against other streams' kernels.  Both halves of 9664 columns of 512 rows 272
// -> 235 us, the shift 259 -> 223; of 20301 of 64 rows 79 -> 73; three fields of nx
// 27, ny 92, nz 431 in turn, exact shift, 10.5 -> 9.4 ms a pass.
static int even_warps(const Geometry& g, int nsm, int W) {
  const int cols = (g.ncol * g.nmem + nsm - 1) / nsm, round = W * 32 / g.P, rounds = (cols + round - 1) / round;
  return ((cols + rounds - 1) / rounds * g.P + 31) / 32;
}

static SolveArgs solve_args(const Geometry& g, const DeviceState& d, const PhysScalars& ps, const SubstepScalars& sc) {
  return {g,      ps,     sc,     d.F[0], d.F[1],  d.F[2], d.F[3],
          d.F[4], d.F[5], d.F[6], d.derS, d.d0tab, d.y,    d.Pp, fac_elems(g.ny, g.P)};
}
static int sm_count(const DeviceState& d) { return d.nsm > 0 ? d.nsm : 148; }

template <int P>
static cudaError_t launch_shift_t(const SolveArgs& a, const DeviceState& d, cudaStream_t st) {
  const Geometry& g = a.g;
  const int mM = slab_rows(g.ny, P), nsm = sm_count(d);
  size_t tabs = ((size_t)d0_fields(mM, P) * P + (size_t)5 * mM * P) * sizeof(double);
  int W = solve_warps(g, nsm, tabs, SHIFT_WARPS);
  const bool sh = W >= 4 || W == solve_warps(g, nsm, 0, SHIFT_WARPS);
  if (!sh) {  // the tables through L1
    tabs = 0;
    W = solve_warps(g, nsm, 0, SHIFT_WARPS);
  }
  if (W < 1) return cudaErrorInvalidValue;
  W = even_warps(g, nsm, W);
  const int groups = W * 32 / P;
  const int nb = std::min(nsm, (g.ncol * g.nmem + groups - 1) / groups);
  auto k = sh ? k_shift<P, true> : k_shift<P, false>;
  smem_limit(d, k, 227 * 1024);
  return launch_after(k, dim3(nb), 32 * W, tabs + W * line_bytes(g.ny, P) * (32 / P), st, a);
}

template <int P>
static cudaError_t launch_dy_sums_t(const SolveArgs& a, const DeviceState& d, double sx, double sz, double* partial,
                                    int* blocks, cudaStream_t st) {
  const Geometry& g = a.g;
  const int mM = slab_rows(g.ny, P), nsm = sm_count(d);
  size_t tabs = ((size_t)d0_fields(mM, P) * P + (size_t)5 * mM * P) * sizeof(double);
  int W = solve_warps(g, nsm, tabs + 1024);
  const bool sh = W >= 4 || W == solve_warps(g, nsm, 1024);
  if (!sh) {
    tabs = 0;
    W = solve_warps(g, nsm, 1024);
  }
  if (W < 1) return cudaErrorInvalidValue;
  const int groups = W * 32 / P;
  *blocks = std::min(nsm, (g.ncol + groups - 1) / groups);
  auto k = sh ? k_dy_sums<P, true> : k_dy_sums<P, false>;
  smem_limit(d, k, 226 * 1024);
  k<<<*blocks, 32 * W, tabs + W * line_bytes(g.ny, P) * (32 / P), st>>>(a, sx, sz, d.dyl, partial);
  return cudaGetLastError();
}

template <int P, int HALF>
static cudaError_t launch_half_t(const SolveArgs& a, const DeviceState& d, cudaStream_t st) {
  const Geometry& g = a.g;
  const int mM = slab_rows(g.ny, P), nsm = sm_count(d);
  size_t tabs = (size_t)half_slices(HALF) * 5 * mM * P * sizeof(double);
  int W = solve_warps(g, nsm, tabs);
  const bool sh = W >= 4 || W == solve_warps(g, nsm, 0);
  if (!sh) {  // der through L1
    tabs = 0;
    W = solve_warps(g, nsm, 0);
  }
  if (W < 1) return cudaErrorInvalidValue;
  W = even_warps(g, nsm, W);
  const int groups = W * 32 / P;
  const int nb = std::min(nsm, (g.ncol * g.nmem + groups - 1) / groups);
  const size_t smem = tabs + W * line_bytes(g.ny, P) * (32 / P);
  auto k = sh ? k_solve_half<P, HALF, true> : k_solve_half<P, HALF, false>;
  smem_limit(d, k, 227 * 1024);
  return launch_after(k, dim3(nb), 32 * W, smem, st, a);
}

template <int P>
static cudaError_t launch_line_solve_t(const Geometry& g, const DeviceState& d, const PhysScalars& ps, int sys,
                                       double lambda, int src, int dst, double sx, double sz, cudaStream_t st) {
  if (sys == K_D0 || sys == K_DY) {
    const size_t line = line_bytes(g.ny, P);
    int groups = 128 / P;
    while (groups > 1 && line * groups > 56 * 1024) groups >>= 1;
    smem_limit(d, k_line_solve_d0<P>, 200 * 1024);
    k_line_solve_d0<P><<<(g.ncol + groups - 1) / groups, groups * P, line * groups, st>>>(
        g, ps, sys == K_DY, d.F[src], d.F[dst], sx, sz, d.der, d.d0tab);
    return cudaGetLastError();
  }
  const size_t per = line_bytes(g.ny, P) + fac_elems(g.ny, P) * sizeof(double2);
  int groups = 32 / P;
  while (groups > 1 && per * groups > 200 * 1024) groups >>= 1;
  if (per * groups > 200 * 1024) return cudaErrorInvalidValue;
  smem_limit(d, k_line_solve<P>, 200 * 1024);
  k_line_solve<P><<<(g.ncol + groups - 1) / groups, groups * P, per * groups, st>>>(g, ps, sys, lambda, d.F[src],
                                                                                   d.F[dst], sx, sz, d.derL);
  return cudaGetLastError();
}

#define HST_LANES(P_, CALL)                \
  switch (P_) {                            \
    case 2: return CALL(2);                \
    case 4: return CALL(4);                \
    case 8: return CALL(8);                \
    case 16: return CALL(16);              \
    case 32: return CALL(32);              \
  }                                        \
  return cudaErrorInvalidValue

cudaError_t launch_shift(const Geometry& g, const DeviceState& d, const PhysScalars& ps, const SubstepScalars& sc,
                         cudaStream_t st) {
  const SolveArgs a = solve_args(g, d, ps, sc);
#define HST_CALL(P) launch_shift_t<P>(a, d, st)
  HST_LANES(g.P, HST_CALL);
#undef HST_CALL
}

cudaError_t launch_dy_sums(const Geometry& g, const DeviceState& d, const PhysScalars& ps, double sx, double sz,
                           double* partial, int* blocks, cudaStream_t st) {
  const SolveArgs a = solve_args(g, d, ps, SubstepScalars{});
#define HST_CALL(P) launch_dy_sums_t<P>(a, d, sx, sz, partial, blocks, st)
  HST_LANES(g.P, HST_CALL);
#undef HST_CALL
}

cudaError_t launch_solve_half(const Geometry& g, const DeviceState& d, const PhysScalars& ps, const SubstepScalars& sc,
                              int half, cudaStream_t st) {
  const SolveArgs a = solve_args(g, d, ps, sc);
#define HST_CALL(P) (half == 0 ? launch_half_t<P, 0>(a, d, st) : launch_half_t<P, 1>(a, d, st))
  HST_LANES(g.P, HST_CALL);
#undef HST_CALL
}

cudaError_t launch_line_solve(const Geometry& g, const DeviceState& d, const PhysScalars& ps, int sys, double lambda,
                              int src, int dst, double sx, double sz, cudaStream_t st) {
#define HST_CALL(P) launch_line_solve_t<P>(g, d, ps, sys, lambda, src, dst, sx, sz, st)
  HST_LANES(sys == K_D0 || sys == K_DY ? g.P : g.PL, HST_CALL);
#undef HST_CALL
}

template <int P>
static cudaError_t launch_d0_t(const Geometry& g, const DeviceState& d, cudaStream_t st) {
  k_d0_table<P><<<1, 32, 0, st>>>(d.der, g.ny, d.d0tab);
  return cudaGetLastError();
}
cudaError_t launch_d0_table(const Geometry& g, const DeviceState& d, cudaStream_t st) {
#define HST_CALL(P) launch_d0_t<P>(g, d, st)
  HST_LANES(g.P, HST_CALL);
#undef HST_CALL
}

}  // namespace hst
