// The transforms of the hst substep for the lengths without a plan of their
// own in hst_xprod.cu and hst_z.cu (FP64), the launches of the three transform stages, and
// the line transforms of the per-piece path:
//
//   zinv    V (u, v, w) -> zero-padded z-inverse transform (Z)
//   xprod   Z -> x-inverse (c2r) of u, v, w; the six products times
//           1/(2 nxd nzd); the CFL maximum; x-forward (r2c) of the products
//           truncated to the nx+1 retained modes (Pp)
//   zfwd    Pp -> z-forward transform truncated to the 2nz+1 modes (Q)
//
// (hst_z.cu and hst_xprod.cu for the compiled lengths.)  Together they are
// transform_to_physical + build_products (both groups) +
// products_to_spectral + compute_cfl of the reference
// (src/hst_transforms.f90:33-179, src/hst_fft.f90:181-237), with the local
// transposes (src/hst_mpi.f90:615-669) absorbed into the index maps.  Only
// the ny interior rows are transformed (see hst_rhs.cu for the ghost-row
// products).  Z and Pp are stored [component][y tile][kz][ix][Ty]: the z
// lines of one x mode and one y tile then span a few huge pages instead of
// one page per kz.
#include <cmath>

#include "hst_dev.cuh"
#include "hst_fft.cuh"
#include "hst_internal.h"

namespace hst {

bool fft_length_ok(int n) { return plan_ok(n); }

// --------------------------------------------------------------- k_zinv ----
// assemble_vvdz + IFT (src/hst_transforms.f90:33-54, src/hst_fft.f90:195-207):
// line yi of the block is row y0 + yi of one x mode of one component; the
// z modes -nz..nz sit at padded index iz (iz >= 0) or nzd + iz.
struct ZinvSrc {
  typedef double2 C;
  const double2* __restrict__ col;  // V + (ix nzT) rows + 2 + y0: row y0 of iz = -nz
  int rows, nz, NZ;
  int gap;  // the edge view: rows -2, -1 at 0, 1 and ny, ny+1 at gap + 2, gap + 3
  __device__ __forceinline__ C operator()(int yi, int kz) const {
    int iz;
    if (kz <= nz) iz = kz;
    else if (kz >= NZ - nz) iz = kz - NZ;
    else return C{0, 0};
    return col[(size_t)(iz + nz) * rows + yi + (yi >= 2 ? gap : 0)];
  }
};
struct TileDst {
  typedef double2 C;  // one (component, y tile, x mode) z-line set of Z / Pp
  C* __restrict__ base;
  size_t zstride;
  __device__ __forceinline__ void operator()(int yi, int kz, C v) const { base[(size_t)kz * zstride + yi] = v; }
};
struct TileSrc {
  typedef double2 C;
  const C* __restrict__ base;
  size_t zstride;
  __device__ __forceinline__ C operator()(int yi, int kz) const { return base[(size_t)kz * zstride + yi]; }
};

template <int NT, int PPT>
__global__ void __launch_bounds__(256)
    k_zinv(Geometry g, const double2* __restrict__ V0, const double2* __restrict__ V1, const double2* __restrict__ V2,
           double2* __restrict__ Z, const double2* __restrict__ twz) {
  extern __shared__ double2 sh[];
  const int ix = blockIdx.x, yt = blockIdx.y, c = blockIdx.z % 3, mem = blockIdx.z / 3;
  const int Ty = g.Ty, NZ = NT ? NT : g.nzd;
  const double2* V = (c == 0 ? V0 : (c == 1 ? V1 : V2)) + (size_t)mem * g.nf;
  const ZinvSrc src = {V + (size_t)ix * g.nzT * g.rows + (g.edge_gap ? 0 : 2) + yt * Ty, g.rows, g.nz, NZ, g.edge_gap};
  const TileDst dst = {Z + ((((size_t)mem * 3 + c) * g.nyT + yt) * NZ) * g.nxB * Ty + (size_t)ix * Ty, (size_t)g.nxB * Ty};
  fft_global<NT, +1, PPT, false, false>(NZ, Ty, twz, sh, src, dst);
}

// --------------------------------------------------------------- k_zfwd ----
// transpose_xTOz + FFT (src/hst_transforms.f90:135-139, src/hst_fft.f90:181-193)
// keeping the 2nz+1 retained modes, stored without ghost rows.
struct ZfwdDst {
  typedef double2 C;
  C* __restrict__ base;  // Q + (p ncol + ix nzT) ny + y0
  int ny, nz, NZ;
  __device__ __forceinline__ void operator()(int yi, int k, C v) const {
    int iz;
    if (k <= nz) iz = k;
    else if (k >= NZ - nz) iz = k - NZ;
    else return;
    base[(size_t)(iz + nz) * ny + yi] = v;
  }
};

template <int NT, int PPT>
__global__ void __launch_bounds__(256)
    k_zfwd(Geometry g, int np, const double2* __restrict__ Pp, double2* __restrict__ Q,
           const double2* __restrict__ twz) {
  extern __shared__ double2 sh[];
  const int yt = blockIdx.x, ix = blockIdx.y, pm = blockIdx.z / np * 6 + blockIdx.z % np;
  const int Ty = g.Ty, NZ = NT ? NT : g.nzd;
  const TileSrc src = {Pp + (((size_t)pm * g.nyT + yt) * NZ) * g.nxB * Ty + (size_t)ix * Ty, (size_t)g.nxB * Ty};
  const ZfwdDst dst = {Q + ((size_t)pm * g.ncol + (size_t)ix * g.nzT) * g.ny + yt * Ty, g.ny, g.nz, NZ};
  fft_global<NT, -1, PPT, false, false>(NZ, Ty, twz, sh, src, dst);
}

// -------------------------------------------------------------- k_xprod ----
// to_x_points (zero padding + RFT), build_products for both groups,
// compute_cfl and HFT of the products (src/hst_transforms.f90:85-133,
// 163-179; src/hst_fft.f90:211-237) for one pair of rows at one z point.
// Two real lines ride on one complex line: u + i v of each row and w0 + i w1
// of the pair on the way in; (uu, vv), (ww, uv), (vw, uw) of each row on
// the way out, separated by Hermitian symmetry.  The c2r reads only the
// real part of the kx = 0 mode, as FFTW's and cuFFT's c2r do.
template <typename C>
struct XinvSrc {
  const C* __restrict__ zb;  // Z tile of component 0 at (y tile, kz), + row offset in the tile
  size_t cs;                 // component stride of Z
  int Ty, nx, NX;
  __device__ __forceinline__ C operator()(int l, int k) const {
    const int m = k <= nx ? k : (k >= NX - nx ? NX - k : -1);
    if (m < 0) return C{0, 0};
    const C* p = zb + (size_t)m * Ty;
    C a, b;
    if (l == 0) {  // u(y0) + i v(y0)
      a = p[0];
      b = p[cs];
    } else if (l == 1) {  // u(y1) + i v(y1)
      a = p[1];
      b = p[cs + 1];
    } else {  // w(y0) + i w(y1)
      a = p[2 * cs];
      b = p[2 * cs + 1];
    }
    if (k == 0) return C{a.x, b.x};
    if (k <= nx) return C{a.x - b.y, a.y + b.x};
    return C{a.x + b.y, b.x - a.y};  // conj(a) + i conj(b)
  }
};
// the products of row yy, pair pl (0: uu, vv; 1: ww, uv; 2: vw, uw; of five
// products 0: uu - vv, ww - vv; 1: uv, vw; 2: uw, 0) at x
template <typename LT, typename C>
struct ProdSrc {
  typedef typename RealOf<C>::T T;
  LT L;
  T f;
  bool five;
  __device__ __forceinline__ C operator()(int l, int x) const {
    const int yy = l >= 3 ? 1 : 0, pl = l - 3 * yy;
    const C a = L(yy, x), b = L(2, x);
    const T u = a.x, v = a.y, w = yy ? b.y : b.x;
    if (five) {
      if (pl == 0) return C{(u * u - v * v) * f, (w * w - v * v) * f};
      if (pl == 1) return C{u * v * f, v * w * f};
      return C{u * w * f, T(0)};
    }
    if (pl == 0) return C{u * u * f, v * v * f};
    if (pl == 1) return C{w * w * f, u * v * f};
    return C{v * w * f, u * w * f};
  }
};

// The x stage of the lengths without a plan in hst_xprod.cu, FP64 (PPT points a
// thread; NT: the length, 0: any)
template <int NT, int PPT>
__global__ void __launch_bounds__(320)
    k_xprod(Geometry g, int np, const double2* __restrict__ Z, double2* __restrict__ Pp, const double2* __restrict__ twx,
            const double* __restrict__ dyl, PhysScalars ps, int want_cfl, unsigned long long* __restrict__ cflmax) {
  typedef double2 C;
  extern __shared__ double2 sh[];
  typedef ShLinesT<C> LT;
  const int NX = NT ? NT : 2 * g.nxd, nx = g.nx, nxB = g.nxB, NZ = g.nzd, Ty = g.Ty;
  const int nyT = g.nyT;
  const int y0 = 2 * blockIdx.x, kz = blockIdx.y % g.nzd, mem = blockIdx.y / g.nzd;
  Z += (size_t)mem * 3 * g.nzd * nyT * Ty * g.nxB;
  Pp += (size_t)mem * 6 * g.nzd * nyT * Ty * g.nxB;
  const int yt = y0 / Ty, yi0 = y0 - yt * Ty;
  const size_t cs = (size_t)NZ * nyT * nxB * Ty;
  const size_t tile = ((size_t)yt * NZ + kz) * nxB * Ty;
  const LT L = {sh, NX + 1};
  // u + i v of both rows and w0 + i w1 on the physical x grid
  const XinvSrc<C> xs = {Z + tile + yi0, cs, Ty, nx, NX};
  fft_global<NT, +1, PPT, false, true>(NX, 3, twx, sh, xs, L);
  __syncthreads();
  if (want_cfl) {
    double cm = 0.0;
    const double rdy0 = 1.0 / dyl[y0], rdy1 = 1.0 / dyl[y0 + 1];
    for (int x = threadIdx.x; x < NX; x += blockDim.x) {
      const C a0 = L(0, x), a1 = L(1, x), b = L(2, x);
      double c0 = fabs(a0.x) * ps.rdx + fabs(a0.y) * rdy0 + fabs(b.x) * ps.rdz;
      double c1 = fabs(a1.x) * ps.rdx + fabs(a1.y) * rdy1 + fabs(b.y) * ps.rdz;
      cm = nan_max(cm, nan_max(c0, c1));
    }
    for (int o = 16; o > 0; o >>= 1) cm = nan_max(cm, __shfl_xor_sync(0xffffffffu, cm, o));
    // a NaN keeps its bits: as an unsigned word it exceeds every finite
    // non-negative double and infinity, so it wins the maximum and the host
    // sees a non-finite CFL number
    if ((threadIdx.x & 31) == 0) atomicMax(cflmax, (unsigned long long)__double_as_longlong(cm));
  }
  // the six product lines, transformed forward in place
  const ProdSrc<LT, C> ps6 = {L, ps.factor, np == 5};
  fft_global<NT, -1, PPT, true, true>(NX, 6, twx, sh, ps6, L);
  __syncthreads();
  // separate the two real transforms of each line, keep kx = 0..nx
  for (int e = threadIdx.x; e < nxB * 3; e += blockDim.x) {
    const int pl = e / nxB, ix = e - pl * nxB;
#pragma unroll
    for (int yy = 0; yy < 2; ++yy) {
      const int ln = pl + 3 * yy;
      const C Zk = L(ln, ix), Zm = L(ln, ix == 0 ? 0 : NX - ix);
      const size_t o = tile + (size_t)ix * Ty + yi0 + yy;
      Pp[(size_t)(2 * pl) * cs + o] = C{0.5 * (Zk.x + Zm.x), 0.5 * (Zk.y - Zm.y)};
      Pp[(size_t)(2 * pl + 1) * cs + o] = C{0.5 * (Zk.y + Zm.y), 0.5 * (Zm.x - Zk.x)};
    }
  }
}

// --------------------------------------- the reference-layout transforms ----
// FFT, IFT, RFT and HFT (src/hst_fft.f90:181-237) on the buffers of the
// per-piece path, which hold the reference's layouts: VVdz(nzd, nx+1,
// -2:ny+1, 3) and VVdx / VVdp(nxd+1, nzd, -2:ny+1, 3), the latter also seen as
// 2(nxd+1) reals a line (rVVdx, products).  A block loads LPB whole lines
// into shared memory, transforms them there with the runtime plan and
// writes them back over the same bytes (every line is read before any is
// written, so the in-place real <-> complex layouts are safe).  These serve
// the drop-in per-piece interface; the fused substep does not use them.
static int fft_threads(int points, int ppt);
struct PieceLines {
  double2* base;  // line l starts at base + l * stride (complex elements)
  size_t stride;
  int kind;       // 0: complex z line; 1: c2r x line (Hermitian, nxd+1 modes in); 2: r2c x line (reals in)
  int N;          // transform length
};
__device__ __forceinline__ double2 piece_load(const PieceLines& P, int l, int k) {
  const double2* b = P.base + (size_t)l * P.stride;
  if (P.kind == 0) return b[k];
  if (P.kind == 1) {
    const int h = P.N / 2;
    if (k <= h) return b[k];
    const double2 c = b[P.N - k];
    return make_double2(c.x, -c.y);
  }
  const double* r = reinterpret_cast<const double*>(b);
  return make_double2(r[k], 0.0);
}
template <int S>
__global__ void __launch_bounds__(256) k_piece_lines(PieceLines P, int nlines, int lpb, const double2* __restrict__ tw) {
  extern __shared__ double2 sh_d[];
  const int N = P.N, LS = N + 1;
  const int l0 = blockIdx.x * lpb;
  const int nl = min(lpb, nlines - l0);
  for (int e = threadIdx.x; e < lpb * N; e += blockDim.x) {
    const int l = e / N, k = e - l * N;
    sh_d[l * LS + k] = l < nl ? piece_load(P, l0 + l, k) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const ShLinesT<double2> L = {sh_d, LS};
  fft_global<0, S, 16, true, true>(N, lpb, tw, sh_d, L, L);
  __syncthreads();
  if (P.kind == 1) {  // real parts: 2(nxd+1) reals a line, the two past N zero
    for (int e = threadIdx.x; e < nl * (N + 2); e += blockDim.x) {
      const int l = e / (N + 2), k = e - l * (N + 2);
      double* r = reinterpret_cast<double*>(P.base + (size_t)(l0 + l) * P.stride);
      r[k] = k < N ? sh_d[l * LS + k].x : 0.0;
    }
  } else {
    const int nout = P.kind == 0 ? N : N / 2 + 1;
    for (int e = threadIdx.x; e < nl * nout; e += blockDim.x) {
      const int l = e / nout, k = e - l * nout;
      P.base[(size_t)(l0 + l) * P.stride + k] = sh_d[l * LS + k];
    }
  }
}

// kind 0/1/2 as PieceLines; S the transform's sign (+1 backward)
cudaError_t launch_piece_lines(const DeviceState& d, double2* base, size_t stride, int nlines, int N, int kind, int S,
                               const double2* tw, cudaStream_t st) {
  if (!plan_ok(N) || nlines <= 0) return cudaErrorInvalidValue;
  const PieceLines P = {base, stride, kind, N};
  const int lpb = N >= 1536 ? 1 : (N >= 768 ? 2 : 4);
  const int threads = fft_threads(lpb * N, 16);
  if (threads > 256) return cudaErrorInvalidValue;
  const size_t smem = (size_t)lpb * (N + 1) * sizeof(double2);
  const int blocks = (nlines + lpb - 1) / lpb;
  if (S > 0) {
    smem_limit(d, k_piece_lines<+1>, 220 * 1024);
    k_piece_lines<+1><<<blocks, threads, smem, st>>>(P, nlines, lpb, tw);
  } else {
    smem_limit(d, k_piece_lines<-1>, 220 * 1024);
    k_piece_lines<-1><<<blocks, threads, smem, st>>>(P, nlines, lpb, tw);
  }
  return cudaGetLastError();
}

bool edge_rows_needed(const Geometry& g, bool s2_active) { return s2_active && g.nzd <= 3 * g.nz; }

// The view of the four ghost rows: the same transforms with ny = 4 and one y
// tile on the edge buffers
static void edge_view(const Geometry& g, const DeviceState& d, Geometry& ge, DeviceState& de) {
  ge = g;
  ge.ny = 4;
  ge.Ty = g.EY;
  ge.nyT = 1;
  ge.edge_gap = g.ny;
  de = d;
  de.Z = d.Zg;
  de.Pp = d.Ppg;
  de.Q = d.Qg;
  de.tmZ = d.tmZg;
  de.tmPp = d.tmPpg;
  de.tmPp2 = d.tmPpg2;
  de.tmPz = d.tmPgz;
}

// -------------------------------------------------------------- launchers ----
static int fft_threads(int points, int ppt) {
  int t = (points + ppt - 1) / ppt;
  t = (t + 31) / 32 * 32;
  return t < 64 ? 64 : t;
}

template <typename K>
static void big_smem(const DeviceState& d, K k) {
  smem_limit(d, k, 220 * 1024);
}

// The lengths known to the compiler, then the runtime plan with 16 or 32 points
// a thread.  Computed at run time, the indices of a short line's few butterflies
// cost as much as the butterflies: x at 48 points (nx 15, ny 64, nz 40) 50.3 us a
// substep, at 24 (nx 7, ny 128, nz 128) 285, known to the compiler 35.9 and 223;
// z inverse at 24 (nx 127, ny 128, nz 8) 37.5 and 31.2.
#define HST_SHORT_Z(n, pts, F) \
  switch (n) {                 \
    case 12: F(12, 16); break; \
    case 24: F(24, 16); break; \
    default:                   \
      if ((pts) <= 16 * 256) { \
        F(0, 16);              \
      } else {                 \
        F(0, 32);              \
      }                        \
  }
#define HST_SHORT_X(n, pts, F) \
  if ((n) == 48) {             \
    F(48, 16);                 \
  } else if ((n) == 64) {      \
    F(64, 16);                 \
  } else                       \
    HST_SHORT_Z(n, pts, F)

bool mp_length_ok(int n) { return x_compiled(n, true) && z_rows(n, true) > 0; }

static cudaError_t launch_zinv_main(const Geometry& g, const DeviceState& d, cudaStream_t st) {
  if (z_rows(g.nzd, g.mp != 0)) return launch_z_inv(g, d, st);
  const int pts = g.nzd * g.Ty;
  const dim3 grid(g.nxB, g.nyT, 3 * g.nmem);
  const size_t smem = (size_t)g.Ty * (g.nzd + 1) * sizeof(double2);
#define HST_ZINV(NT, PPT)        \
  big_smem(d, k_zinv<NT, PPT>); \
  k_zinv<NT, PPT><<<grid, fft_threads(pts, PPT), smem, st>>>(g, d.F[0], d.F[1], d.F[2], d.Z, d.twz)
  HST_SHORT_Z(g.nzd, pts, HST_ZINV)
#undef HST_ZINV
  return cudaGetLastError();
}

static cudaError_t launch_zfwd_main(const Geometry& g, const DeviceState& d, int np, cudaStream_t st) {
  if (z_rows(g.nzd, g.mp != 0)) return launch_z_fwd(g, d, np, st);
  const int pts = g.nzd * g.Ty;
  const dim3 grid(g.nyT, g.nxB, np * g.nmem);
  const size_t smem = (size_t)g.Ty * (g.nzd + 1) * sizeof(double2);
#define HST_ZFWD(NT, PPT)        \
  big_smem(d, k_zfwd<NT, PPT>); \
  k_zfwd<NT, PPT><<<grid, fft_threads(pts, PPT), smem, st>>>(g, np, d.Pp, d.Q, d.twz)
  HST_SHORT_Z(g.nzd, pts, HST_ZFWD)
#undef HST_ZFWD
  return cudaGetLastError();
}

static cudaError_t launch_xprod_main(const Geometry& g, const DeviceState& d, const PhysScalars& ph, int want_cfl, int np,
                                     cudaStream_t st) {
  const int NX = 2 * g.nxd;
  if (x_compiled(NX, g.mp != 0)) return launch_x(g, d, ph, want_cfl, np, st);
  if (g.mp) return cudaErrorInvalidValue;
  const dim3 grid(g.ny / 2, g.nzd * g.nmem);
  const size_t smem = (size_t)6 * (NX + 1) * sizeof(double2);
#define HST_XPROD(NT, PPT)        \
  big_smem(d, k_xprod<NT, PPT>); \
  k_xprod<NT, PPT><<<grid, fft_threads(6 * NX, PPT), smem, st>>>(g, np, d.Z, d.Pp, d.twx, d.dyl, ph, want_cfl, d.cfl)
  HST_SHORT_X(NX, 6 * NX, HST_XPROD)
#undef HST_XPROD
  return cudaGetLastError();
}

// each transform of the interior rows, then (when the context keeps them)
// of the four ghost rows; the ghost rows take no part in the CFL number
cudaError_t launch_zinv(const Geometry& g, const DeviceState& d, cudaStream_t st) {
  cudaError_t e = launch_zinv_main(g, d, st);
  if (e != cudaSuccess || !d.Qg) return e;
  Geometry ge;
  DeviceState de;
  edge_view(g, d, ge, de);
  return launch_zinv_main(ge, de, st);
}
cudaError_t launch_xprod(const Geometry& g, const DeviceState& d, const PhysScalars& ph, int want_cfl, int np,
                         cudaStream_t st) {
  cudaError_t e = launch_xprod_main(g, d, ph, want_cfl, np, st);
  if (e != cudaSuccess || !d.Qg) return e;
  Geometry ge;
  DeviceState de;
  edge_view(g, d, ge, de);
  return launch_xprod_main(ge, de, ph, 0, np, st);
}
cudaError_t launch_zfwd(const Geometry& g, const DeviceState& d, int np, cudaStream_t st) {
  cudaError_t e = launch_zfwd_main(g, d, np, st);
  if (e != cudaSuccess || !d.Qg) return e;
  Geometry ge;
  DeviceState de;
  edge_view(g, d, ge, de);
  return launch_zfwd_main(ge, de, np, st);
}

}  // namespace hst
