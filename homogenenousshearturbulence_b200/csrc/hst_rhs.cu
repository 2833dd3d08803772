// The right-hand-side stage of the substep as a streaming kernel:
//
//   k_rhs_tiled  buildrhs_prepare (src/hst_equations.f90:92-141), buildrhs for
//                both product groups (:151-213), the hard damping mask
//                (src/hst_damping.f90:119-133) and the default mean-shear
//                phase shift (src/hst_equations.f90:245-257)
//
// One warp walks the rows of one Fourier column in tiles of 32.  The rows a
// tile adds to the five-point window (of the three velocities, the five product
// spectra and the two carried terms) arrive by TMA bulk copies; the tile
// after it is in flight while this one computes.
//
// The products enter the two right-hand sides through four combinations of
// constants of the column, formed once a row before any stencil is taken:
//   rhs of d2v:  D1 A + (D2 + k^2 D0) B,  A = -alfa^2 (uu - vv) - beta^2 (ww - vv) - 2 alfa beta uw,
//                                         B = i (alfa uv + beta vw)
//   rhs of eta:  D0 C + D1 D,             C = alfa beta ((uu - vv) - (ww - vv)) + (beta^2 - alfa^2) uw,
//                                         D = i (alfa vw - beta uv)
// and u, w through f = i (beta u - alfa w) (the mean column: f = (Re u, Re w), D =
// -(Re uv, Re vw)), so that a row takes nine stencils instead of twenty-three.
// What bounds it: at 768^2 x 512 the 14 Ns values of 16 B that it must move
// (2.93 ms FP64, 5.1 TB/s, 3.1 in a long run under the power cap; 3.67 with
// twenty-three stencils and six products.  2.37 in FP32, from 3.34); 384^2 x 256
// 0.536 -> 0.393 ms.  Any even ny takes this kernel:
// the last tile is ragged (nx 100, nz 75, 150 stretched rows: 0.620 -> 0.155 ms).
#include "hst_dev.cuh"
#include "hst_internal.h"
#include "hst_rhs.cuh"

namespace hst {

struct RhsArgs {
  Geometry g;
  PhysScalars ps;
  SubstepScalars sc;
  const double2 *V1, *V2, *V3;
  double2 *O1, *O2, *R1, *R2;
  const double2 *Q, *Qg;  // the product spectra, and the ghost rows' own (null: their wrap images)
  const double* derU;     // the distinct rows of der (DerRows)
  const int* derI;
  int nderU;
  const double* y;
  const double* gdamp;
  int* err;
};

constexpr int RT_WARPS = 4;
constexpr int RT_WAIT_LIMIT = 1 << 22;
#ifndef RT_MINB
#define RT_MINB 5
#endif

// shared memory of one warp: the raw rows of a tile (u, v, w, the five
// products, the two carried terms), then the 36-row window of v, f, A, B, C, D
// (with FP32 spectra: v and f in FP64, and all six in FP32)
template <typename QT>
struct RhsShape {
  static constexpr bool F32 = sizeof(QT) == 8;
  static constexpr int W = 36;
  static constexpr size_t raw = 5 * 32 * sizeof(double2) + 5 * 32 * sizeof(QT);
  static constexpr size_t win = (F32 ? 2 * W * sizeof(double2) : 0) + 6 * W * sizeof(QT);
  static constexpr size_t warp = raw + win;
};

template <typename QT>
struct Combos {
  QT A, B, C, D;
};
// the column's constants in the products' precision
template <typename R>
struct ComboConst {
  R al, be, kk, a2, b2, ab2, ab, bma;
  bool c00;
};
template <typename QT, typename R>
__device__ __forceinline__ Combos<QT> combos(const ComboConst<R>& k, QT du, QT dw, QT uv, QT vw, QT uw) {
  Combos<QT> o;
  o.A = QT{-(k.a2 * du.x + k.b2 * dw.x + k.ab2 * uw.x), -(k.a2 * du.y + k.b2 * dw.y + k.ab2 * uw.y)};
  o.B = QT{-(k.al * uv.y + k.be * vw.y), k.al * uv.x + k.be * vw.x};
  o.C = QT{k.ab * (du.x - dw.x) + k.bma * uw.x, k.ab * (du.y - dw.y) + k.bma * uw.y};
  o.D = k.c00 ? QT{-uv.x, -vw.x} : QT{k.be * uv.y - k.al * vw.y, k.al * vw.x - k.be * uv.x};
  return o;
}

template <bool EXACT, bool NONLIN, typename QT>
__global__ void __launch_bounds__(32 * RT_WARPS, RT_MINB) k_rhs_tiled(RhsArgs a) {
  typedef RhsShape<QT> S;
  typedef typename RealOf<QT>::T R;
  constexpr bool F32 = S::F32;
  constexpr int W = S::W;
  constexpr unsigned QE = sizeof(QT);
  extern __shared__ __align__(128) unsigned char smt[];
  __shared__ __align__(8) uint64_t bars[RT_WARPS];
  const Geometry& g = a.g;
  const SubstepScalars& sc = a.sc;
  const int ny = g.ny;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cgl = blockIdx.x * RT_WARPS + warp;  // the column over all members
  if (cgl >= g.ncol * g.nmem) return;
  const int mem = cgl / g.ncol, col = cgl - mem * g.ncol;
  double2* const raw = reinterpret_cast<double2*>(smt + warp * S::warp);  // u, v, w [32] each, old1, old2 [32]
  QT* const rawq = reinterpret_cast<QT*>(raw + 5 * 32);                   // five products [32]
  double2* const wv = reinterpret_cast<double2*>(smt + warp * S::warp + S::raw);  // v, f
  double2* const wf = wv + W;
  QT* const wq = reinterpret_cast<QT*>(wv) + (F32 ? 4 * W : 2 * W);  // A, B, C, D (then v, f in FP32)
  float2* const wv32 = reinterpret_cast<float2*>(wq + 4 * W);
  uint64_t* const bar = &bars[warp];
  if (lane == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
  const size_t cb = (size_t)cgl * g.rows + 2;  // row 0 of the column
  const QT* const Qc = reinterpret_cast<const QT*>(a.Q) + ((size_t)mem * 6 * g.ncol + col) * ny;
  const size_t qs = (size_t)g.ncol * ny;
  const QT* const Qgc =
      a.Qg ? reinterpret_cast<const QT*>(a.Qg) + ((size_t)mem * 6 * g.ncol + col) * 4 : nullptr;
  const size_t qgs = (size_t)g.ncol * 4;
  // lane 0 queues the rows r0 + 2 .. r0 + nr + 1 that tile t adds to the
  // window, and its carried terms
  auto issue = [&](int t) {
    const int r0 = t * 32, nr = min(32, ny - r0);
    mbar_arrive_expect_tx(bar, (unsigned)nr * (5 * 16 + (NONLIN ? 5 * QE : 0)));
    const double2* const Vg[3] = {a.V1, a.V2, a.V3};
#pragma unroll
    for (int c = 0; c < 3; ++c) bulk_g2s(raw + c * 32, Vg[c] + cb + r0 + 2, nr * 16, bar);
    bulk_g2s(raw + 3 * 32, a.O1 + cb + r0, nr * 16, bar);
    bulk_g2s(raw + 4 * 32, a.O2 + cb + r0, nr * 16, bar);
    if (NONLIN) {
      // rows ny, ny + 1: the wrapped interior rows (their phase is applied
      // to the combinations), or the ghost rows' own spectra
      const int n1 = min(nr, ny - r0 - 2);
#pragma unroll 1
      for (int p = 0; p < 5; ++p) {
        if (n1 > 0) bulk_g2s(rawq + p * 32, Qc + p * qs + r0 + 2, (unsigned)n1 * QE, bar);
        if (n1 < nr) bulk_g2s(rawq + p * 32 + n1, Qgc ? Qgc + p * qgs + 2 : Qc + p * qs, (unsigned)(nr - n1) * QE, bar);
      }
    }
  };
  wait_predecessor();
  if (lane == 0) issue(0);
  const ColConst cc = col_const(col, g, a.ps, sc, a.gdamp);
  const double al = cc.al, be = cc.be, kk = cc.kk, ni = cc.ni, gs = cc.gs;
  const ComboConst<R> kc = {(R)al,        (R)be, (R)kk, (R)(al * al), (R)(be * be), (R)(2.0 * al * be), (R)(al * be),
                            (R)(be * be - al * al), cc.c00};
  const QT ph_q = QT{(R)cc.ph_t.x, (R)cc.ph_t.y};
  // row i of the window from the raw values of one row; s != 0: the row
  // lies beyond the box, its products times the wrap phase (s < 0: conjugate)
  auto fill = [&](int i, cxd u, cxd v, cxd w, QT du, QT dw, QT uv, QT vw, QT uw, int s) {
    const cxd f = cc.c00 ? mkc(u.x, w.x) : mkc(al * w.y - be * u.y, be * u.x - al * w.x);
    wv[i] = v;
    wf[i] = f;
    if (F32) {
      wv32[i] = make_float2((float)v.x, (float)v.y);
      wv32[W + i] = make_float2((float)f.x, (float)f.y);
    }
    if (NONLIN) {
      Combos<QT> k = combos<QT, R>(kc, du, dw, uv, vw, uw);
      if (s != 0) {
        const QT e = s < 0 ? cconj(ph_q) : ph_q;
        k.A = cmul(k.A, e);
        k.B = cmul(k.B, e);
        k.C = cmul(k.C, e);
        k.D = cmul(k.D, e);
      }
      wq[i] = k.A;
      wq[W + i] = k.B;
      wq[2 * W + i] = k.C;
      wq[3 * W + i] = k.D;
    }
  };
  // rows -2 .. 1 into the window's last four rows, whence each tile moves them
  if (lane < 4) {
    const int r = lane - 2;
    QT q[5];
#pragma unroll
    for (int p = 0; p < 5; ++p) {
      if (!NONLIN) q[p] = QT{0, 0};
      else if (r >= 0) q[p] = __ldcg(Qc + p * qs + r);
      else q[p] = __ldcg(Qgc ? Qgc + p * qgs + r + 2 : Qc + p * qs + ny + r);
    }
    fill(32 + lane, load_field(a.V1 + cb + r), load_field(a.V2 + cb + r), load_field(a.V3 + cb + r), q[0], q[1], q[2], q[3], q[4],
         (r < 0 && !Qgc) ? -1 : 0);
  }
  // the default-form shift factor exp(-i gsh y(r)) of row t 32 + lane on a
  // uniform grid: the factor of the tile's first row (lane t of tbase) times
  // that of row `lane`, so that a column takes two sines a lane
  const double gsh = al * sc.dgx + be * sc.dgz;
  const int ntile = (ny + 31) / 32;
  const bool fact = !EXACT && sc.yuni && ntile <= 32;
  cxd fl = mkc(1.0, 0.0), tbase = mkc(1.0, 0.0);
  if (fact) {
    if (lane < ny) fl = cexpi(-gsh * a.y[lane + 2]);
    if (lane < ntile) tbase = cexpi(-gsh * a.y[lane * 32 + 2]);
  }
  __syncwarp();
  for (int t = 0; t < ntile; ++t) {
    const int r0 = t * 32, nr = min(32, ny - r0);
    // the last four window rows become the first four (every tile but the
    // last is full, so they are rows r0 - 2 .. r0 + 1)
    if (lane < 8) {
      const int q = lane >> 2, i = lane & 3;
      wv[q * W + i] = wv[q * W + 32 + i];
    }
    if (lane < (F32 ? 24 : 16)) {
      const int q = lane >> 2, i = lane & 3;
      wq[q * W + i] = wq[q * W + 32 + i];
    }
    __syncwarp();
    if (!mbar_wait_bounded(bar, t & 1, RT_WAIT_LIMIT)) {
      // record the failure, give the copies in flight a second bounded wait
      // to land, and leave
      if (lane == 0) atomicExch(a.err, 1);
      mbar_wait_bounded(bar, t & 1, RT_WAIT_LIMIT);
      return;
    }
    cxd o1in = mkc(0, 0), o2in = mkc(0, 0);
    if (lane < nr) {
      o1in = raw[3 * 32 + lane];
      o2in = raw[4 * 32 + lane];
      fill(4 + lane, raw[lane], raw[32 + lane], raw[64 + lane], rawq[lane], rawq[32 + lane], rawq[64 + lane],
           rawq[96 + lane], rawq[128 + lane], (r0 + 2 + lane >= ny && !Qgc) ? 1 : 0);
    }
    __syncwarp();
    if (lane == 0 && t + 1 < ntile) {
      fence_proxy_async();
      issue(t + 1);
    }
    const int r = r0 + lane;
    cxd fsh = mkc(1.0, 0.0);
    if (fact) fsh = cmul(shfl_c(0xffffffffu, tbase, t, 32), fl);
    if (lane < nr) {
      const DerRows der = {a.derU, a.derI, a.nderU};
      const int iu = __ldg(a.derI + r);
      auto dr = [&](int n, int j) { return __ldg(der.tab + (n + 4 * j) * der.nu + iu); };
      cxd r1, r2, o1, o2;
      if constexpr (!F32) {
        cxd v0 = mkc(0, 0), v2 = v0, v4 = v0, f0 = v0, f2 = v0, sA = v0, sB = v0, sC = v0, sD = v0;
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          const double d0 = dr(0, j), d1 = dr(1, j), d2 = dr(2, j), d4 = dr(3, j);
          const cxd v = wv[lane + j], f = wf[lane + j];
          v0 = mkc(v0.x + d0 * v.x, v0.y + d0 * v.y);
          v2 = mkc(v2.x + d2 * v.x, v2.y + d2 * v.y);
          v4 = mkc(v4.x + d4 * v.x, v4.y + d4 * v.y);
          f0 = mkc(f0.x + d0 * f.x, f0.y + d0 * f.y);
          f2 = mkc(f2.x + d2 * f.x, f2.y + d2 * f.y);
          if (NONLIN) {
            const double e = d2 + kk * d0;
            const QT A = wq[lane + j], B = wq[W + lane + j], C = wq[2 * W + lane + j], D = wq[3 * W + lane + j];
            sA = mkc(sA.x + d1 * A.x, sA.y + d1 * A.y);
            sB = mkc(sB.x + e * B.x, sB.y + e * B.y);
            sC = mkc(sC.x + d0 * C.x, sC.y + d0 * C.y);
            sD = mkc(sD.x + d1 * D.x, sD.y + d1 * D.y);
          }
        }
        // v equation
        const cxd un = mkc(v2.x - kk * v0.x, v2.y - kk * v0.y);
        const cxd bi = mkc(v4.x - kk * (2.0 * v2.x - kk * v0.x), v4.y - kk * (2.0 * v2.y - kk * v0.y));
        const cxd ex = mkc(sA.x + sB.x - gs * un.x, sA.y + sB.y - gs * un.y);
        r2 = mkc(sc.lambda * un.x + ni * bi.x - sc.ode2 * o2in.x + sc.ode1 * ex.x,
                 sc.lambda * un.y + ni * bi.y - sc.ode2 * o2in.y + sc.ode1 * ex.y);
        o2 = ex;
        // eta equation (mean column: u, w packed)
        o1 = mkc(sC.x + sD.x - cc.kappa * v0.y - gs * f0.x, sC.y + sD.y + cc.kappa * v0.x - gs * f0.y);
        r1 = mkc(sc.lambda * f0.x + ni * (f2.x - kk * f0.x) - sc.ode2 * o1in.x + sc.ode1 * o1.x,
                 sc.lambda * f0.y + ni * (f2.y - kk * f0.y) - sc.ode2 * o1in.y + sc.ode1 * o1.y);
      } else {
        // The mixed-precision form: the derivative right-hand sides are FP32
        // with FP32 accumulation -- the explicit half of the viscous terms,
        // the mean-shear tilting, the damping, the carried terms and the
        // products (stencil weights formed in FP64 from der, k^2 and nu and
        // rounded once, taps rounded to FP32) -- and one term stays FP64:
        // ODE(1)/dt times the unknowns (D2 - k^2 D0) v and D0 eta, the
        // Crank-Nicolson operator applied to the old state, which is larger
        // than the rest by about 1/(nu k^2 dt) and sets the increment the
        // FP64 solve resolves (all of it in FP32 measured 1.3e-5 relative L2
        // from the oracle after 30 substeps of 96^2 x 64 and 6.5e-5 at 768^2 x
        // 512, over the 1e-5 bound).
        const float k32 = kc.kk;
        cxd un = mkc(0, 0), f0 = mkc(0, 0);
        float2 bi = make_float2(0.f, 0.f), fi = bi, v0 = bi, sA = bi, sB0 = bi, sB2 = bi, sC = bi, sD = bi;
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          const double d0 = dr(0, j), d1 = dr(1, j), d2 = dr(2, j), d4 = dr(3, j);
          const double helm = d2 - kk * d0;
          const float nb = (float)(ni * (d4 - 2.0 * kk * d2 + kk * kk * d0)), nh = (float)(ni * helm);
          const cxd v = wv[lane + j], f = wf[lane + j];
          un = mkc(un.x + helm * v.x, un.y + helm * v.y);
          f0 = mkc(f0.x + d0 * f.x, f0.y + d0 * f.y);
          const float2 vf = wv32[lane + j], ff = wv32[W + lane + j];
          const float e0 = (float)d0, e1 = (float)d1, e2 = (float)d2;
          bi = make_float2(bi.x + nb * vf.x, bi.y + nb * vf.y);
          fi = make_float2(fi.x + nh * ff.x, fi.y + nh * ff.y);
          v0 = make_float2(v0.x + e0 * vf.x, v0.y + e0 * vf.y);
          if (NONLIN) {
            const QT A = wq[lane + j], B = wq[W + lane + j], C = wq[2 * W + lane + j], D = wq[3 * W + lane + j];
            sA = make_float2(sA.x + e1 * A.x, sA.y + e1 * A.y);
            sB0 = make_float2(sB0.x + e0 * B.x, sB0.y + e0 * B.y);
            sB2 = make_float2(sB2.x + e2 * B.x, sB2.y + e2 * B.y);
            sC = make_float2(sC.x + e0 * C.x, sC.y + e0 * C.y);
            sD = make_float2(sD.x + e1 * D.x, sD.y + e1 * D.y);
          }
        }
        const float gsf = (float)gs, ode2 = (float)sc.ode2, ode1 = (float)sc.ode1, kap = (float)cc.kappa;
        const float2 u2 = make_float2((float)un.x, (float)un.y), u1 = make_float2((float)f0.x, (float)f0.y);
        const float2 ex = make_float2(sA.x + (sB2.x + k32 * sB0.x) - gsf * u2.x, sA.y + (sB2.y + k32 * sB0.y) - gsf * u2.y);
        const float2 ez = make_float2(sC.x + sD.x - kap * v0.y - gsf * u1.x, sC.y + sD.y + kap * v0.x - gsf * u1.y);
        r2 = mkc(sc.lambda * un.x + (double)(bi.x - ode2 * (float)o2in.x + ode1 * ex.x),
                 sc.lambda * un.y + (double)(bi.y - ode2 * (float)o2in.y + ode1 * ex.y));
        r1 = mkc(sc.lambda * f0.x + (double)(fi.x - ode2 * (float)o1in.x + ode1 * ez.x),
                 sc.lambda * f0.y + (double)(fi.y - ode2 * (float)o1in.y + ode1 * ez.y));
        o2 = mkc(ex.x, ex.y);
        o1 = mkc(ez.x, ez.y);
      }
      if (cc.masked) r1 = r2 = o1 = o2 = mkc(0, 0);  // damping_mask
      if (!EXACT) {                                  // shear_shift, default form
        if (!fact) fsh = cexpi(-gsh * a.y[r + 2]);
        r1 = cmul(r1, fsh);
        r2 = cmul(r2, fsh);
        o1 = cmul(o1, fsh);
        o2 = cmul(o2, fsh);
      }
      a.O1[cb + r] = o1;
      a.O2[cb + r] = o2;
      a.R1[cb + r] = r1;
      a.R2[cb + r] = r2;
    }
    __syncwarp();
  }
}

template <bool EXACT, bool NONLIN, typename QT>
static cudaError_t launch_rhs_t(const RhsArgs& a, const DeviceState& d, cudaStream_t st) {
  const size_t smem = RT_WARPS * RhsShape<QT>::warp;
  const int blocks = (a.g.ncol * a.g.nmem + RT_WARPS - 1) / RT_WARPS;
  auto k = k_rhs_tiled<EXACT, NONLIN, QT>;
  smem_limit(d, k, (int)smem);
  return launch_after(k, dim3(blocks), 32 * RT_WARPS, smem, st, a);
}

cudaError_t launch_rhs_tiled(const Geometry& g, const DeviceState& d, const PhysScalars& ps, const SubstepScalars& sc,
                             int exact, int nonlin, cudaStream_t st) {
  const RhsArgs a = {g,      ps,     sc,     d.F[0], d.F[1], d.F[2],  d.F[3], d.F[4],  d.F[5],
                     d.F[6], d.Q,    d.Qg,   d.derU, d.derI, d.nderU, d.y,    d.gdamp, d.err};
  if (g.mp) {
    if (exact)
      return nonlin ? launch_rhs_t<true, true, float2>(a, d, st) : launch_rhs_t<true, false, float2>(a, d, st);
    return nonlin ? launch_rhs_t<false, true, float2>(a, d, st) : launch_rhs_t<false, false, float2>(a, d, st);
  }
  if (exact)
    return nonlin ? launch_rhs_t<true, true, double2>(a, d, st) : launch_rhs_t<true, false, double2>(a, d, st);
  return nonlin ? launch_rhs_t<false, true, double2>(a, d, st) : launch_rhs_t<false, false, double2>(a, d, st);
}

}  // namespace hst
