// The line solver of the hst substep: cyclic pentadiagonal systems, one a
// Fourier column, each solved by a group of P lanes (P a power of two, 2..32).
//
// Lane s owns a slab of consecutive rows; the slabs differ by at most one row,
// so that any number of rows runs on any P.  The algorithm is the
// reference's multi-slab bordering (src/hst_linsolve.f90:1-64, penta_forward
// :282-354, the reduced system of penta_backward :377-435) with every lane a
// slab: each lane factors its slab interior (real arithmetic, complex
// right-hand side); the 2P border unknowns then satisfy a block-cyclic
// tridiagonal system with real 2x2 blocks, solved by parallel cyclic
// reduction across the lanes; the back substitution runs per slab
// (penta_backward :461-482).  The wrap phase exp(-i theta) enters only where a
// neighbour lies across the box edge.
#pragma once
#include "hst_dev.cuh"

namespace hst {

// ------------------------------------------------- line buffer layout ----
// A line lives in shared memory slab by slab: slab s starts at s MS, MS odd
// and at least the longest slab, so that the P lanes reading their own slab at
// the same offset hit different 16-byte bank groups.
struct LineGeom {
  int n, m, rem, MS;  // rows; lane s owns m + (s < rem) of them
  unsigned inv0, inv1;  // ceil(2^20 / m), ceil(2^20 / (m + 1)): exact quotients for r (m + 1) < 2^20
  __device__ __forceinline__ int rows(int s) const { return m + (s < rem ? 1 : 0); }
  __device__ __forceinline__ int first(int s) const { return s * m + min(s, rem); }
  __device__ __forceinline__ int at(int r) const {
    const int cut = rem * (m + 1);
    if (r < cut) {
      const int s = (int)(((unsigned)r * inv1) >> 20);
      return s * MS + (r - s * (m + 1));
    }
    const int q = r - cut, s = (int)(((unsigned)q * inv0) >> 20);
    return (rem + s) * MS + (q - s * m);
  }
};
__host__ __device__ __forceinline__ LineGeom line_geom(int n, int P) {
  LineGeom G;
  G.n = n;
  G.m = n / P;
  G.rem = n - G.m * P;
  G.MS = (G.m + (G.rem ? 1 : 0)) | 1;
  G.inv0 = (unsigned)((1u << 20) + G.m - 1) / (unsigned)G.m;
  G.inv1 = (unsigned)((1u << 20) + G.m) / (unsigned)(G.m + 1);
  return G;
}
// rows of the longest slab
__host__ __device__ __forceinline__ int slab_rows(int n, int P) { return (n + P - 1) / P; }

// der in slab-major order for groups of P lanes, mM = slab_rows(n, P):
// derS[((n*5 + j)*mM + i)*P + s] = der(first(s) + i, n, j - 2), so that the P
// lanes reading row i of their own slabs read consecutive addresses.
// SH: the table (or some of its slices) copied into shared memory
template <bool SH = false>
struct SlabDerT {
  const double* __restrict__ p;
  int mM, P;
  __device__ __forceinline__ double operator()(int s, int i, int n, int j) const {
    const double* q = p + ((n * 5 + j) * mM + i) * P + s;
    if constexpr (SH)
      return *q;
    else
      return __ldg(q);
  }
};

// D0 of the slabs straight from der (Fortran order), first row r0 of slab s
struct SlabD0 {
  const double* __restrict__ der;
  int ny, r0;
  __device__ __forceinline__ double operator()(int, int i, int, int j) const { return __ldg(der + r0 + i + ny * (4 * j)); }
};

// A system's band entries before the wrap phase are c0 D0 + c2 D2 + c4 D4 with
// constants of the column (coef, src/hst_linsolve.f90:236-252): NT = 3 (D2V),
// 2 (ETA, POISSON: c4 = 0) or 1 (D0, DY: D0 itself).
struct BandConst {
  double c0, c2, c4;
};
__device__ __forceinline__ BandConst band_const(int sys, double lambda, double ni, double kk) {
  if (sys == K_D2V) return {-(kk * (lambda + ni * kk)), lambda + 2.0 * ni * kk, -ni};
  if (sys == K_ETA) return {lambda + ni * kk, -ni, 0.0};
  if (sys == K_POISSON) return {-kk, 1.0, 0.0};
  return {1.0, 0.0, 0.0};
}
template <int NT, class DST>
__device__ __forceinline__ void band_row(const BandConst& c, const DST& D, int s, int i, double a[5]) {
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    a[j] = D(s, i, 0, j);
    if (NT >= 2) a[j] = c.c0 * a[j] + c.c2 * D(s, i, 2, j);
    if (NT >= 3) a[j] += c.c4 * D(s, i, 3, j);
  }
}

__device__ __forceinline__ V2c shfl_rhs(unsigned mask, V2c v, int src, int w, bool wrap, cxd ph) {
  V2c o = shfl_v2(mask, v, src, w);
  if (wrap) {
    o.u = cmul(o.u, ph);
    o.v = cmul(o.v, ph);
  }
  return o;
}
// complex a / det by one real reciprocal
__device__ __forceinline__ V2c c2solve1(C2 m, V2c r) {
  const cxd det = csub(cmul(m.a, m.d), cmul(m.b, m.c));
  const double q = 1.0 / (det.x * det.x + det.y * det.y);
  const cxd inv = mkc(det.x * q, -det.y * q);
  const cxd n1 = csub(cmul(m.d, r.u), cmul(m.b, r.v));
  const cxd n2 = csub(cmul(m.a, r.v), cmul(m.c, r.u));
  return V2c{cmul(n1, inv), cmul(n2, inv)};
}

// Solves the line whose slab of m rows lane s holds at sb (right-hand side
// in, solution out).  ph: the wrap phase exp(-i theta).  fac: the lane's
// factor scratch, two double2 a row at fac[(2 i + k) P].
template <int P, int NT, class DST>
__device__ __forceinline__ void line_solve(const BandConst& bc, cxd ph, const DST& DS, int m, cxd* sb, double2* fac,
                                           int s, unsigned gmask) {
  const int mi = m - 2;
  // ---- forward sweep of the slab interior (penta_forward): rows 0 and 1,
  // which meet the border of the slab below, then the rest
  double u11, u12, p1, q1, u21, u22, p2, q2, w1, w2, v1, v2, sp0, sq0, sp1, sq1;
  cxd x1, x2, sx0, sx1;
  {
    double a[5];
    band_row<NT>(bc, DS, s, 0, a);
    double rp = 1.0 / a[2];
    u21 = a[3] * rp;
    u22 = a[4] * rp;
    p2 = a[0] * rp;
    q2 = a[1] * rp;
    x2 = cscale(rp, sb[0]);
    sb[0] = x2;
    fac[0] = make_double2(u21, u22);
    fac[P] = make_double2(p2, q2);
    band_row<NT>(bc, DS, s, 1, a);
    const double l = a[1];
    rp = 1.0 / (a[2] - l * u21);
    u11 = (a[3] - l * u22) * rp;
    u12 = a[4] * rp;
    p1 = -(l * p2) * rp;
    q1 = (a[0] - l * q2) * rp;
    x1 = cscale(rp, cfms(sb[1], l, x2));
    sb[1] = x1;
    fac[2 * P] = make_double2(u11, u12);
    fac[3 * P] = make_double2(p1, q1);
    w1 = -u21;
    w2 = 1.0;
    v1 = 1.0;
    v2 = 0.0;
    sx0 = mkc(x2.x + w1 * x1.x, x2.y + w1 * x1.y);
    sp0 = p2 + w1 * p1;
    sq0 = q2 + w1 * q1;
    sx1 = x1;
    sp1 = p1;
    sq1 = q1;
  }
#pragma unroll 2
  for (int i = 2; i < mi; ++i) {
    double a[5];
    band_row<NT>(bc, DS, s, i, a);
    const double l0 = a[0], l1 = a[1] - l0 * u21;
    const double rp = 1.0 / (a[2] - l0 * u22 - l1 * u11);
    const double t1 = (a[3] - l1 * u12) * rp, t2 = a[4] * rp;
    const double p = -(l0 * p2 + l1 * p1) * rp, q = -(l0 * q2 + l1 * q1) * rp;
    const cxd bx = cscale(rp, cfms(cfms(sb[i], l0, x2), l1, x1));
    sb[i] = bx;
    fac[2 * i * P] = make_double2(t1, t2);
    fac[(2 * i + 1) * P] = make_double2(p, q);
    const double w = -(u11 * w1 + u22 * w2), v = -(u11 * v1 + u22 * v2);
    sx0 = mkc(sx0.x + w * bx.x, sx0.y + w * bx.y);
    sp0 = sp0 + w * p;
    sq0 = sq0 + w * q;
    sx1 = mkc(sx1.x + v * bx.x, sx1.y + v * bx.y);
    sp1 = sp1 + v * p;
    sq1 = sq1 + v * q;
    w2 = w1;
    w1 = w;
    v2 = v1;
    v1 = v;
    u21 = u11;
    u22 = u12;
    x2 = x1;
    p2 = p1;
    q2 = q1;
    u11 = t1;
    u12 = t2;
    x1 = bx;
    p1 = p;
    q1 = q;
  }
  // the record of the slab (rec(1..28) of penta_forward): its rows 0, 1 and
  // its last two interior rows in terms of the borders below and above
  M2 L, U;
  V2c r;
  {
    const double R5 = w2 * u22 + w1 * u11, R6 = w1 * u12, R11 = v2 * u22 + v1 * u11, R12 = v1 * u12;
    const cxd XM2 = csub(x2, cscale(u21, x1));
    const double R15 = p2 - u21 * p1, R16 = q2 - u21 * q1, R17 = u22 - u21 * u11, R18 = -u21 * u12;
    // rows 0, 1 of the slab above (t = s+1)
    const int t = (s + 1) & (P - 1);
    cxd TX0 = shfl_c(gmask, sx0, t, P), TX1 = shfl_c(gmask, sx1, t, P);
    if (s == P - 1) {
      TX0 = cmul(TX0, ph);
      TX1 = cmul(TX1, ph);
    }
    const double T3 = shfl_d(gmask, sp0, t, P), T4 = shfl_d(gmask, sq0, t, P), T5 = shfl_d(gmask, R5, t, P),
                 T6 = shfl_d(gmask, R6, t, P), T9 = shfl_d(gmask, sp1, t, P), T10 = shfl_d(gmask, sq1, t, P),
                 T11 = shfl_d(gmask, R11, t, P), T12 = shfl_d(gmask, R12, t, P);
    // the two border rows of the slab (its rows mi, mi+1): L c_{s-1} + D c_s +
    // U c_{s+1} = r, scaled by D^-1
    double e[5], f[5];
    band_row<NT>(bc, DS, s, mi, e);
    band_row<NT>(bc, DS, s, mi + 1, f);
    const M2 D = {e[2] - (e[0] * R17 + e[1] * u11) - e[4] * T3, e[3] - (e[0] * R18 + e[1] * u12) - e[4] * T4,
                  f[1] - f[0] * u11 - (f[3] * T3 + f[4] * T9), f[2] - f[0] * u12 - (f[3] * T4 + f[4] * T10)};
    const M2 Di = m2inv(D);
    L = m2mul(Di, M2{-(e[0] * R15 + e[1] * p1), -(e[0] * R16 + e[1] * q1), -(f[0] * p1), -(f[0] * q1)});
    U = m2mul(Di, M2{-(e[4] * T5), -(e[4] * T6), -(f[3] * T5 + f[4] * T11), -(f[3] * T6 + f[4] * T12)});
    const cxd RB1 = sb[mi], RB2 = sb[mi + 1];
    V2c b;
    b.u = mkc(RB1.x - e[0] * XM2.x - e[1] * x1.x - e[4] * TX0.x, RB1.y - e[0] * XM2.y - e[1] * x1.y - e[4] * TX0.y);
    b.v = mkc(RB2.x - f[0] * x1.x - f[3] * TX0.x - f[4] * TX1.x, RB2.y - f[0] * x1.y - f[3] * TX0.y - f[4] * TX1.y);
    r = m2vec(Di, b);
  }
  // parallel cyclic reduction with unit diagonal blocks: strides d = 1, 2, .., P/4
  const cxd phc = cconj(ph);
#pragma unroll 1
  for (int d = 1; 2 * d < P; d <<= 1) {
    const int sm = (s - d) & (P - 1), sp = (s + d) & (P - 1);
    const M2 Lm = shfl_m2(gmask, L, sm, P), Um = shfl_m2(gmask, U, sm, P);
    const M2 Lp = shfl_m2(gmask, L, sp, P), Up = shfl_m2(gmask, U, sp, P);
    const V2c rm = shfl_rhs(gmask, r, sm, P, s < d, phc), rq = shfl_rhs(gmask, r, sp, P, s + d >= P, ph);
    const M2 X = m2mul(L, Um), Y = m2mul(U, Lp);
    const M2 Di = m2inv(M2{1.0 - X.a - Y.a, -X.b - Y.b, -X.c - Y.c, 1.0 - X.d - Y.d});
    r = m2vec(Di, v2sub(v2sub(r, m2vec(L, rm)), m2vec(U, rq)));
    L = m2neg(m2mul(Di, m2mul(L, Lm)));
    U = m2neg(m2mul(Di, m2mul(U, Up)));
  }
  // last level: both neighbours are lane s ^ P/2, one of them across the edge
  V2c c;
  {
    const int q = s ^ (P >> 1);
    const bool lo = s < (P >> 1);
    const M2 Wr = lo ? L : U, Nr = lo ? U : L;  // the block whose neighbour wraps, the other
    const cxd e = lo ? phc : ph;
    const C2 M = {mkc(Nr.a + Wr.a * e.x, Wr.a * e.y), mkc(Nr.b + Wr.b * e.x, Wr.b * e.y),
                  mkc(Nr.c + Wr.c * e.x, Wr.c * e.y), mkc(Nr.d + Wr.d * e.x, Wr.d * e.y)};
    const C2 Mq = shfl_c2(gmask, M, q, P);
    const V2c rq = shfl_v2(gmask, r, q, P);
    const C2 S = c2mul(M, Mq);
    c = c2solve1(C2{mkc(1.0 - S.a.x, -S.a.y), cneg(S.b), cneg(S.c), mkc(1.0 - S.d.x, -S.d.y)}, v2sub(r, c2vec(M, rq)));
  }
  // the border of the slab below, then the back substitution (penta_backward :467-482)
  const V2c y = shfl_rhs(gmask, c, (s - 1) & (P - 1), P, s == 0, phc);
  sb[mi] = c.u;
  sb[mi + 1] = c.v;
  cxd xk1 = c.u, xk2 = c.v;
#pragma unroll 4
  for (int i = mi - 1; i >= 0; --i) {
    const double2 t = fac[2 * i * P], b = fac[(2 * i + 1) * P];
    const cxd xr = sb[i];
    const cxd xk = mkc(xr.x - b.x * y.u.x - b.y * y.v.x - t.x * xk1.x - t.y * xk2.x,
                       xr.y - b.x * y.u.y - b.y * y.v.y - t.x * xk1.y - t.y * xk2.y);
    sb[i] = xk;
    xk2 = xk1;
    xk1 = xk;
  }
}

// ------------------------------------- the D0 system, factored once ----
// The matrix of KIND_D0 and KIND_DY (the compact D0 operator) is the same
// for every Fourier column; only the wrap phase differs.  d0_factor runs the
// matrix half of the solve once per context and keeps, per lane s of the
// group, every matrix quantity that the right-hand side meets: per interior
// row the two elimination multipliers, the pivot reciprocal, the record
// weights w, v and the back-substitution factors; the border-row
// coefficients; each reduction level's two 2x2 blocks; the blocks of the last
// level.  d0_forward and d0_back then run only the right-hand-side half, so that
// the divisions, the block inverses and all matrix shuffles leave every column's
// dependency chain.  Field f of lane s sits at tab[f P + s]; the fields that
// follow the rows start at 9 (mM - 2) on every lane.
__host__ __device__ constexpr int d0_levels(int P) {
  int n = 0;
  for (int d = 1; 2 * d < P; d <<= 1) ++n;
  return n;
}
__host__ __device__ constexpr int d0_fields(int mM, int P) { return 9 * (mM - 2) + 7 + 8 * d0_levels(P) + 24; }

template <int P, class DST>
__device__ void d0_factor(const DST& DS, int m, int mM, int s, unsigned gmask, double* __restrict__ tab) {
  const int mi = m - 2;
  const BandConst bc = {1.0, 0.0, 0.0};
  auto put = [&](int f, double v) { tab[(size_t)f * P + s] = v; };
  double u11 = 0, u12 = 0, p1 = 0, q1 = 0, u21 = 0, u22 = 0, p2 = 0, q2 = 0;
  double w1 = 0, w2 = 0, v1 = 0, v2 = 0, sp0 = 0, sq0 = 0, sp1 = 0, sq1 = 0;
  // (the next row's entries are loaded before this row's fields are stored: the
  // one warp's chain of rows would wait for them)
  double next[5];
  band_row<1>(bc, DS, s, 0, next);
  for (int i = 0; i < mi; ++i) {
    double a[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) a[j] = next[j];
    band_row<1>(bc, DS, s, i + 1, next);  // (row mi is the first border row)
    double p = 0, q = 0, l0 = 0, l1 = 0;
    if (i == 0) {
      p = a[0];
      q = a[1];
    }
    if (i == 1) q = a[0];
    if (i >= 2) {
      l0 = a[0];
      a[1] = a[1] - l0 * u21;
      a[2] = a[2] - l0 * u22;
      p = p - l0 * p2;
      q = q - l0 * q2;
    }
    if (i >= 1) {
      l1 = a[1];
      a[2] = a[2] - l1 * u11;
      a[3] = a[3] - l1 * u12;
      p = p - l1 * p1;
      q = q - l1 * q1;
    }
    const double rp = 1.0 / a[2];
    const double t1 = a[3] * rp, t2 = a[4] * rp;
    p = p * rp;
    q = q * rp;
    const double w = (i == 0) ? 1.0 : -(u11 * w1 + u22 * w2);
    const double v = (i == 1) ? 1.0 : -(u11 * v1 + u22 * v2);
    put(9 * i + 0, l0);
    put(9 * i + 1, l1);
    put(9 * i + 2, rp);
    put(9 * i + 3, w);
    put(9 * i + 4, v);
    put(9 * i + 5, t1);
    put(9 * i + 6, t2);
    put(9 * i + 7, p);
    put(9 * i + 8, q);
    sp0 = sp0 + w * p;
    sq0 = sq0 + w * q;
    sp1 = sp1 + v * p;
    sq1 = sq1 + v * q;
    w2 = w1;
    w1 = w;
    v2 = v1;
    v1 = v;
    u21 = u11;
    u22 = u12;
    p2 = p1;
    q2 = q1;
    u11 = t1;
    u12 = t2;
    p1 = p;
    q1 = q;
  }
  const double R3 = sp0, R4 = sq0, R5 = w2 * u22 + w1 * u11, R6 = w1 * u12;
  const double R9 = sp1, R10 = sq1, R11 = v2 * u22 + v1 * u11, R12 = v1 * u12;
  const double R15 = p2 - u21 * p1, R16 = q2 - u21 * q1, R17 = u22 - u21 * u11, R18 = -u21 * u12;
  const double R21 = p1, R22 = q1, R23 = u11, R24 = u12;
  const int t = (s + 1) & (P - 1);
  const double T3 = shfl_d(gmask, R3, t, P), T4 = shfl_d(gmask, R4, t, P), T5 = shfl_d(gmask, R5, t, P),
               T6 = shfl_d(gmask, R6, t, P), T9 = shfl_d(gmask, R9, t, P), T10 = shfl_d(gmask, R10, t, P),
               T11 = shfl_d(gmask, R11, t, P), T12 = shfl_d(gmask, R12, t, P);
  double ab1[5], ab2[5];
  band_row<1>(bc, DS, s, mi, ab1);
  band_row<1>(bc, DS, s, mi + 1, ab2);
  const double c1m4 = ab1[0], c1m3 = ab1[1], d11 = ab1[2], d12 = ab1[3], c10 = ab1[4];
  const double c2m3 = ab2[0], d21 = ab2[1], d22 = ab2[2], c20 = ab2[3], c21 = ab2[4];
  const int B = 9 * (mM - 2);
  put(B + 0, u21);
  put(B + 1, c1m4);
  put(B + 2, c1m3);
  put(B + 3, c10);
  put(B + 4, c2m3);
  put(B + 5, c20);
  put(B + 6, c21);
  M2 L = {-(c1m4 * R15 + c1m3 * R21), -(c1m4 * R16 + c1m3 * R22), -(c2m3 * R21), -(c2m3 * R22)};
  M2 D = {d11 - (c1m4 * R17 + c1m3 * R23) - c10 * T3, d12 - (c1m4 * R18 + c1m3 * R24) - c10 * T4,
          d21 - c2m3 * R23 - (c20 * T3 + c21 * T9), d22 - c2m3 * R24 - (c20 * T4 + c21 * T10)};
  M2 U = {-(c10 * T5), -(c10 * T6), -(c20 * T5 + c21 * T11), -(c20 * T6 + c21 * T12)};
  auto put2 = [&](int f, M2 x) {
    put(f, x.a);
    put(f + 1, x.b);
    put(f + 2, x.c);
    put(f + 3, x.d);
  };
  int f = B + 7;
  for (int d = 1; 2 * d < P; d <<= 1, f += 8) {
    const int sm = (s - d) & (P - 1), sp = (s + d) & (P - 1);
    M2 Lm = shfl_m2(gmask, L, sm, P), Dm = shfl_m2(gmask, D, sm, P), Um = shfl_m2(gmask, U, sm, P);
    M2 Lp = shfl_m2(gmask, L, sp, P), Dp = shfl_m2(gmask, D, sp, P), Up = shfl_m2(gmask, U, sp, P);
    M2 A = m2mul(L, m2inv(Dm));
    M2 Gm = m2mul(U, m2inv(Dp));
    M2 Ln = m2neg(m2mul(A, Lm));
    M2 Un = m2neg(m2mul(Gm, Up));
    M2 Dn = m2sub(m2sub(D, m2mul(A, Um)), m2mul(Gm, Lp));
    put2(f, A);
    put2(f + 4, Gm);
    L = Ln;
    U = Un;
    D = Dn;
  }
  // the last level with unit diagonal: D^-1 L, D^-1 U, the same of lane
  // s ^ P/2, and the two inverses
  const int q = s ^ (P >> 1);
  const M2 Di = m2inv(D);
  const M2 l = m2mul(Di, L), u = m2mul(Di, U);
  put2(f, l);
  put2(f + 4, u);
  put2(f + 8, shfl_m2(gmask, l, q, P));
  put2(f + 12, shfl_m2(gmask, u, q, P));
  put2(f + 16, Di);
  put2(f + 20, shfl_m2(gmask, Di, q, P));
}

// The solve with the D0 matrix from the table of d0_factor (sb as line_solve's).
// d0_forward runs the forward sweep and the reduction and leaves each lane the
// borders of its slab (c: its own last two rows, y: those of the slab below).
template <int P, bool SH>
struct D0Table {
  const double* __restrict__ ts;  // tab + s
  __device__ __forceinline__ double operator()(int f) const {
    if constexpr (SH)
      return ts[f * P];
    else
      return __ldg(ts + f * P);
  }
  __device__ __forceinline__ M2 m2(int f) const {
    return M2{(*this)(f), (*this)(f + 1), (*this)(f + 2), (*this)(f + 3)};
  }
};
template <int P, class TAB>
__device__ __forceinline__ void d0_forward(cxd ph, const TAB& T, int mM, int m, cxd* sb, int s, unsigned gmask, V2c& c,
                                           V2c& y) {
  const int mi = m - 2;
  cxd x1, x2, sx0, sx1;
  {
    const double rp0 = T(2), l1 = T(10), rp1 = T(11), w = T(12);
    x2 = cscale(rp0, sb[0]);
    sb[0] = x2;
    x1 = cscale(rp1, cfms(sb[1], l1, x2));
    sb[1] = x1;
    sx0 = mkc(x2.x + w * x1.x, x2.y + w * x1.y);
    sx1 = x1;
  }
#pragma unroll 2
  for (int i = 2; i < mi; ++i) {
    const double l0 = T(9 * i + 0), l1 = T(9 * i + 1), rp = T(9 * i + 2), w = T(9 * i + 3), v = T(9 * i + 4);
    const cxd bx = cscale(rp, cfms(cfms(sb[i], l0, x2), l1, x1));
    sb[i] = bx;
    sx0 = mkc(sx0.x + w * bx.x, sx0.y + w * bx.y);
    sx1 = mkc(sx1.x + v * bx.x, sx1.y + v * bx.y);
    x2 = x1;
    x1 = bx;
  }
  const int B = 9 * (mM - 2);
  V2c r;
  {
    const double u21 = T(B), c1m4 = T(B + 1), c1m3 = T(B + 2), c10 = T(B + 3), c2m3 = T(B + 4), c20 = T(B + 5),
                 c21 = T(B + 6);
    const int t = (s + 1) & (P - 1);
    cxd TX0 = shfl_c(gmask, sx0, t, P), TX1 = shfl_c(gmask, sx1, t, P);
    if (s == P - 1) {
      TX0 = cmul(TX0, ph);
      TX1 = cmul(TX1, ph);
    }
    const cxd XM2 = csub(x2, cscale(u21, x1));
    const cxd RB1 = sb[mi], RB2 = sb[mi + 1];
    r.u = mkc(RB1.x - c1m4 * XM2.x - c1m3 * x1.x - c10 * TX0.x, RB1.y - c1m4 * XM2.y - c1m3 * x1.y - c10 * TX0.y);
    r.v = mkc(RB2.x - c2m3 * x1.x - c20 * TX0.x - c21 * TX1.x, RB2.y - c2m3 * x1.y - c20 * TX0.y - c21 * TX1.y);
  }
  const cxd phc = cconj(ph);
  int f = B + 7;
#pragma unroll
  for (int d = 1; 2 * d < P; d <<= 1, f += 8) {
    const int sm = (s - d) & (P - 1), sp = (s + d) & (P - 1);
    const M2 A = T.m2(f), Gm = T.m2(f + 4);
    const V2c rm = shfl_rhs(gmask, r, sm, P, s < d, phc), rq = shfl_rhs(gmask, r, sp, P, s + d >= P, ph);
    r = v2sub(v2sub(r, m2vec(A, rm)), m2vec(Gm, rq));
  }
  {
    const int q = s ^ (P >> 1);
    const bool lo = s < (P >> 1);
    // the wrapping block of this lane is l when s < P/2 (conjugate phase), u
    // otherwise; of lane q the other way round
    const M2 l = T.m2(f), u = T.m2(f + 4), lq = T.m2(f + 8), uq = T.m2(f + 12);
    const M2 Wr = lo ? l : u, Nr = lo ? u : l, Wq = lo ? uq : lq, Nq = lo ? lq : uq;
    const cxd e = lo ? phc : ph, eq = cconj(e);
    const C2 M = {mkc(Nr.a + Wr.a * e.x, Wr.a * e.y), mkc(Nr.b + Wr.b * e.x, Wr.b * e.y),
                  mkc(Nr.c + Wr.c * e.x, Wr.c * e.y), mkc(Nr.d + Wr.d * e.x, Wr.d * e.y)};
    const C2 Mq = {mkc(Nq.a + Wq.a * eq.x, Wq.a * eq.y), mkc(Nq.b + Wq.b * eq.x, Wq.b * eq.y),
                   mkc(Nq.c + Wq.c * eq.x, Wq.c * eq.y), mkc(Nq.d + Wq.d * eq.x, Wq.d * eq.y)};
    const C2 S = c2mul(M, Mq);
    const C2 S1 = {mkc(1.0 - S.a.x, -S.a.y), cneg(S.b), cneg(S.c), mkc(1.0 - S.d.x, -S.d.y)};
    const M2 Di = T.m2(f + 16), Dq = T.m2(f + 20);
    const V2c rr = m2vec(Di, r), rq = m2vec(Dq, shfl_v2(gmask, r, q, P));
    c = c2solve1(S1, v2sub(rr, c2vec(M, rq)));
  }
  y = shfl_rhs(gmask, c, (s - 1) & (P - 1), P, s == 0, phc);
}
// one row of the back substitution: row i of the slab from its forward value,
// the borders below and the two rows above
template <class TAB>
__device__ __forceinline__ cxd d0_back(const TAB& T, int i, cxd xr, const V2c& y, cxd xk1, cxd xk2) {
  const double U1 = T(9 * i + 5), U2 = T(9 * i + 6), B1 = T(9 * i + 7), B2 = T(9 * i + 8);
  return mkc(xr.x - B1 * y.u.x - B2 * y.v.x - U1 * xk1.x - U2 * xk2.x,
             xr.y - B1 * y.u.y - B2 * y.v.y - U1 * xk1.y - U2 * xk2.y);
}
template <int P, bool SH>
__device__ __forceinline__ void line_solve_d0(cxd ph, const double* __restrict__ tab, int mM, int m, cxd* sb, int s,
                                              unsigned gmask) {
  const int mi = m - 2;
  const D0Table<P, SH> T = {tab + s};
  V2c c, y;
  d0_forward<P>(ph, T, mM, m, sb, s, gmask, c, y);
  cxd xk1 = c.u, xk2 = c.v;
  sb[mi] = xk1;
  sb[mi + 1] = xk2;
#pragma unroll 2
  for (int i = mi - 1; i >= 0; --i) {
    const cxd xk = d0_back(T, i, sb[i], y, xk1, xk2);
    sb[i] = xk;
    xk2 = xk1;
    xk1 = xk;
  }
}

// A line shifted in place (shift_unweighted, src/hst_equations.f90:263-293):
// the D0 solve with the wrap pt, row r times the node phase, the D0 stencil
// with the ghost images of pn.  The stencil follows two rows behind the back
// substitution in registers; the rows at the slab's ends wait for the
// neighbours' (the sums run over j = -2..2 in order).  node(i): the phase of row
// i of the slab, asked for from the last row down.
template <int P, class TAB, class DST, class NODE>
__device__ __forceinline__ void shift_line(cxd pt, cxd pn, const TAB& T, const DST& DS, int mM, int m, cxd* sb, int s,
                                           unsigned gmask, NODE& node) {
  V2c c, y;
  d0_forward<P>(pt, T, mM, m, sb, s, gmask, c, y);
  cxd xk1, xk2;        // rows i + 1, i + 2 of the solution
  cxd z1, z2, z3, z4;  // rows i + 1 .. i + 4 times their phases
  cxd top0, top1;      // rows m - 2, m - 1 likewise
  {
    const cxd e1 = node(m - 1), e0 = node(m - 2), f1 = node(m - 3), f0 = node(m - 4);
    top1 = cmul(c.v, e1);
    top0 = cmul(c.u, e0);
    const cxd a = d0_back(T, m - 3, sb[m - 3], y, c.u, c.v);
    const cxd b = d0_back(T, m - 4, sb[m - 4], y, a, c.u);
    xk1 = b;
    xk2 = a;
    z4 = top1;
    z3 = top0;
    z2 = cmul(a, f1);
    z1 = cmul(b, f0);
    // the sums of rows m - 1 and m - 2 over the rows of this slab
    const double h0 = DS(s, m - 1, 0, 0), h1 = DS(s, m - 1, 0, 1), h2 = DS(s, m - 1, 0, 2);
    const double g0 = DS(s, m - 2, 0, 0), g1 = DS(s, m - 2, 0, 1), g2 = DS(s, m - 2, 0, 2), g3 = DS(s, m - 2, 0, 3);
    sb[m - 1] = mkc(h0 * z2.x + h1 * z3.x + h2 * z4.x, h0 * z2.y + h1 * z3.y + h2 * z4.y);
    sb[m - 2] = mkc(g0 * z1.x + g1 * z2.x + g2 * z3.x + g3 * z4.x, g0 * z1.y + g1 * z2.y + g2 * z3.y + g3 * z4.y);
  }
#pragma unroll 2
  for (int i = m - 5; i >= 0; --i) {
    const cxd e = node(i);
    const double c0 = DS(s, i + 2, 0, 0), c1 = DS(s, i + 2, 0, 1), c2 = DS(s, i + 2, 0, 2), c3 = DS(s, i + 2, 0, 3),
                 c4 = DS(s, i + 2, 0, 4);
    const cxd x = d0_back(T, i, sb[i], y, xk1, xk2);
    const cxd z = cmul(x, e);
    sb[i + 2] = mkc(c0 * z.x + c1 * z1.x + c2 * z2.x + c3 * z3.x + c4 * z4.x,
                    c0 * z.y + c1 * z1.y + c2 * z2.y + c3 * z3.y + c4 * z4.y);
    xk2 = xk1;
    xk1 = x;
    z4 = z3;
    z3 = z2;
    z2 = z1;
    z1 = z;
  }
  // the slab's ends
  const int up = (s + 1) & (P - 1), dn = (s - 1) & (P - 1);
  cxd a0 = shfl_c(gmask, z1, up, P), a1 = shfl_c(gmask, z2, up, P);
  cxd b0 = shfl_c(gmask, top0, dn, P), b1 = shfl_c(gmask, top1, dn, P);
  if (s == P - 1) {
    a0 = cmul(a0, pn);
    a1 = cmul(a1, pn);
  }
  if (s == 0) {
    b0 = cmul(b0, cconj(pn));
    b1 = cmul(b1, cconj(pn));
  }
  const double h3 = DS(s, m - 1, 0, 3), h4 = DS(s, m - 1, 0, 4), g4 = DS(s, m - 2, 0, 4);
  const cxd t1 = sb[m - 1], t0 = sb[m - 2];
  sb[m - 1] = mkc(t1.x + h3 * a0.x + h4 * a1.x, t1.y + h3 * a0.y + h4 * a1.y);
  sb[m - 2] = mkc(t0.x + g4 * a0.x, t0.y + g4 * a0.y);
  const double p0 = DS(s, 0, 0, 0), p1 = DS(s, 0, 0, 1), p2 = DS(s, 0, 0, 2), p3 = DS(s, 0, 0, 3), p4 = DS(s, 0, 0, 4);
  const double q0 = DS(s, 1, 0, 0), q1 = DS(s, 1, 0, 1), q2 = DS(s, 1, 0, 2), q3 = DS(s, 1, 0, 3), q4 = DS(s, 1, 0, 4);
  sb[0] = mkc(p0 * b0.x + p1 * b1.x + p2 * z1.x + p3 * z2.x + p4 * z3.x,
              p0 * b0.y + p1 * b1.y + p2 * z1.y + p3 * z2.y + p4 * z3.y);
  sb[1] = mkc(q0 * b1.x + q1 * z1.x + q2 * z2.x + q3 * z3.x + q4 * z4.x,
              q0 * b1.y + q1 * z1.y + q2 * z2.y + q3 * z3.y + q4 * z4.y);
}

// The five-point stencil n (0: D0, 1: D1) of a line held slab by slab in
// shared memory, in place: lane s computes the m rows of its slab with a
// sliding window, the two rows beyond each end of the slab from the
// neighbouring lanes (by shuffle, taken before anything is written) and,
// across the box edge, the shear-periodic ghost images f(ny + k) = f(k) ph,
// f(-k) = f(ny - k) conj(ph) (wrap_rows, src/hst_mpi.f90:340-355), or, with
// `ghosts` (rows -2, -1, ny, ny + 1), those rows.  The sum runs over j = -2..2
// in order, as the reference's stencils do.
template <int P, class DST>
__device__ __forceinline__ void slab_stencil(int n, const DST& DS, cxd* sb, int m, int s, cxd ph, unsigned gmask,
                                             const cxd* ghosts = nullptr) {
  const cxd f0 = sb[0], f1 = sb[1], l0 = sb[m - 2], l1 = sb[m - 1];
  const int up = (s + 1) & (P - 1), dn = (s - 1) & (P - 1);
  cxd a0 = shfl_c(gmask, f0, up, P), a1 = shfl_c(gmask, f1, up, P);  // rows m, m + 1 of the slab
  cxd b0 = shfl_c(gmask, l0, dn, P), b1 = shfl_c(gmask, l1, dn, P);  // rows -2, -1
  if (s == P - 1) {
    a0 = cmul(a0, ph);
    a1 = cmul(a1, ph);
  }
  if (s == 0) {
    b0 = cmul(b0, cconj(ph));
    b1 = cmul(b1, cconj(ph));
  }
  if (ghosts) {
    if (s == 0) b0 = ghosts[0], b1 = ghosts[1];
    if (s == P - 1) a0 = ghosts[2], a1 = ghosts[3];
  }
  cxd w0 = b0, w1 = b1, w2 = f0, w3 = f1, w4 = sb[2];
#pragma unroll 2
  for (int i = 0; i < m; ++i) {
    const double c0 = DS(s, i, n, 0), c1 = DS(s, i, n, 1), c2 = DS(s, i, n, 2), c3 = DS(s, i, n, 3),
                 c4 = DS(s, i, n, 4);
    const int nx = i + 3;
    const cxd nxt = nx < m ? sb[nx] : (nx == m ? a0 : a1);
    sb[i] = mkc(c0 * w0.x + c1 * w1.x + c2 * w2.x + c3 * w3.x + c4 * w4.x,
                c0 * w0.y + c1 * w1.y + c2 * w2.y + c3 * w3.y + c4 * w4.y);
    w0 = w1;
    w1 = w2;
    w2 = w3;
    w3 = w4;
    w4 = nxt;
  }
}

}  // namespace hst
