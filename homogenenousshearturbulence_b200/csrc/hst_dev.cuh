// Device building blocks of the hst substep on sm_100a: complex FP64
// arithmetic, TMA copies, the compact-stencil coefficients and 2x2 blocks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hst {

// ------------------------------------------------------------ complex ----
typedef double2 cxd;
__device__ __forceinline__ cxd mkc(double r, double i) { return make_double2(r, i); }
__device__ __forceinline__ cxd cadd(cxd a, cxd b) { return mkc(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ cxd csub(cxd a, cxd b) { return mkc(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ cxd cmul(cxd a, cxd b) { return mkc(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ cxd cscale(double s, cxd a) { return mkc(s * a.x, s * a.y); }
__device__ __forceinline__ cxd cconj(cxd a) { return mkc(a.x, -a.y); }
__device__ __forceinline__ cxd cneg(cxd a) { return mkc(-a.x, -a.y); }
// a - s * b (s real)
__device__ __forceinline__ cxd cfms(cxd a, double s, cxd b) { return mkc(a.x - s * b.x, a.y - s * b.y); }
// max that propagates NaN (fmax returns the other operand), as a positive
// quiet NaN
__device__ __forceinline__ double nan_max(double a, double b) {
  if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000LL);
  return fmax(a, b);
}
__device__ __forceinline__ cxd cexpi(double x) {
  double s, c;
  sincos(x, &s, &c);
  return mkc(c, s);
}
// the same operations on complex64 (the transforms of the mixed-precision form)
typedef float2 cxf;
__device__ __forceinline__ cxf cadd(cxf a, cxf b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ cxf csub(cxf a, cxf b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ cxf cmul(cxf a, cxf b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ cxf cscale(float s, cxf a) { return make_float2(s * a.x, s * a.y); }
__device__ __forceinline__ cxf cconj(cxf a) { return make_float2(a.x, -a.y); }
// the real scalar type of a complex type
template <typename C>
struct RealOf;
template <>
struct RealOf<double2> {
  typedef double T;
};
template <>
struct RealOf<float2> {
  typedef float T;
};
__device__ __forceinline__ double shfl_d(unsigned mask, double v, int src, int width) {
  return __shfl_sync(mask, v, src, width);
}
__device__ __forceinline__ cxd shfl_c(unsigned mask, cxd v, int src, int width) {
  return mkc(__shfl_sync(mask, v.x, src, width), __shfl_sync(mask, v.y, src, width));
}

// ------------------------------------------- TMA bulk copies, mbarriers ----
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// 1-D bulk copy global -> this CTA's shared memory, completion counted on
// bar (16-byte aligned addresses, size a multiple of 16; no multicast)
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// 4-D tiled tensor copy global -> this CTA's shared memory (no multicast);
// c0 is the innermost coordinate, in elements of the map's type
__device__ __forceinline__ void tma_load_4d(void* dst, const void* map, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
// 4-D tiled tensor copy shared -> global, completion tracked by bulk groups
__device__ __forceinline__ void tma_store_4d(const void* map, int c0, int c1, int c2, int c3, const void* src) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(map),
      "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(src))
      : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// waits until the shared memory of every committed store has been read
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase `parity` of bar to complete, at most `limit` polls;
// false when the limit ran out (the caller records an error and returns).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity, int limit) {
  for (int i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// waits until the kernels before this one in the stream have finished and their
// writes are visible (a launch_after kernel may start a little earlier)
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// a load of a field another kernel of the substep writes: an ordinary load,
// which the wait orders, never one of read-only data (no __restrict__ on the
// way to it)
__device__ __forceinline__ cxd load_field(const double2* p) { return *p; }

// line-solve kinds (src/hst_linsolve.f90:83)
enum { K_D2V = 1, K_ETA = 2, K_POISSON = 3, K_D0 = 4, K_DY = 5 };

// der(iy, n, j), n = 0..3 (D0, D1, D2, D4), j = -2..2; Fortran order
// der(0:ny-1, 0:3, -2:2) as set up by src/hst_derivatives.f90:30-56.
__device__ __forceinline__ double derv(const double* __restrict__ der, int ny, int iy, int n, int j) {
  return __ldg(der + iy + ny * (n + 4 * (j + 2)));
}
// der(iy, n, j) through a table of its distinct rows: row iy of der is row
// idx[iy] of tab, stored coefficient-major (tab[(n + 4 (j + 2)) nu + u]) so
// that the lanes of a warp, whose rows map to a few distinct rows, read a
// few neighbouring words.  On a uniform grid ny rows have a few dozen
// distinct coefficient sets (rounding of the grid differences), so the
// table stays in L1 where der itself (20 ny doubles) does not.
struct DerRows {
  const double* __restrict__ tab;
  const int* __restrict__ idx;
  int nu;
  __device__ __forceinline__ double operator()(int iy, int n, int j) const {
    return __ldg(tab + (n + 4 * (j + 2)) * nu + __ldg(idx + iy));
  }
};
struct DerFull {
  const double* __restrict__ der;
  int ny;
  __device__ __forceinline__ double operator()(int iy, int n, int j) const { return derv(der, ny, iy, n, j); }
};

// ------------------------------------------------ 2x2 block helpers ----
struct M2 {
  double a, b, c, d;  // [[a, b], [c, d]]
};
__device__ __forceinline__ M2 m2inv(M2 m) {
  double det = m.a * m.d - m.b * m.c;
  double r = 1.0 / det;
  M2 o = {m.d * r, -m.b * r, -m.c * r, m.a * r};
  return o;
}
__device__ __forceinline__ M2 m2mul(M2 x, M2 y) {
  M2 o = {x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
  return o;
}
__device__ __forceinline__ M2 m2sub(M2 x, M2 y) {
  M2 o = {x.a - y.a, x.b - y.b, x.c - y.c, x.d - y.d};
  return o;
}
__device__ __forceinline__ M2 m2neg(M2 x) {
  M2 o = {-x.a, -x.b, -x.c, -x.d};
  return o;
}
struct V2c {
  cxd u, v;
};
__device__ __forceinline__ V2c m2vec(M2 m, V2c x) {
  V2c o = {mkc(m.a * x.u.x + m.b * x.v.x, m.a * x.u.y + m.b * x.v.y),
           mkc(m.c * x.u.x + m.d * x.v.x, m.c * x.u.y + m.d * x.v.y)};
  return o;
}
__device__ __forceinline__ V2c v2sub(V2c x, V2c y) {
  V2c o = {csub(x.u, y.u), csub(x.v, y.v)};
  return o;
}
// complex 2x2
struct C2 {
  cxd a, b, c, d;
};
__device__ __forceinline__ C2 c2mul(C2 x, C2 y) {
  C2 o = {cadd(cmul(x.a, y.a), cmul(x.b, y.c)), cadd(cmul(x.a, y.b), cmul(x.b, y.d)),
          cadd(cmul(x.c, y.a), cmul(x.d, y.c)), cadd(cmul(x.c, y.b), cmul(x.d, y.d))};
  return o;
}
__device__ __forceinline__ V2c c2vec(C2 m, V2c x) {
  V2c o = {cadd(cmul(m.a, x.u), cmul(m.b, x.v)), cadd(cmul(m.c, x.u), cmul(m.d, x.v))};
  return o;
}
__device__ __forceinline__ M2 shfl_m2(unsigned mask, M2 m, int src, int w) {
  M2 o = {shfl_d(mask, m.a, src, w), shfl_d(mask, m.b, src, w), shfl_d(mask, m.c, src, w), shfl_d(mask, m.d, src, w)};
  return o;
}
__device__ __forceinline__ V2c shfl_v2(unsigned mask, V2c v, int src, int w) {
  V2c o = {shfl_c(mask, v.u, src, w), shfl_c(mask, v.v, src, w)};
  return o;
}
__device__ __forceinline__ C2 shfl_c2(unsigned mask, C2 m, int src, int w) {
  C2 o = {shfl_c(mask, m.a, src, w), shfl_c(mask, m.b, src, w), shfl_c(mask, m.c, src, w), shfl_c(mask, m.d, src, w)};
  return o;
}

}  // namespace hst
