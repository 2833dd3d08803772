// The x stage of the hst substep for the compiled transform lengths:
//
//   k_x   Z -> x-inverse (c2r) of u, v, w; the products times 1/(2 nxd nzd);
//         the CFL maximum; x-forward (r2c) of the products truncated to the
//         nx+1 retained modes (Pp)
//
// The right-hand sides of the v-eta form depend on uu, vv and ww through uu - vv
// and ww - vv alone (k^2 vv = alfa^2 vv + beta^2 vv), so the substep takes five
// products, uu - vv, ww - vv, uv, vw, uw (NP = 5); the pressure needs all six,
// uu, vv, ww, uv, vw, uw (NP = 6).
//
// (to_x_points with zero padding and RFT, build_products for both groups,
// compute_cfl and HFT: src/hst_transforms.f90:85-133, 163-179,
// src/hst_fft.f90:211-237).  Other lengths run k_xprod (hst_transforms.cu).
//
// One tile is two rows y0, y0 + 1 at one z point.  Two real lines ride on one
// complex line, the two rows of one component: three lines in (u, v, w), five
// or six out (one a product), separated by Hermitian symmetry.  N = R0 R1 R2 splits
// the transform into three register stages with two exchanges each way, and
// what bounds the kernel is the shared-memory traffic of those exchanges and
// the FP64 arithmetic, so the split is chosen to keep both small:
//   - the first inverse and the last forward stage work on the butterflies j
//     and N/R0 - j together, so that every mode m and its mirror N - m meet
//     in one thread's registers: a retained mode is read once from global
//     memory (both rows side by side), and the separation of the two real
//     spectra needs no exchange;
//   - the last inverse stage, the products and the first forward stage are one
//     pass: the x points v + (N/R2) r that a radix-R2 butterfly of each of
//     the three lines leaves in a thread's registers are the inputs of the
//     first forward radix-R2 butterfly of each product;
//   - the stages run in place (decimation in frequency on the way in, in time
//     on the way out), so that one barrier separates two stages, and the
//     last inverse and first forward twiddles are loaded once for all lines.
// Line layout: element (p0, j), p0 < R0, j < N/R0, at p0 S0 + j with S0 odd;
// lanes run over p0 first in the two inner stages, over j in the outer ones,
// which keeps 16-byte accesses (R0 = 8) and 8-byte accesses (R0 = 16) free of
// bank conflicts.  The tile comes in and goes out by tensor copies of 32
// bytes a mode (two rows in FP64, four in FP32 up to 768 points): lane-wise
// loads and stores of the same 32 bytes at the 64-byte stride of the
// [ix][Ty] layout took 75 of the kernel's 185 million L1 wavefronts and 848
// against 668 us at 768 points.
// Measured a substep, against a Stockham kernel of four exchanges each way and
// staged lines (k_xprod's form), B200: 768^2 x 512 FP64 9.70 -> 4.86 ms, FP32
// 7.26 -> 2.38; 384^2 x 256 FP64 1.10 -> 0.556 ms, FP32 0.79 -> 0.307; 1536^2 x 128
// FP32 9.40 -> 3.11; 512 x 256 x 200 2.40 -> 0.387.  In FP64
// at 768 points the L1 pipe is 70 % and the FP64 pipe 53 % busy, in FP32 62 %
// with issue at 70 %: both near what one tile's exchanges and butterflies allow,
// HBM at 40 %.
#include "hst_dev.cuh"
#include "hst_fft.cuh"
#include "hst_internal.h"

namespace hst {

// The plan of length N: radices, row pairs a tile, threads a tile, tiles a
// block (G > 1: a warp each, for the shortest lengths), resident blocks asked
// of the compiler.
template <int N, typename C>
struct XPlan;
#define HST_XPLAN(N_, C_, r0, r1, r2, rp, t, g, mb)                                  \
  template <>                                                                        \
  struct XPlan<N_, C_> {                                                             \
    static constexpr int R0 = r0, R1 = r1, R2 = r2, RP = rp, T = t, G = g, MINB = mb; \
  };
HST_XPLAN(96, double2, 8, 3, 4, 1, 32, 4, 4)
HST_XPLAN(128, double2, 8, 4, 4, 1, 32, 4, 4)
HST_XPLAN(192, double2, 8, 6, 4, 1, 64, 1, 9)
HST_XPLAN(256, double2, 8, 8, 4, 1, 64, 1, 8)
HST_XPLAN(384, double2, 8, 12, 4, 1, 96, 1, 5)
HST_XPLAN(512, double2, 8, 16, 4, 1, 96, 1, 4)
HST_XPLAN(768, double2, 8, 16, 6, 1, 160, 1, 3)
HST_XPLAN(1024, double2, 8, 16, 8, 1, 192, 1, 2)
HST_XPLAN(1536, double2, 8, 24, 8, 1, 384, 1, 1)
HST_XPLAN(96, float2, 16, 1, 6, 2, 32, 4, 4)
HST_XPLAN(192, float2, 16, 3, 4, 2, 64, 1, 8)
HST_XPLAN(384, float2, 16, 6, 4, 2, 128, 1, 5)
HST_XPLAN(768, float2, 16, 12, 4, 2, 192, 1, 3)
HST_XPLAN(1536, float2, 16, 16, 6, 1, 192, 1, 3)
#undef HST_XPLAN

// Modes of one tensor copy of a tile with nxB modes: all of them up to 256
// (the largest box), else half of them rounded up to a multiple of eight, so
// that the second copy's shared address (three components of at least 16
// bytes a mode further) stays 128-byte aligned.
__host__ __device__ constexpr int x_box(int nxB) { return nxB <= 256 ? nxB : ((nxB + 1) / 2 + 7) / 8 * 8; }

constexpr int X_WAIT_LIMIT = 1 << 22;  // polls of the tile's TMA barrier before giving up

template <int N, typename C>
struct XShape {
  typedef XPlan<N, C> P;
  static constexpr int R0 = P::R0, R1 = P::R1, R2 = P::R2, T = P::T, G = P::G;
  static_assert(R0 * R1 * R2 == N, "the radices multiply to N");
  static constexpr int RP = P::RP;       // row pairs a tile
  static_assert(RP == 1 || sizeof(C) == 8, "two row pairs in FP32 only");
  static constexpr int M = N / R0;       // butterflies of an outer stage
  static constexpr int H = M / 2;        // pairs (j, M - j) of them
  static constexpr int S0 = M | 1;       // stride of the p0 blocks
  static constexpr int LS = R0 * S0;     // line stride
  static constexpr int SP = 3 * LS + (RP > 1 ? 8 : 0);  // stride of the row pairs' three lines (half a bank row off)
  static constexpr int NU = R0 * R2;     // butterflies of the middle stage
  static constexpr int NV = R0 * R1;     // butterflies of the fused stage
  static constexpr int NO = RP * 3 * H;  // units of an outer stage on three lines a row pair
  // the retained modes m <= nx <= (N - 2) / 3 lie at r < RH in m = j + r M
  static constexpr int RH = (N - 2) / 3 / M + 1 < R0 / 2 ? (N - 2) / 3 / M + 1 : R0 / 2;
  static constexpr int NB = (N + 1) / 3 > 256 ? 2 : 1;  // the most tensor copies a tile (x_box)
  // half a tile's lines: three lines of every row pair, a multiple of 128 bytes
  static constexpr int HALF = (int)((RP * SP * sizeof(C) + 127) / 128 * 128 / sizeof(C));
  static_assert(M % 2 == 0 && T % 32 == 0, "pairs of butterflies, whole warps");
  static_assert(RP == 1 ? NO <= T : (NO + 7) / 8 * 8 <= T, "an outer stage in one pass of the threads");
  static_assert((size_t)HALF * sizeof(C) >= (size_t)3 * ((N + 1) / 3 + 15) * 2 * RP * sizeof(C), "the staging tile fits half the lines");
  static constexpr size_t smem = (size_t)2 * HALF * sizeof(C) * G + 16 * G;
};

// The twiddles of a plan: the middle stage's exp(-2 pi i p0 (j' + R2 r) / N) as
// [r][p0 + R0 j'], then the fused stage's exp(-2 pi i j p1 / (R1 R2)) as
// [j][p1]: N + R1 R2 entries.
template <int N, typename C>
static void x_twiddles_t(C* out) {
  typedef XPlan<N, C> P;
  typedef typename RealOf<C>::T T;
  const long double w = -2.0L * 3.141592653589793238462643383279502884L;
  for (int r = 0; r < P::R1; ++r)
    for (int v = 0; v < P::R0 * P::R2; ++v) {
      const long e = (long)(v % P::R0) * (v / P::R0 + P::R2 * r) % N;
      const long double a = w * (long double)e / (long double)N;
      *out++ = C{(T)cosl(a), (T)sinl(a)};
    }
  const int n = P::R1 * P::R2;
  for (int j = 0; j < P::R2; ++j)
    for (int p = 0; p < P::R1; ++p) {
      const long double a = w * (long double)((j * p) % n) / (long double)n;
      *out++ = C{(T)cosl(a), (T)sinl(a)};
    }
}

// Unit u of an outer stage: row pair sub, line c of three, butterfly pair j.
// FP32: four lanes of one row pair, then the same four of the other, so that
// the 16-byte accesses of the [mode][row] tile hit distinct banks.
template <typename X>
__device__ __forceinline__ bool outer_unit(int u, int& sub, int& c, int& j) {
  int e = u;
  sub = 0;
  if (X::RP > 1) {
    sub = (u >> 2) & 1;
    e = (u >> 3) * 4 + (u & 3);
  }
  c = e / X::H;
  j = e - c * X::H;
  return e < 3 * X::H;
}
// the two rows of a mode in the staging tile; in FP64 every other four lanes
// take the rows in reverse order, which spreads their 32-byte stride over
// distinct banks
__device__ __forceinline__ void tile_load(const double2* p, bool rev, double2& a, double2& b) {
  const double2 x = p[rev], y = p[!rev];
  a = rev ? y : x;
  b = rev ? x : y;
}
__device__ __forceinline__ void tile_load(const float2* p, bool, float2& a, float2& b) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  a = make_float2(q.x, q.y);
  b = make_float2(q.z, q.w);
}
__device__ __forceinline__ void tile_store(double2* p, bool rev, double2 a, double2 b) {
  p[rev] = rev ? b : a;
  p[!rev] = rev ? a : b;
}
__device__ __forceinline__ void tile_store(float2* p, bool, float2 a, float2 b) {
  *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
}

template <int N, int NP, typename C>
__global__ void __launch_bounds__(XPlan<N, C>::T* XPlan<N, C>::G, XPlan<N, C>::MINB)
    k_x(Geometry g, const C* __restrict__ tw, const double* __restrict__ dyl, PhysScalars ps, int want_cfl,
        unsigned long long* __restrict__ cflmax, const __grid_constant__ CUtensorMap tmZ,
        const __grid_constant__ CUtensorMap tmP, const __grid_constant__ CUtensorMap tmP2, int* __restrict__ err) {
  typedef XShape<N, C> X;
  typedef typename RealOf<C>::T T;
  constexpr int R0 = X::R0, R1 = X::R1, R2 = X::R2, M = X::M, H = X::H, S0 = X::S0, LS = X::LS, RH = X::RH;
  constexpr int TT = X::T, NU = X::NU, NV = X::NV, RP = X::RP, SP = X::SP, HALF = X::HALF, NB = X::NB;
  constexpr int MP = 2 * RP;  // elements (rows) of one mode in the staging tile
  extern __shared__ __align__(128) double2 sh_d[];
  const int warp_tile = X::G > 1 ? threadIdx.x / TT : 0;
  const int tid = X::G > 1 ? threadIdx.x % TT : threadIdx.x;
  // the lines of u, v, w (later the first three products), then those of the
  // other products; the tile comes in over the second half
  C* const sh = reinterpret_cast<C*>(sh_d) + (size_t)warp_tile * 2 * HALF;
  C* const sh1 = sh + HALF;
  uint64_t* const bar = reinterpret_cast<uint64_t*>(reinterpret_cast<C*>(sh_d) + (size_t)X::G * 2 * HALF) + 2 * warp_tile;
  const int rb = blockIdx.x * X::G + warp_tile;  // rows 2 RP rb ..
  static_assert(X::G == 1 || TT == 32, "several tiles a block: one warp each");
  if (X::G > 1 && 2 * RP * rb >= g.ny) return;  // a whole warp, which meets no block barrier
  auto sync = [] {
    if constexpr (X::G > 1)
      __syncwarp();
    else
      __syncthreads();
  };
  const int y0 = 2 * RP * rb, kz = blockIdx.y % g.nzd, mem = blockIdx.y / g.nzd;
  const int nx = g.nx, nxB = g.nxB, Ty = g.Ty;
  const int yt = y0 / Ty, yi0 = y0 - yt * Ty;
  const int BX = x_box(nxB);  // modes a tensor copy
  const int nb = NB == 1 || BX >= nxB ? 1 : 2;
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
    wait_predecessor();
    mbar_arrive_expect_tx(bar, 3u * (unsigned)(MP * sizeof(C) * nb * BX));
    for (int b = 0; b < nb; ++b)
      tma_load_4d(sh1 + b * 3 * BX * MP, &tmZ, 2 * yi0, b * BX, yt * g.nzd + kz, 3 * mem, bar);
  }
  sync();
  wait_predecessor();
  if (!mbar_wait_bounded(bar, 0, X_WAIT_LIMIT)) {
    // record the failure and give the copy a second bounded wait before the
    // block (and its shared memory) goes away
    if (tid == 0) atomicExch(err, 1);
    mbar_wait_bounded(bar, 0, X_WAIT_LIMIT);
    return;
  }
  // mode m of component c (of nc) in a staging tile
  auto slot = [&](int c, int m, int nc) -> int {
    if (NB == 1) return (c * BX + m) * MP;
    const int b = m >= BX ? 1 : 0;
    return ((b * nc + c) * BX + m - b * BX) * MP;
  };
  const bool rev = (threadIdx.x >> 2) & 1;

  // first inverse stage: butterflies j and M - j (0 and M/2 for j = 0); mode
  // m is a + i b of its two rows, mode N - m the conjugates
  {
    int sub, c, j;
    if (outer_unit<X>(tid, sub, c, j)) {
      const int jB = j ? M - j : H;
      C A[R0], B[R0], nA[RH + 1], nB[RH + 1];
#pragma unroll
      for (int r = 0; r < R0; ++r) A[r] = B[r] = C{0, 0};
#pragma unroll
      for (int r = 0; r <= RH; ++r) nA[r] = nB[r] = C{0, 0};
#pragma unroll
      for (int r = 0; r < RH; ++r) {
        const int mA = j + r * M, mB = jB + r * M;
        C a, b;
        if (mA <= nx) {
          tile_load(sh1 + slot(c, mA, 3) + 2 * sub, rev, a, b);
          A[r] = C{a.x - b.y, a.y + b.x};
          nA[r] = C{a.x + b.y, b.x - a.y};
          if (r == 0 && j == 0) A[r] = C{a.x, b.x};  // the c2r ignores the mean's imaginary part
        }
        if (mB <= nx) {
          tile_load(sh1 + slot(c, mB, 3) + 2 * sub, rev, a, b);
          B[r] = C{a.x - b.y, a.y + b.x};
          nB[r] = C{a.x + b.y, b.x - a.y};
        }
      }
#pragma unroll
      for (int r = 0; r < RH; ++r) {
        // j = 0 mirrors within each butterfly: 0's mode r M at R0 - r, M/2's at R0 - 1 - r
        A[R0 - 1 - r] = j ? nB[r] : nA[r + 1];
        B[R0 - 1 - r] = j ? nA[r] : nB[r];
      }
      DFT<R0, +1>::run(A);
      DFT<R0, +1>::run(B);
      C* const s = sh + sub * SP + c * LS;
#pragma unroll
      for (int p = 0; p < R0; ++p) {
        s[p * S0 + j] = A[p];
        s[p * S0 + jB] = B[p];
      }
    }
  }
  sync();
  // middle inverse stage
  if constexpr (R1 > 1) {
#pragma unroll 1
    for (int u = tid; u < RP * 3 * NU; u += TT) {
      const int l = u / NU, v = u - l * NU;
      const int sub = RP > 1 ? l / 3 : 0, c = l - 3 * sub;
      C* const s = sh + sub * SP + c * LS + (v % R0) * S0 + v / R0;
      C x[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) x[r] = cmul(s[r * R2], cconj(__ldg(tw + r * NU + v)));
      DFT<R1, +1>::run(x);
#pragma unroll
      for (int r = 0; r < R1; ++r) s[r * R2] = x[r];
    }
    sync();
  }
  // last inverse stage, products, first forward stage: x points v + NV r.
  // Without a middle stage (R1 = 1) the outer twiddles are applied here.
  double cm = 0.0;
  const T f = (T)ps.factor;
#pragma unroll 1
  for (int u = tid; u < RP * NV; u += TT) {
    const int sub = RP > 1 ? u / NV : 0, v = u - sub * NV;
    const int p0 = v % R0, p1 = v / R0;
    C* const s = sh + sub * SP + p0 * S0 + p1 * R2;
    C w[R2], U[3][R2];
#pragma unroll
    for (int r = 1; r < R2; ++r) w[r] = __ldg(R1 > 1 ? tw + N + r * R1 + p1 : tw + r * R0 + p0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      U[c][0] = s[c * LS];
#pragma unroll
      for (int r = 1; r < R2; ++r) U[c][r] = cmul(s[c * LS + r], cconj(w[r]));
      DFT<R2, +1>::run(U[c]);
    }
    if (want_cfl) {
      const double r0 = 1.0 / dyl[y0 + 2 * sub], r1 = 1.0 / dyl[y0 + 2 * sub + 1];
#pragma unroll
      for (int r = 0; r < R2; ++r) {
        const double c0 = fabs((double)U[0][r].x) * ps.rdx + fabs((double)U[1][r].x) * r0 + fabs((double)U[2][r].x) * ps.rdz;
        const double c1 = fabs((double)U[0][r].y) * ps.rdx + fabs((double)U[1][r].y) * r1 + fabs((double)U[2][r].y) * ps.rdz;
        cm = nan_max(cm, nan_max(c0, c1));
      }
    }
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      // NP = 6: uu, vv, ww, uv, vw, uw; NP = 5: uu - vv, ww - vv, uv, vw, uw
      constexpr int ia[2][6] = {{0, 1, 2, 0, 1, 0}, {0, 2, 0, 1, 0, 0}}, ib[2][6] = {{0, 1, 2, 1, 2, 2}, {0, 2, 1, 2, 2, 0}};
      const int i = ia[6 - NP][q], j = ib[6 - NP][q];
      C P[R2];
#pragma unroll
      for (int r = 0; r < R2; ++r) {
        // a difference of squares: in FP64 as one product, which leaves no spills
        // (601 against 687 us for 768 points, 384 z points and 128 rows); in FP32
        // as two (307 against 314 us for 384 points, 192 z points and 256 rows)
        if (NP == 5 && q < 2 && sizeof(T) == 8)
          P[r] = C{(U[i][r].x - U[1][r].x) * ((U[i][r].x + U[1][r].x) * f), (U[i][r].y - U[1][r].y) * ((U[i][r].y + U[1][r].y) * f)};
        else
          P[r] = C{U[i][r].x * (U[j][r].x * f), U[i][r].y * (U[j][r].y * f)};
        if (NP == 5 && q < 2 && sizeof(T) == 4)
          P[r] = C{P[r].x - U[1][r].x * (U[1][r].x * f), P[r].y - U[1][r].y * (U[1][r].y * f)};
      }
      DFT<R2, -1>::run(P);
      C* const o = s + (q >= 3 ? HALF + (q - 3) * LS : q * LS);
      o[0] = P[0];
#pragma unroll
      for (int r = 1; r < R2; ++r) o[r] = cmul(P[r], w[r]);
    }
  }
  if (want_cfl) {
    for (int o = 16; o > 0; o >>= 1) cm = nan_max(cm, __shfl_xor_sync(0xffffffffu, cm, o));
    // a NaN keeps its bits: as an unsigned word it exceeds every finite
    // non-negative double and infinity, so it wins the maximum and the host
    // sees a non-finite CFL number
    if ((threadIdx.x & 31) == 0) atomicMax(cflmax, (unsigned long long)__double_as_longlong(cm));
  }
  sync();
  // middle forward stage
  if constexpr (R1 > 1) {
#pragma unroll 1
    for (int u = tid; u < RP * NP * NU; u += TT) {
      const int l = u / NU, v = u - l * NU;
      const int sub = RP > 1 ? l / NP : 0, q = l - NP * sub, hf = q >= 3 ? 1 : 0, c = q - 3 * hf;
      C* const s = sh + hf * HALF + sub * SP + c * LS + (v % R0) * S0 + v / R0;
      C x[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) x[r] = s[r * R2];
      DFT<R1, -1>::run(x);
#pragma unroll
      for (int r = 0; r < R1; ++r) s[r * R2] = cmul(x[r], __ldg(tw + r * NU + v));
    }
    sync();
  }
  // last forward stage on the pairs (j, M - j), and the two rows' spectra,
  // three products at a time: the staging tile of a half goes over its lines
  // once every thread has read them
#pragma unroll 1
  for (int hf = 0; hf < 2; ++hf) {
    int sub, c, j;
    const bool on = outer_unit<X>(tid, sub, c, j) && (hf == 0 || c < NP - 3);
    const int jB = j ? M - j : H;
    C A[R0], B[R0];
    C* const half = sh + hf * HALF;
    if (on) {
      const C* const s = half + sub * SP + c * LS;
#pragma unroll
      for (int p = 0; p < R0; ++p) {
        A[p] = s[p * S0 + j];
        B[p] = s[p * S0 + jB];
      }
      DFT<R0, -1>::run(A);
      DFT<R0, -1>::run(B);
    }
    if (hf == 1) fence_proxy_async();
    sync();
    if (hf == 1 && tid == 0) {
      for (int b = 0; b < nb; ++b)
        tma_store_4d(&tmP, 2 * yi0, b * BX, yt * g.nzd + kz, 6 * mem, sh + b * 3 * BX * MP);
      bulk_commit();
    }
    if (on) {
      const T h = T(0.5);
#pragma unroll
      for (int r = 0; r < RH; ++r) {
        const int kA = j + r * M, kB = jB + r * M;
        const C mA = j ? B[R0 - 1 - r] : A[(R0 - r) % R0], mB = j ? A[R0 - 1 - r] : B[R0 - 1 - r];
        if (kA <= nx)
          tile_store(half + slot(c, kA, hf ? NP - 3 : 3) + 2 * sub, rev, C{h * (A[r].x + mA.x), h * (A[r].y - mA.y)},
                     C{h * (A[r].y + mA.y), h * (mA.x - A[r].x)});
        if (kB <= nx)
          tile_store(half + slot(c, kB, hf ? NP - 3 : 3) + 2 * sub, rev, C{h * (B[r].x + mB.x), h * (B[r].y - mB.y)},
                     C{h * (B[r].y + mB.y), h * (mB.x - B[r].x)});
      }
    }
  }
  fence_proxy_async();
  sync();
  if (tid == 0) {
    for (int b = 0; b < nb; ++b)
      tma_store_4d(NP == 6 ? &tmP : &tmP2, 2 * yi0, b * BX, yt * g.nzd + kz, 6 * mem + 3, sh1 + b * (NP - 3) * BX * MP);
    bulk_commit();
    bulk_wait_read_all();
  }
}

// ------------------------------------------------------------- dispatch ----
#define HST_X_LENGTHS64(F) F(96) F(128) F(192) F(256) F(384) F(512) F(768) F(1024) F(1536)
#define HST_X_LENGTHS32(F) F(96) F(192) F(384) F(768) F(1536)

bool x_compiled(int N, bool fp32) {
  switch (N) {
#define HST_X(n) case n:
    HST_X_LENGTHS32(HST_X) return true;
    case 128: case 256: case 512: case 1024: return !fp32;
#undef HST_X
  }
  return false;
}

static int x_row_pairs(int N, bool fp32) {
  switch (N) {
#define HST_X(n) case n: return fp32 ? XPlan<n, float2>::RP : 1;
    HST_X_LENGTHS32(HST_X)
#undef HST_X
  }
  return 1;
}

int x_twiddles(int N, double2* out) {
  switch (N) {
#define HST_X(n) \
  case n: x_twiddles_t<n, double2>(out); return n + XPlan<n, double2>::R1 * XPlan<n, double2>::R2;
    HST_X_LENGTHS64(HST_X)
#undef HST_X
  }
  return 0;
}
int x_twiddles(int N, float2* out) {
  switch (N) {
#define HST_X(n) \
  case n: x_twiddles_t<n, float2>(out); return n + XPlan<n, float2>::R1 * XPlan<n, float2>::R2;
    HST_X_LENGTHS32(HST_X)
#undef HST_X
  }
  return 0;
}

// ------------------------------------------------------------- TMA maps ----
// Z and Pp seen as 4-D real tensors: d0 = the 2 Ty reals of one y tile
// (innermost), d1 = ix, d2 = (y tile, kz) as yt nzd + kz, d3 = component.
// The box is {the rows of a tile, modes, 1, three components (two: the second
// half of five products)}.
EncodeTiled encode_tiled() {
  static const EncodeTiled enc = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiled>(fn) : nullptr;
  }();
  return enc;
}

static cudaError_t encode_map(EncodeTiled enc, const Geometry& g, void* base, int comps, int box_comps, int Ty, int nyT,
                              int rp, CUtensorMap* map) {
  const cuuint64_t es = g.mp ? 8 : 16;  // bytes of one complex element
  cuuint64_t dims[4] = {(cuuint64_t)2 * Ty, (cuuint64_t)g.nxB, (cuuint64_t)g.nzd * nyT, (cuuint64_t)comps * g.nmem};
  cuuint64_t strides[3] = {es * Ty, es * Ty * g.nxB, es * Ty * g.nxB * g.nzd * nyT};
  cuuint32_t box[4] = {(cuuint32_t)(4 * rp), (cuuint32_t)x_box(g.nxB), 1, (cuuint32_t)box_comps};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(map, g.mp ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, base, dims,
                         strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t make_x_maps(const Geometry& g, DeviceState& d) {
  if (!x_compiled(2 * g.nxd, g.mp != 0)) return cudaSuccess;
  const EncodeTiled enc = encode_tiled();
  if (!enc) return cudaErrorNotSupported;
  const int rp = x_row_pairs(2 * g.nxd, g.mp != 0);
  cudaError_t e = encode_map(enc, g, d.Z, 3, 3, g.Ty, g.nyT, rp, &d.tmZ);
  if (e == cudaSuccess) e = encode_map(enc, g, d.Pp, 6, 3, g.Ty, g.nyT, rp, &d.tmPp);
  if (e == cudaSuccess) e = encode_map(enc, g, d.Pp, 6, 2, g.Ty, g.nyT, rp, &d.tmPp2);
  if (e == cudaSuccess && d.Zg) {  // the ghost rows' buffers: one tile
    e = encode_map(enc, g, d.Zg, 3, 3, g.EY, 1, rp, &d.tmZg);
    if (e == cudaSuccess) e = encode_map(enc, g, d.Ppg, 6, 3, g.EY, 1, rp, &d.tmPpg);
    if (e == cudaSuccess) e = encode_map(enc, g, d.Ppg, 6, 2, g.EY, 1, rp, &d.tmPpg2);
  }
  return e;
}

template <int N, int NP, typename C>
static cudaError_t launch_x_t(const Geometry& g, const DeviceState& d, const PhysScalars& ps, int want_cfl,
                              const C* tw, cudaStream_t st) {
  typedef XShape<N, C> X;
  if (g.Ty % (2 * X::RP) != 0) return cudaErrorInvalidValue;
  smem_limit(d, k_x<N, NP, C>, (int)X::smem);
  const int nt = g.ny / (2 * X::RP);
  const dim3 grid((nt + X::G - 1) / X::G, g.nzd * g.nmem);
  return launch_after(k_x<N, NP, C>, grid, X::T * X::G, X::smem, st, g, tw + N, d.dyl, ps, want_cfl, d.cfl, d.tmZ, d.tmPp, d.tmPp2, d.err);
}

cudaError_t launch_x(const Geometry& g, const DeviceState& d, const PhysScalars& ps, int want_cfl, int np,
                     cudaStream_t st) {
  if (g.mp) {
    switch (2 * g.nxd) {
#define HST_X(n) \
  case n:    \
    return np == 5 ? launch_x_t<n, 5, float2>(g, d, ps, want_cfl, d.twxf, st)    \
                   : launch_x_t<n, 6, float2>(g, d, ps, want_cfl, d.twxf, st);
      HST_X_LENGTHS32(HST_X)
#undef HST_X
    }
    return cudaErrorInvalidValue;
  }
  switch (2 * g.nxd) {
#define HST_X(n) \
  case n:    \
    return np == 5 ? launch_x_t<n, 5, double2>(g, d, ps, want_cfl, d.twx, st)    \
                   : launch_x_t<n, 6, double2>(g, d, ps, want_cfl, d.twx, st);
    HST_X_LENGTHS64(HST_X)
#undef HST_X
  }
  return cudaErrorInvalidValue;
}

}  // namespace hst
