// The register DFTs of the 3/2-dealiased x and z transforms (radices up to 24,
// built from radix-2/3/4 pieces), and a Stockham FFT for the lengths without a
// plan of their own in hst_xprod.cu and hst_z.cu: 12, 24, 48 and 64 known to the
// compiler, the others with a runtime plan.
//
// A block transforms nl lines of length N = 2^a 3^b.  Each
// radix-R stage is one pass: a thread gathers the R inputs of its butterflies
// into registers, applies the stage twiddles, computes a radix-R DFT in
// registers, and scatters the outputs.  The first stage reads through a
// caller's loader (global memory, or a function of other lines) and the last
// stage writes through a caller's storer, so only the exchanges between
// stages go through shared memory.  Threads are mapped line-fastest so that
// global accesses of consecutive threads touch consecutive lines (the y rows,
// contiguous in memory).  Stage twiddles come from W[e] = exp(-2 pi i e / N) in
// global memory (computed on the host in extended precision), the twiddles
// inside a register DFT from a 48-entry table in constant memory (all threads
// read the same entry).  Unnormalised both ways, like the reference's FFTW
// and cuFFT plans (src/hst_fft.f90:98-121): S = -1 forward, S = +1 backward.
#pragma once
#include <type_traits>

#include "hst_dev.cuh"

namespace hst {

#define HST_SQRT3_2 0.86602540378443864676

// exp(-2 pi i k / 48), k = 0..47, rounded from extended precision (one copy
// in the constant memory of each translation unit that includes this header)
static __constant__ double2 c_w48[48] = {
    {1.0, 0.0}, {0.9914448613738104, -0.1305261922200516},
    {0.9659258262890683, -0.25881904510252074}, {0.9238795325112867, -0.3826834323650898},
    {0.8660254037844386, -0.5}, {0.7933533402912352, -0.6087614290087207},
    {0.7071067811865476, -0.7071067811865476}, {0.6087614290087207, -0.7933533402912352},
    {0.5, -0.8660254037844386}, {0.3826834323650898, -0.9238795325112867},
    {0.25881904510252074, -0.9659258262890683}, {0.1305261922200516, -0.9914448613738104},
    {0.0, -1.0}, {-0.1305261922200516, -0.9914448613738104},
    {-0.25881904510252074, -0.9659258262890683}, {-0.3826834323650898, -0.9238795325112867},
    {-0.5, -0.8660254037844386}, {-0.6087614290087207, -0.7933533402912352},
    {-0.7071067811865476, -0.7071067811865476}, {-0.7933533402912352, -0.6087614290087207},
    {-0.8660254037844386, -0.5}, {-0.9238795325112867, -0.3826834323650898},
    {-0.9659258262890683, -0.25881904510252074}, {-0.9914448613738104, -0.1305261922200516},
    {-1.0, 0.0}, {-0.9914448613738104, 0.1305261922200516},
    {-0.9659258262890683, 0.25881904510252074}, {-0.9238795325112867, 0.3826834323650898},
    {-0.8660254037844386, 0.5}, {-0.7933533402912352, 0.6087614290087207},
    {-0.7071067811865476, 0.7071067811865476}, {-0.6087614290087207, 0.7933533402912352},
    {-0.5, 0.8660254037844386}, {-0.3826834323650898, 0.9238795325112867},
    {-0.25881904510252074, 0.9659258262890683}, {-0.1305261922200516, 0.9914448613738104},
    {0.0, 1.0}, {0.1305261922200516, 0.9914448613738104},
    {0.25881904510252074, 0.9659258262890683}, {0.3826834323650898, 0.9238795325112867},
    {0.5, 0.8660254037844386}, {0.6087614290087207, 0.7933533402912352},
    {0.7071067811865476, 0.7071067811865476}, {0.7933533402912352, 0.6087614290087207},
    {0.8660254037844386, 0.5}, {0.9238795325112867, 0.3826834323650898},
    {0.9659258262890683, 0.25881904510252074}, {0.9914448613738104, 0.1305261922200516}};
static __constant__ float2 c_w48f[48] = {
    {1.0f, 0.0f}, {0.991444886f, -0.130526185f}, {0.965925813f, -0.258819044f}, {0.923879504f, -0.382683426f},
    {0.866025388f, -0.5f}, {0.793353319f, -0.60876143f}, {0.707106769f, -0.707106769f}, {0.60876143f, -0.793353319f},
    {0.5f, -0.866025388f}, {0.382683426f, -0.923879504f}, {0.258819044f, -0.965925813f}, {0.130526185f, -0.991444886f},
    {0.0f, -1.0f}, {-0.130526185f, -0.991444886f}, {-0.258819044f, -0.965925813f}, {-0.382683426f, -0.923879504f},
    {-0.5f, -0.866025388f}, {-0.60876143f, -0.793353319f}, {-0.707106769f, -0.707106769f}, {-0.793353319f, -0.60876143f},
    {-0.866025388f, -0.5f}, {-0.923879504f, -0.382683426f}, {-0.965925813f, -0.258819044f}, {-0.991444886f, -0.130526185f},
    {-1.0f, 0.0f}, {-0.991444886f, 0.130526185f}, {-0.965925813f, 0.258819044f}, {-0.923879504f, 0.382683426f},
    {-0.866025388f, 0.5f}, {-0.793353319f, 0.60876143f}, {-0.707106769f, 0.707106769f}, {-0.60876143f, 0.793353319f},
    {-0.5f, 0.866025388f}, {-0.382683426f, 0.923879504f}, {-0.258819044f, 0.965925813f}, {-0.130526185f, 0.991444886f},
    {0.0f, 1.0f}, {0.130526185f, 0.991444886f}, {0.258819044f, 0.965925813f}, {0.382683426f, 0.923879504f},
    {0.5f, 0.866025388f}, {0.60876143f, 0.793353319f}, {0.707106769f, 0.707106769f}, {0.793353319f, 0.60876143f},
    {0.866025388f, 0.5f}, {0.923879504f, 0.382683426f}, {0.965925813f, 0.258819044f}, {0.991444886f, 0.130526185f}};
template <typename C>
__device__ __forceinline__ C w48(int i);
template <>
__device__ __forceinline__ double2 w48<double2>(int i) { return c_w48[i]; }
template <>
__device__ __forceinline__ float2 w48<float2>(int i) { return c_w48f[i]; }

// t exp(S 2 pi i e / 48), e known at compile time: quarter turns are free and
// odd eighths take two multiplications
template <int S, typename C>
__device__ __forceinline__ C mul_w48(C t, int e) {
  typedef typename RealOf<C>::T T;
  if (e == 0) return t;
  if (e == 12) return S < 0 ? C{t.y, -t.x} : C{-t.y, t.x};
  if (e == 24) return C{-t.x, -t.y};
  if (e == 36) return S < 0 ? C{-t.y, t.x} : C{t.y, -t.x};
  if (e % 6 == 0) {
    const T h = T(0.70710678118654752440);
    const T p = h * (t.x + t.y), m = h * (t.y - t.x);
    const int q = e / 6;  // exp(-i pi q / 4) = (+-1 -+ i) / sqrt 2
    if (S < 0) return q == 1 ? C{p, m} : (q == 3 ? C{m, -p} : (q == 5 ? C{-p, -m} : C{-m, p}));
    return q == 1 ? C{-m, p} : (q == 3 ? C{-p, -m} : (q == 5 ? C{m, -p} : C{p, m}));
  }
  C w = w48<C>(e);
  if (S > 0) w.y = -w.y;
  return cmul(t, w);
}

template <int R, int S>
struct DFT;

template <int S>
struct DFT<2, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) {
    C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};
template <int S>
struct DFT<4, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) {
    C a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]), a2 = cadd(v[1], v[3]), a3 = csub(v[1], v[3]);
    C a3r = S < 0 ? C{a3.y, -a3.x} : C{-a3.y, a3.x};
    v[0] = cadd(a0, a2);
    v[2] = csub(a0, a2);
    v[1] = cadd(a1, a3r);
    v[3] = csub(a1, a3r);
  }
};
template <int S>
struct DFT<3, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) {
    typedef typename RealOf<C>::T T;
    const T h = T(0.5), q = T(HST_SQRT3_2);
    C t1 = cadd(v[1], v[2]), t2 = csub(v[1], v[2]);
    C m = C{v[0].x - h * t1.x, v[0].y - h * t1.y};
    C r = S < 0 ? C{q * t2.y, -q * t2.x} : C{-q * t2.y, q * t2.x};
    v[0] = cadd(v[0], t1);
    v[1] = cadd(m, r);
    v[2] = csub(m, r);
  }
};
// R = A B: B DFTs of size A on the elements b + B a, the twiddles
// W_R^(b ka), A DFTs of size B; output k = ka + A kb.
template <int A, int B, int S, typename C>
__device__ __forceinline__ void dft_ab(C* v) {
  C o[A * B];
#pragma unroll
  for (int b = 0; b < B; ++b) {
    C t[A];
#pragma unroll
    for (int a = 0; a < A; ++a) t[a] = v[b + B * a];
    DFT<A, S>::run(t);
#pragma unroll
    for (int ka = 0; ka < A; ++ka) {
      v[b + B * ka] = mul_w48<S>(t[ka], (b * ka * (48 / (A * B))) % 48);
    }
  }
#pragma unroll
  for (int ka = 0; ka < A; ++ka) {
    C t[B];
#pragma unroll
    for (int b = 0; b < B; ++b) t[b] = v[b + B * ka];
    DFT<B, S>::run(t);
#pragma unroll
    for (int kb = 0; kb < B; ++kb) o[ka + A * kb] = t[kb];
  }
#pragma unroll
  for (int k = 0; k < A * B; ++k) v[k] = o[k];
}
template <int S>
struct DFT<6, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) { dft_ab<3, 2, S>(v); }
};
template <int S>
struct DFT<8, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) { dft_ab<4, 2, S>(v); }
};
template <int S>
struct DFT<12, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) { dft_ab<4, 3, S>(v); }
};
template <int S>
struct DFT<16, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) { dft_ab<4, 4, S>(v); }
};
template <int S>
struct DFT<24, S> {
  template <typename C>
  static __device__ __forceinline__ void run(C* v) { dft_ab<8, 3, S>(v); }
};

// The runtime radix plan of N: radix-16 stages while more than 24 is left,
// then the rest in one stage (2, 3, 4, 6, 8, 12, 16 or 24).
struct FftPlan {
  int n;
  int r[4];
};
__host__ __device__ constexpr FftPlan make_plan(int N) {
  FftPlan p = {0, {0, 0, 0, 0}};
  int m = N;
  while (m > 24 && m % 16 == 0 && p.n < 3) {
    p.r[p.n++] = 16;
    m /= 16;
  }
  if (m > 1) p.r[p.n++] = m;
  return p;
}
__host__ inline bool plan_ok(int N) {
  FftPlan p = make_plan(N);
  int prod = 1;
  for (int i = 0; i < p.n; ++i) {
    int r = p.r[i];
    if (!(r == 2 || r == 3 || r == 4 || r == 6 || r == 8 || r == 12 || r == 16 || r == 24)) return false;
    prod *= r;
  }
  return prod == N;
}

// Shared-memory line access (line stride LS)
template <typename C>
struct ShLinesT {
  C* p;
  int LS;
  __device__ __forceinline__ C operator()(int l, int i) const { return p[l * LS + i]; }
  __device__ __forceinline__ void operator()(int l, int i, C v) const { p[l * LS + i] = v; }
};
// One radix-R stage.  Butterfly b of the block: line l = b % nl, index
// j = b / nl.  Inputs ld(l, j + r N/R), outputs st(l, (j/Ns) Ns R + j%Ns + r Ns).
// SYNC: the stage reads and writes the same shared lines (all reads, then
// a barrier, then all writes).
template <int R, int S, int PPT, bool SYNC, typename LD, typename ST, typename C = cxd>
__device__ __forceinline__ void fft_stage_io(int N, int nl, int Ns, const C* __restrict__ tw, const LD& ld,
                                             const ST& st) {
  constexpr int MAXB = (PPT + R - 1) / R;
  const int nb = N / R;
  const int total = nb * nl;
  const int tstride = N / (Ns * R);
  C v[MAXB][R];
  int lj[MAXB];
#pragma unroll
  for (int k = 0; k < MAXB; ++k) {
    int b = threadIdx.x + k * blockDim.x;
    lj[k] = -1;
    if (b < total) {
      int l = b % nl, j = b / nl;
      int kk = j % Ns;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        C x = ld(l, j + r * nb);
        if (r > 0 && kk > 0) {
          C w = __ldg(tw + kk * r * tstride);
          if (S > 0) w.y = -w.y;
          x = cmul(x, w);
        }
        v[k][r] = x;
      }
      DFT<R, S>::run(v[k]);
      lj[k] = b;
    }
  }
  if (SYNC) __syncthreads();
#pragma unroll
  for (int k = 0; k < MAXB; ++k) {
    if (lj[k] >= 0) {
      int l = lj[k] % nl, j = lj[k] / nl;
      int kk = j % Ns;
      int base = (j / Ns) * Ns * R + kk;
#pragma unroll
      for (int r = 0; r < R; ++r) st(l, base + r * Ns, v[k][r]);
    }
  }
}

template <int S, int PPT, bool SYNC, typename LD, typename ST, typename C>
__device__ __forceinline__ void fft_stage_r(int R, int N, int nl, int Ns, const C* __restrict__ tw, const LD& ld,
                                            const ST& st) {
  switch (R) {
    case 2: fft_stage_io<2, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    case 3: fft_stage_io<3, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    case 4: fft_stage_io<4, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    case 6: fft_stage_io<6, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    case 8: fft_stage_io<8, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    case 12: fft_stage_io<12, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    case 16: fft_stage_io<16, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    case 24: fft_stage_io<24, S, PPT, SYNC>(N, nl, Ns, tw, ld, st); break;
    default: break;
  }
}

// The whole transform of nl lines: the first stage reads through src, the
// last writes through dst, the stages between exchange through `sh` (nl lines
// of stride N+1).  SRC_SH / DST_SH: src reads, dst writes the same shared
// buffer (the stage then synchronises between its reads and its writes).
// NT: the length, with its one or two radices known to the compiler; 0: the
// plan of the runtime length N.  Requires nl N <= PPT blockDim.x.
template <int NT, int S, int PPT, bool SRC_SH, bool DST_SH, typename LD, typename ST, typename C>
__device__ void fft_global(int N, int nl, const C* __restrict__ tw, C* sh, const LD& src, const ST& dst) {
  if constexpr (NT > 0) {
    constexpr FftPlan P = make_plan(NT);
    static_assert(P.n <= 2, "short lengths");
    if constexpr (P.n == 1) {
      fft_stage_io<P.r[0], S, PPT, SRC_SH && DST_SH>(NT, nl, 1, tw, src, dst);
    } else {
      const ShLinesT<C> L = {sh, NT + 1};
      fft_stage_io<P.r[0], S, PPT, SRC_SH>(NT, nl, 1, tw, src, L);
      __syncthreads();
      fft_stage_io<P.r[1], S, PPT, DST_SH>(NT, nl, P.r[0], tw, L, dst);
    }
  } else {
    const FftPlan P = make_plan(N);
    const ShLinesT<C> L = {sh, N + 1};
    int Ns = 1;
    if (P.n == 1) {
      fft_stage_r<S, PPT, SRC_SH && DST_SH>(P.r[0], N, nl, Ns, tw, src, dst);
      return;
    }
    fft_stage_r<S, PPT, SRC_SH>(P.r[0], N, nl, Ns, tw, src, L);
    Ns *= P.r[0];
    __syncthreads();
    for (int s = 1; s + 1 < P.n; ++s) {
      fft_stage_r<S, PPT, true>(P.r[s], N, nl, Ns, tw, L, L);
      Ns *= P.r[s];
      __syncthreads();
    }
    fft_stage_r<S, PPT, DST_SH>(P.r[P.n - 1], N, nl, Ns, tw, L, dst);
  }
}

}  // namespace hst
