// The z transforms of the hst substep for the compiled lengths:
//
//   k_z_inv  V (u, v, w) -> zero-padded z-inverse transform (Z): assemble_vvdz
//            + IFT (src/hst_transforms.f90:33-54, src/hst_fft.f90:195-207)
//   k_z_fwd  Pp -> z-forward transform truncated to the 2nz+1 modes (Q):
//            transpose_xTOz + FFT (src/hst_transforms.f90:135-139,
//            src/hst_fft.f90:181-193)
//
// Other lengths run k_zinv and k_zfwd (hst_transforms.cu).
//
// One tile is TY rows of one x mode of one component, all N z points, in
// shared memory as [z][row].  N = R0 R1 R2 in three register stages in place
// (decimation in frequency); lanes run over the rows first, so that an access
// of a warp is whole runs of the [z][row] tile, free of bank conflicts where
// a run fills 128 bytes or R2 is odd.
//
// The forward transform waits on its loads (64-byte runs 16 KB apart at
// 768^2 x 512), so it runs on a persistent grid whose tiles land by tensor copies
// in one of NBUF buffers while the previous tile is transformed: 4.66 -> 2.80
// ms a substep at 768^2 x 512 FP64 (five products; 3.28 for six), 3.16 -> 1.58 FP32;
// 0.490 -> 0.357 and 0.302 -> 0.215 ms at 384^2 x 256.  It reads and writes 74 %
// of what a copy could in that time at 768 points.
//
// The inverse one hides its loads of V (16-byte rows, runs of TY) behind other
// blocks' arithmetic, so all R0 loads of a butterfly are issued before the
// first is converted, and its radices keep the registers low enough for a
// full SM of blocks where that is faster: FP32 768 points 8 x 12 x 8 and 12 x 8 x 8
// 620 and 611 us against 636 with the forward kernel's 16 x 16 x 3 (961 with each
// value converted as it is loaded); 384 points 8 x 12 x 4 159 us against 224
// (226); FP64 384 points 8 x 8 x 6 216 against 220 (232); FP64 768 points stays at
// 16 x 16 x 3 (504; 529 before; 616 with 12 x 8 x 8, which spills).
#include <algorithm>

#include "hst_dev.cuh"
#include "hst_fft.cuh"
#include "hst_internal.h"

namespace hst {

// The plan of length N: the forward kernel's radices; rows a tile; threads a
// block, buffers and resident blocks of the forward kernel; radices, threads
// and resident blocks of the inverse one.
template <int N, typename C>
struct ZPlan;
#define HST_ZPLAN(N_, C_, r0, r1, r2, ty, tf, nb, mbf, i0, i1, i2, ti, mbi)          \
  template <>                                                                        \
  struct ZPlan<N_, C_> {                                                             \
    static constexpr int R0 = r0, R1 = r1, R2 = r2, TY = ty, NBUF = nb;              \
    static constexpr int TF = tf, MBF = mbf;                                         \
    static constexpr int I0 = i0, I1 = i1, I2 = i2, TI = ti, MBI = mbi;              \
  };
HST_ZPLAN(48, double2, 4, 4, 3, 8, 96, 2, 8, 4, 4, 3, 96, 8)
HST_ZPLAN(64, double2, 4, 4, 4, 8, 128, 2, 6, 4, 4, 4, 128, 6)
HST_ZPLAN(96, double2, 8, 4, 3, 8, 96, 2, 6, 8, 4, 3, 96, 8)
HST_ZPLAN(128, double2, 8, 4, 4, 8, 128, 2, 5, 8, 4, 4, 128, 5)
HST_ZPLAN(192, double2, 8, 8, 3, 8, 192, 2, 4, 8, 8, 3, 192, 4)
HST_ZPLAN(256, double2, 8, 8, 4, 8, 256, 2, 3, 8, 8, 4, 256, 3)
HST_ZPLAN(384, double2, 16, 8, 3, 8, 192, 2, 2, 8, 8, 6, 192, 4)
HST_ZPLAN(512, double2, 8, 8, 8, 4, 256, 2, 3, 8, 8, 8, 128, 4)
HST_ZPLAN(768, double2, 16, 16, 3, 4, 192, 2, 2, 16, 16, 3, 192, 2)
HST_ZPLAN(1024, double2, 16, 16, 4, 4, 256, 1, 2, 16, 16, 4, 256, 2)
HST_ZPLAN(1536, double2, 16, 16, 6, 4, 384, 2, 1, 16, 16, 6, 192, 2)
HST_ZPLAN(96, float2, 8, 4, 3, 8, 96, 2, 8, 8, 4, 3, 96, 8)
HST_ZPLAN(192, float2, 8, 8, 3, 8, 192, 2, 4, 8, 8, 3, 192, 5)
HST_ZPLAN(384, float2, 16, 8, 3, 8, 192, 2, 4, 8, 12, 4, 192, 6)
HST_ZPLAN(768, float2, 16, 16, 3, 8, 384, 2, 2, 12, 8, 8, 256, 4)
HST_ZPLAN(1536, float2, 16, 16, 6, 4, 384, 2, 2, 16, 16, 6, 192, 4)
#undef HST_ZPLAN

#define HST_Z_LENGTHS64(F) F(48) F(64) F(96) F(128) F(192) F(256) F(384) F(512) F(768) F(1024) F(1536)
#define HST_Z_LENGTHS32(F) F(96) F(192) F(384) F(768) F(1536)

constexpr int Z_WAIT_LIMIT = 1 << 22;  // polls of a tile's TMA barrier before giving up

template <int N, typename C, bool INV = false>
struct ZShape {
  typedef ZPlan<N, C> P;
  static constexpr int R0 = INV ? P::I0 : P::R0, R1 = INV ? P::I1 : P::R1, R2 = INV ? P::I2 : P::R2, TY = P::TY;
  static_assert(R0 * R1 * R2 == N, "the radices multiply to N");
  static constexpr int M = N / R0;                     // butterflies of the first stage a row
  static constexpr int KB = N <= 256 ? N : (N % 256 == 0 ? 256 : 192);  // z points of one tensor copy
  static_assert(N % KB == 0 && KB * TY * sizeof(C) % 128 == 0, "whole copies, aligned in shared memory");
  static constexpr size_t tile = (size_t)N * TY * sizeof(C);
};
template <int N, typename C>
constexpr size_t z_fwd_smem() {
  return ZPlan<N, C>::NBUF * ZShape<N, C>::tile + 16;
}

// the twiddles W_N^(j p) as [p][j], j < M, p < R0 (p = 0 left out), then those
// of the middle stage W_M^(j' p) as [p][j'], j' < R2, p < R1: N - R2 entries
template <int N, typename C, bool INV>
static void z_table(C* o) {
  typedef ZShape<N, C, INV> S;
  typedef typename RealOf<C>::T T;
  const long double w = -2.0L * 3.141592653589793238462643383279502884L;
  auto put = [&](long e, int n) {
    const long double a = w * (long double)(e % n) / (long double)n;
    *o++ = C{(T)cosl(a), (T)sinl(a)};
  };
  for (int p = 1; p < S::R0; ++p)
    for (int j = 0; j < S::M; ++j) put((long)j * p, N);
  for (int p = 1; p < S::R1; ++p)
    for (int j = 0; j < S::R2; ++j) put((long)j * p, S::M);
}
// the forward table, then (N entries on) the inverse one
template <int N, typename C>
static int z_twiddles_t(C* out) {
  z_table<N, C, false>(out);
  z_table<N, C, true>(out + N);
  return 2 * N;
}

// the first two stages on one tile; LD(k, l) gives z point k of row l, all R0
// of a butterfly loaded before the first is converted to the transform's type
// (PAD: zero between N / 3 and 2 N / 3, where nothing is loaded)
template <int N, int S, int T, bool PAD, typename C, typename LD>
__device__ __forceinline__ void z_stages(C* __restrict__ sh, const C* __restrict__ tw, const LD& ld) {
  typedef typename RealOf<C>::T R;
  typedef ZShape<N, C, (S > 0)> Z;
  constexpr int R0 = Z::R0, R1 = Z::R1, R2 = Z::R2, M = Z::M, TY = Z::TY;
#pragma unroll 1
  for (int u = threadIdx.x; u < TY * M; u += T) {
    const int l = u % TY, j = u / TY;
    decltype(ld(0, 0)) v[R0];
#pragma unroll
    for (int r = 0; r < R0; ++r)
      if (!(PAD && r * M > N / 3 && (r + 1) * M <= N - N / 3)) v[r] = ld(j + r * M, l);
      else v[r] = {0, 0};
    C x[R0];
#pragma unroll
    for (int r = 0; r < R0; ++r) x[r] = C{(R)v[r].x, (R)v[r].y};
    DFT<R0, S>::run(x);
    sh[j * TY + l] = x[0];
#pragma unroll
    for (int p = 1; p < R0; ++p) {
      C w = __ldg(tw + (p - 1) * M + j);
      if (S > 0) w.y = -w.y;
      sh[(j + p * M) * TY + l] = cmul(x[p], w);
    }
  }
  __syncthreads();
  const C* const tw2 = tw + (R0 - 1) * M;
#pragma unroll 1
  for (int u = threadIdx.x; u < TY * R0 * R2; u += T) {
    const int l = u % TY, v = u / TY, jp = v % R2, p0 = v / R2;
    C* const s = sh + (p0 * M + jp) * TY + l;
    C x[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) x[r] = s[r * R2 * TY];
    DFT<R1, S>::run(x);
    s[0] = x[0];
#pragma unroll
    for (int p = 1; p < R1; ++p) {
      C w = __ldg(tw2 + (p - 1) * R2 + jp);
      if (S > 0) w.y = -w.y;
      s[p * R2 * TY] = cmul(x[p], w);
    }
  }
  __syncthreads();
}
// the last stage: ST(k, l, value) takes output k of row l
template <int N, int S, int T, typename C, typename ST>
__device__ __forceinline__ void z_last(const C* __restrict__ sh, const ST& st) {
  typedef ZShape<N, C, (S > 0)> Z;
  constexpr int R0 = Z::R0, R1 = Z::R1, R2 = Z::R2, TY = Z::TY;
#pragma unroll 2
  for (int u = threadIdx.x; u < TY * R0 * R1; u += T) {
    const int l = u % TY, v = u / TY, p1 = v % R1, p0 = v / R1;
    const C* const s = sh + v * R2 * TY + l;
    C x[R2];
#pragma unroll
    for (int r = 0; r < R2; ++r) x[r] = s[r * TY];
    DFT<R2, S>::run(x);
#pragma unroll
    for (int r = 0; r < R2; ++r) st(p0 + R0 * p1 + R0 * R1 * r, l, x[r]);
  }
}

// ------------------------------------------------------------- inverse ----
// x modes that run side by side
template <int N, typename C>
__host__ __device__ __forceinline__ int z_inv_group(int nxB) {
  return sizeof(C) == 8 ? 4 : nxB;
}
// V row of tile row i: row i of the field, or (edge view: gap = ny) rows -2,
// -1, ny, ny + 1
template <int N, typename C>
__global__ void __launch_bounds__(ZPlan<N, C>::TI, ZPlan<N, C>::MBI)
    k_z_inv(Geometry g, const double2* V0, const double2* V1, const double2* V2, C* Zo, const C* __restrict__ tw) {
  typedef ZShape<N, C> Z;
  typedef typename RealOf<C>::T T;
  constexpr int TY = Z::TY;
  extern __shared__ __align__(128) double2 sh_d[];
  C* const sh = reinterpret_cast<C*>(sh_d);
  // FP64: the x modes of one y tile run side by side, so that consecutive
  // blocks write adjacent runs of the [yt][kz][ix][Ty] tiles (768 points, 64 x
  // modes, 512 rows: 504 us; 588 in the order below).  FP32, whose runs of V are
  // twice as long as those it writes: four x modes and then the y tiles, whose
  // runs of V adjoin (768 points, 128 x modes, 512 rows: 636 us against 723 in
  // the order above; 1536^2 x 128 2.07 against 2.45 ms).
  const int nyT = (g.ny + TY - 1) / TY, nz = g.nz, grp = z_inv_group<N, C>(g.nxB);
  const int bg = blockIdx.x / grp, ix = bg / nyT * grp + blockIdx.x % grp, yt = bg % nyT;
  const int c = blockIdx.y % 3, mem = blockIdx.y / 3;
  if (ix >= g.nxB) return;
  const int y0 = yt * TY;
  const double2* const V = (c == 0 ? V0 : (c == 1 ? V1 : V2)) + (size_t)mem * g.nf + (size_t)ix * g.nzT * g.rows +
                           (g.edge_gap ? 0 : 2) + y0;
  auto ld = [&](int k, int l) -> double2 {
    const int iz = k <= nz ? k : k - N;
    double2 v = mkc(0, 0);
    if (iz >= -nz && y0 + l < g.ny) v = load_field(V + (size_t)(iz + nz) * g.rows + l + (l >= 2 ? g.edge_gap : 0));
    return v;
  };
  wait_predecessor();
  z_stages<N, +1, ZPlan<N, C>::TI, true>(sh, tw, ld);
  const size_t zs = (size_t)g.nxB * TY;
  C* const o = Zo + ((((size_t)mem * 3 + c) * nyT + yt) * N) * zs + (size_t)ix * TY;
  z_last<N, +1, ZPlan<N, C>::TI>(sh, [&](int k, int l, C v) { o[(size_t)k * zs + l] = v; });
}

// ------------------------------------------------------------- forward ----
template <int N, typename C>
__global__ void __launch_bounds__(ZPlan<N, C>::TF, ZPlan<N, C>::MBF)
    k_z_fwd(Geometry g, int np, C* __restrict__ Q, const C* __restrict__ tw, const __grid_constant__ CUtensorMap tmP,
            int* __restrict__ err) {
  typedef ZShape<N, C> Z;
  constexpr int TY = Z::TY, KB = Z::KB, NBUF = ZPlan<N, C>::NBUF;
  extern __shared__ __align__(128) double2 sh_d[];
  C* const sh = reinterpret_cast<C*>(sh_d);
  uint64_t* const bar = reinterpret_cast<uint64_t*>(sh + (size_t)NBUF * N * TY);
  const int nyT = (g.ny + TY - 1) / TY, nz = g.nz, nxP = (g.nxB + 3) / 4 * 4;
  const int ntile = nyT * nxP * np * g.nmem;
  // tile t: four x modes of one y tile side by side (whole 256-byte runs of
  // Pp), then the y tiles, then the next four x modes
  struct Tile {
    int ix, yt, pm;
  };
  auto tile_of = [&](int t) -> Tile {
    // pm: the product's component among the six of every member
    const int per = nyT * nxP, k = t / per, e = t - k * per, q = e >> 2;
    return Tile{(q / nyT) * 4 + (e & 3), q % nyT, k / np * 6 + k % np};
  };
  auto next = [&](int t) {  // the first tile from t on whose x mode exists
    while (t < ntile && tile_of(t).ix >= g.nxB) t += gridDim.x;
    return t;
  };
  auto issue = [&](int t, int b) {
    const Tile q = tile_of(t);
    mbar_arrive_expect_tx(&bar[b], (unsigned)Z::tile);
#pragma unroll 1
    for (int k = 0; k < N; k += KB)
      tma_load_4d(sh + ((size_t)b * N + k) * TY, &tmP, 0, q.ix, q.yt * N + k, q.pm, &bar[b]);
  };
  if (threadIdx.x == 0) {
    for (int b = 0; b < NBUF; ++b) mbar_init(&bar[b], 1);
    fence_mbar_init();
  }
  __syncthreads();
  wait_predecessor();
  int t = next(blockIdx.x), tn = t;  // this tile, the next one to fetch
  if (threadIdx.x == 0)
    for (int b = 0; b < NBUF && tn < ntile; ++b) {
      issue(tn, b);
      tn = next(tn + gridDim.x);
    }
  for (int i = 0; t < ntile; ++i, t = next(t + gridDim.x)) {
    const int b = NBUF > 1 ? i & 1 : 0;
    const unsigned parity = (NBUF > 1 ? i >> 1 : i) & 1;
    if (!mbar_wait_bounded(&bar[b], parity, Z_WAIT_LIMIT)) {
      // record the failure, give the copies in flight a second bounded wait
      // to land, and leave
      if (threadIdx.x == 0) atomicExch(err, 1);
      mbar_wait_bounded(&bar[b], parity, Z_WAIT_LIMIT);
      if (NBUF > 1) mbar_wait_bounded(&bar[b ^ 1], ((i + 1) >> 1) & 1, Z_WAIT_LIMIT);
      return;
    }
    C* const s = sh + (size_t)b * N * TY;
    z_stages<N, -1, ZPlan<N, C>::TF, false>(s, tw, [&](int k, int l) { return s[k * TY + l]; });
    const Tile q = tile_of(t);
    const int y0 = q.yt * TY;
    C* const o = Q + ((size_t)q.pm * g.ncol + (size_t)q.ix * g.nzT) * g.ny + y0;
    z_last<N, -1, ZPlan<N, C>::TF>(s, [&](int k, int l, C v) {
      int iz;
      if (k <= nz) iz = k;
      else if (k >= N - nz) iz = k - N;
      else return;
      if (y0 + l < g.ny) o[(size_t)(iz + nz) * g.ny + l] = v;
    });
    __syncthreads();
    if (threadIdx.x == 0 && tn < ntile) {
      fence_proxy_async();
      issue(tn, b);
      tn = next(tn + gridDim.x);
    }
  }
}

// ------------------------------------------------------------- dispatch ----
int z_rows(int N, bool fp32) {
  switch (N) {
#define HST_Z(n) \
  case n: return fp32 ? ZPlan<n, float2>::TY : ZPlan<n, double2>::TY;
    HST_Z_LENGTHS32(HST_Z)
#undef HST_Z
#define HST_Z(n) \
  case n: return fp32 ? 0 : ZPlan<n, double2>::TY;
    HST_Z(48) HST_Z(64) HST_Z(128) HST_Z(256) HST_Z(512) HST_Z(1024)
#undef HST_Z
  }
  return 0;
}
static int z_box(int N) { return N <= 256 ? N : (N % 256 == 0 ? 256 : 192); }

int z_twiddles(int N, double2* out) {
  switch (N) {
#define HST_Z(n) \
  case n: return z_twiddles_t<n, double2>(out);
    HST_Z_LENGTHS64(HST_Z)
#undef HST_Z
  }
  return 0;
}
int z_twiddles(int N, float2* out) {
  switch (N) {
#define HST_Z(n) \
  case n: return z_twiddles_t<n, float2>(out);
    HST_Z_LENGTHS32(HST_Z)
#undef HST_Z
  }
  return 0;
}

// The map of Pp (or Ppg) for the forward kernel: 4-D reals {2 Ty, nxB, nzd
// tiles, comps}, box {2 Ty, 1, z points of a copy, 1}.
cudaError_t make_z_maps(const Geometry& g, DeviceState& d) {
  if (!z_rows(g.nzd, g.mp != 0)) return cudaSuccess;
  const EncodeTiled enc = encode_tiled();
  if (!enc) return cudaErrorNotSupported;
  for (int which = 0; which < 2; ++which) {
    double2* const base = which == 0 ? d.Pp : d.Ppg;
    if (!base) continue;
    const cuuint64_t es = g.mp ? 8 : 16;
    const int nyT = which == 0 ? g.nyT : 1;
    cuuint64_t dims[4] = {(cuuint64_t)2 * g.Ty, (cuuint64_t)g.nxB, (cuuint64_t)g.nzd * nyT, (cuuint64_t)6 * g.nmem};
    cuuint64_t strides[3] = {es * g.Ty, es * g.Ty * g.nxB, es * g.Ty * g.nxB * g.nzd * nyT};
    cuuint32_t box[4] = {(cuuint32_t)(2 * g.Ty), 1, (cuuint32_t)z_box(g.nzd), 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(which == 0 ? &d.tmPz : &d.tmPgz, g.mp ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                           4, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
  }
  return cudaSuccess;
}

template <int N, typename C>
static cudaError_t z_inv_t(const Geometry& g, const DeviceState& d, const C* tw, cudaStream_t st) {
  smem_limit(d, k_z_inv<N, C>, (int)ZShape<N, C>::tile);
  const int grp = z_inv_group<N, C>(g.nxB), nyT = (g.ny + ZPlan<N, C>::TY - 1) / ZPlan<N, C>::TY;
  const dim3 grid((g.nxB + grp - 1) / grp * grp * nyT, 3 * g.nmem);
  return launch_after(k_z_inv<N, C>, grid, ZPlan<N, C>::TI, ZShape<N, C>::tile, st, g, d.F[0], d.F[1], d.F[2],
                      reinterpret_cast<C*>(d.Z), tw + 2 * N);
}
template <int N, typename C>
static cudaError_t z_fwd_t(const Geometry& g, const DeviceState& d, int np, const C* tw, cudaStream_t st) {
  typedef ZPlan<N, C> P;
  static_assert(z_fwd_smem<N, C>() <= 227 * 1024, "the buffers fit one block");
  smem_limit(d, k_z_fwd<N, C>, (int)z_fwd_smem<N, C>());
  const int ntile = (g.ny + P::TY - 1) / P::TY * ((g.nxB + 3) / 4 * 4) * np * g.nmem;
  const int nb = std::min(ntile, (d.nsm > 0 ? d.nsm : 148) * P::MBF);
  return launch_after(k_z_fwd<N, C>, dim3(nb), P::TF, z_fwd_smem<N, C>(), st, g, np, reinterpret_cast<C*>(d.Q), tw + N, d.tmPz,
                      d.err);
}

#define HST_Z_DISPATCH(F)                                    \
  if (g.mp) {                                                \
    switch (g.nzd) { HST_Z_LENGTHS32(HST_Z32) }              \
    return cudaErrorInvalidValue;                            \
  }                                                          \
  switch (g.nzd) { HST_Z_LENGTHS64(HST_Z64) }                \
  return cudaErrorInvalidValue
cudaError_t launch_z_inv(const Geometry& g, const DeviceState& d, cudaStream_t st) {
#define HST_Z32(n) case n: return z_inv_t<n, float2>(g, d, d.twzf, st);
#define HST_Z64(n) case n: return z_inv_t<n, double2>(g, d, d.twz, st);
  HST_Z_DISPATCH();
#undef HST_Z32
#undef HST_Z64
}
cudaError_t launch_z_fwd(const Geometry& g, const DeviceState& d, int np, cudaStream_t st) {
#define HST_Z32(n) case n: return z_fwd_t<n, float2>(g, d, np, d.twzf, st);
#define HST_Z64(n) case n: return z_fwd_t<n, double2>(g, d, np, d.twz, st);
  HST_Z_DISPATCH();
#undef HST_Z32
#undef HST_Z64
}

}  // namespace hst
