// Fused, pruned column transforms of the FP32 form.
//
// A w-plane's 2-D transform is done as row transforms (gb_rows.cu, or batched
// 1-D cuFFT for other widths) plus column transforms written here.  Column mode
// applies when the grid height is a power of two and exactly twice the
// image height (sigma = 2), so the image occupies the middle half of every
// column (checkerboarded grids) and only the image's nx columns need
// transforms.  The column length n = N1 N2 is split four-step
// (q = N2 q1 + q2, k = k1 + N1 k2):
//
//   step A  for each q2: the N1-point DFT over q1 of x[N2 q1 + q2], times
//           exp(s 2 pi i q2 k1 / n), stored back at rows N2 k1 + q2;
//   step B  for each k1: the N2-point DFT over the contiguous rows
//           N2 k1 + q2 gives X[k1 + N1 k2].
//
// Each CTA transforms a tile of kCW = 32 adjacent columns (256-byte row
// segments; lane = column).  A column of length N is split N = T M over
// the T warps: warp t holds elements t + T m (m < M) in registers, does an
// M-point DFT in registers, multiplies by exp(s 2 pi i t k1 / N), and one
// exchange through shared memory gives each warp the T-point DFTs of
// outputs k1 + M k2 -- one shared-memory round trip per tile instead of a
// pass per radix stage.
//
// Fusions:
//   invert  (rows first, then columns)  step B never writes the plane back:
//           it keeps only the image rows (outputs k2 in [T/4, 3T/4) of every
//           warp), applies each plane's w-screen and accumulates the image
//           in registers over the batch's planes and pols, with the next
//           tile's loads in flight (cp.async, double-buffered);
//   predict (columns first, then rows)  step A builds its input from the
//           corrected image (inputs m in [M/4, 3M/4) of every warp, zero
//           elsewhere) times each plane's w-screen, and step B writes in
//           place, so physical row N2 k1 + k2 holds logical row k1 + N1 k2;
//           the degridder reads rows through that permutation (RowPerm).
//
// The w-screen of plane k at a pixel is exp(s 2 pi i (A + k D)) with A, D the
// pixel's FP64 phase terms stored as 64-bit fixed-point turns, so the
// per-plane phase is exact integer arithmetic (no FP64 work per plane) and
// only the final sincos of the reduced phase is FP32.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cufft.h>

#include <mutex>

#include "gb_async.cuh"
#include "gb_dft.cuh"
#include "gb_fft.cuh"

namespace gb {

constexpr int kCW = 32;  // columns per tile: one lane per column

template <int N>
struct ColShape {
  static constexpr int T = N <= 32 ? 4 : (N <= 128 ? 8 : 16);  // warps per column tile
  static constexpr int M = N / T;                              // elements per thread
  static constexpr int THREADS = kCW * T;
  static_assert(M % T == 0 && M % 4 == 0 && T % 4 == 0, "column split");
};

// In-register L-point DFTs in natural order, z_q = sum_p a_p exp(s 2 pi i p q / L).
template <int S> __device__ __forceinline__ void dft4(float2 *a) {
  const float2 s02 = cadd(a[0], a[2]), d02 = csub(a[0], a[2]);
  const float2 s13 = cadd(a[1], a[3]), d13 = csub(a[1], a[3]);
  a[0] = cadd(s02, s13);
  a[2] = csub(s02, s13);
  a[1] = cadd_si<S>(d02, d13);
  a[3] = csub_si<S>(d02, d13);
}

template <int S> __device__ __forceinline__ void dft8(float2 *a) {
  float2 e[4] = {a[0], a[2], a[4], a[6]};
  float2 o[4] = {a[1], a[3], a[5], a[7]};
  dft4<S>(e);
  dft4<S>(o);
  const float2 t0 = o[0], t1 = cmulc(o[1], kR2, S * kR2), t3 = cmulc(o[3], -kR2, S * kR2);
  a[0] = cadd(e[0], t0);
  a[4] = csub(e[0], t0);
  a[1] = cadd(e[1], t1);
  a[5] = csub(e[1], t1);
  a[2] = cadd_si<S>(e[2], o[2]);
  a[6] = csub_si<S>(e[2], o[2]);
  a[3] = cadd(e[3], t3);
  a[7] = csub(e[3], t3);
}

// 16 = 4 x 4: n = 4 n1 + n2, k = k1 + 4 k2.
template <int S> __device__ __forceinline__ void dft16(float2 *a) {
  float2 y[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    float2 b[4] = {a[n2], a[4 + n2], a[8 + n2], a[12 + n2]};
    dft4<S>(b);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) y[n2][k1] = b[k1];
  }
  // twiddles exp(s 2 pi i n2 k1 / 16)
  y[1][1] = cmulc(y[1][1], kC8, S * kS8);
  y[1][2] = cmulc(y[1][2], kR2, S * kR2);
  y[1][3] = cmulc(y[1][3], kS8, S * kC8);
  y[2][1] = cmulc(y[2][1], kR2, S * kR2);
  y[2][2] = mul_si<S>(y[2][2]);
  y[2][3] = cmulc(y[2][3], -kR2, S * kR2);
  y[3][1] = cmulc(y[3][1], kS8, S * kC8);
  y[3][2] = cmulc(y[3][2], -kR2, S * kR2);
  y[3][3] = cmulc(y[3][3], -kC8, -S * kS8);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    float2 b[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
    dft4<S>(b);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) a[k1 + 4 * k2] = b[k2];
  }
}

// 32 = 2 x 16: X[k] = E[k] + w^k O[k], X[k + 16] = E[k] - w^k O[k].
template <int S> __device__ __forceinline__ void dft32(float2 *a) {
  float2 e[16], o[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    e[i] = a[2 * i];
    o[i] = a[2 * i + 1];
  }
  dft16<S>(e);
  dft16<S>(o);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const float2 t = k == 0 ? o[0] : cmulc(o[k], kCos32[k], S * kSin32[k]);
    a[k] = cadd(e[k], t);
    a[k + 16] = csub(e[k], t);
  }
}

template <int L, int S> __device__ __forceinline__ void dft(float2 *a) {
  if constexpr (L == 4) dft4<S>(a);
  else if constexpr (L == 8) dft8<S>(a);
  else if constexpr (L == 16) dft16<S>(a);
  else dft32<S>(a);
}

// N-point DFT of every column of a tile.  On entry x[m] holds column
// element t + T m of this thread's column (lane c, warp t); on exit
// y[ii][k2] holds output k1 + M k2 with k1 = t + T ii.  xb: N * kCW
// exchange slots; this thread writes only slots (r T + t) kCW + c, r < M,
// before the barrier.  The caller synchronises before xb is reused.
// tw[m] = exp(s 2 pi i m / N).
template <int N, int S>
__device__ __forceinline__ void col_dft_in(float2 (&x)[ColShape<N>::M], float2 *__restrict__ xb,
                                           const float2 *__restrict__ tw, int t, int c) {
  constexpr int T = ColShape<N>::T, M = ColShape<N>::M;
  dft<M, S>(x);
#pragma unroll
  for (int k1 = 1; k1 < M; ++k1) x[k1] = cmul(x[k1], tw[t * k1]);
#pragma unroll
  for (int k1 = 0; k1 < M; ++k1) xb[(k1 * T + t) * kCW + c] = x[k1];
}
// The second half of it, after the barrier: outputs t + T ii + M k2 in y[k2].
template <int N, int S>
__device__ __forceinline__ void col_dft_out(const float2 *__restrict__ xb, int t, int c, int ii,
                                            float2 (&y)[ColShape<N>::T]) {
  constexpr int T = ColShape<N>::T;
#pragma unroll
  for (int tt = 0; tt < T; ++tt) y[tt] = xb[((t + T * ii) * T + tt) * kCW + c];
  dft<T, S>(y);
}
template <int N, int S>
__device__ __forceinline__ void col_dft(float2 (&x)[ColShape<N>::M], float2 *__restrict__ xb,
                                        const float2 *__restrict__ tw, int t, int c,
                                        float2 (&y)[ColShape<N>::M / ColShape<N>::T]
                                                   [ColShape<N>::T]) {
  col_dft_in<N, S>(x, xb, tw, t, c);
  __syncthreads();
#pragma unroll
  for (int ii = 0; ii < ColShape<N>::M / ColShape<N>::T; ++ii)
    col_dft_out<N, S>(xb, t, c, ii, y[ii]);
}

// exp(s 2 pi i m / N), m < N, from the n-point table exp(+2 pi i m / n).
template <int N, int S>
__device__ __forceinline__ void load_twiddles(float2 *tw, const float2 *__restrict__ twn, int n) {
  const int step = n / N;
  for (int m = threadIdx.x; m < N; m += blockDim.x) {
    const float2 w = twn[m * step];
    tw[m] = S > 0 ? w : conjf2(w);
  }
}

// sin / cos of plane k's w-screen phase 2 pi (A + k D) at a pixel.
__device__ __forceinline__ void screen_sincos(ulonglong2 ad, int k, float *sn, float *cs) {
  const unsigned long long ph = ad.x + (unsigned long long)(unsigned)k * ad.y;
  const int hi = (int)(unsigned)(ph >> 32);  // turns * 2^32 in [-2^31, 2^31)
  sincospif((float)hi * 0x1p-31f, sn, cs);
}

// The screens of planes b0, b0 + 1, ... at one pixel by rotation: (cs, sn)
// of plane b0 from its exact fixed-point phase, then one complex multiply
// by exp(2 pi i D) per plane (an error of a few FP32 roundings per plane
// step; the batches hold a handful of planes), instead of a sincos per plane.
struct ScreenRot {
  float cs, sn, dc, ds;
  __device__ __forceinline__ void start(ulonglong2 ad, int k) {
    screen_sincos(ad, k, &sn, &cs);
    screen_sincos(make_ulonglong2(ad.y, 0ull), 0, &ds, &dc);
  }
  __device__ __forceinline__ void unit() {
    cs = 1.f;
    sn = 0.f;
    dc = 1.f;
    ds = 0.f;
  }
  __device__ __forceinline__ void next() {
    const float c = cs * dc - sn * ds, s = sn * dc + cs * ds;
    cs = c;
    sn = s;
  }
};

// ----------------------------------------------------------------------
// The in-place steps: invert step A (A: N = N1, one CTA column per (column
// tile, q2)) and predict step B (N = N2, per (column tile, k1)).  A CTA runs
// `per` consecutive plane-pols of the batch through S shared-memory tiles: a
// warp copies the rows it transforms (rows m T + t of the tile) with 16-byte
// cp.async S - 1 tiles ahead, and the exchange reuses their slots, so one
// barrier per tile serves both the exchange and the refill of the tile before.
// Step A reads only rows in the occupancy mask (the others were never zeroed
// nor gridded) and takes the rest as zero; step B writes only those rows (the
// others' transforms are never degridded).
// HBM bound: two tiles per CTA and as many CTAs as fit keep more bytes in
// flight than three tiles did, and both more than loads into registers behind
// one CTA per plane-pol.  8192 x 4096 columns, 42 planes of 4 pols: step A
// (N = 64) 15.2 ms in registers, 11.8 with three tiles and 4 CTAs, 11.2 with
// two and 5; step B (N = 128) 11.9, 12.7 with three tiles and 2 CTAs, 10.3
// with two and 3.
template <int N> struct ColPipe {
  static constexpr int S = 2;  // tiles
  static constexpr int CTAS = N <= 32 ? 8 : N == 64 ? 5 : N == 128 ? 3 : 1;  // per SM
};
template <int N, bool A>
__global__ void __launch_bounds__(ColShape<N>::THREADS, ColPipe<N>::CTAS)
    k_cols_inplace(const ColGeom cg, const float2 *__restrict__ twn, float2 *__restrict__ grid,
                   int npp, int per) {
  using CS = ColShape<N>;
  constexpr int T = CS::T, M = CS::M, S = ColPipe<N>::S;
  extern __shared__ __align__(128) float2 smem[];
  float2 *tw = smem + S * N * kCW;
  float2 *st = tw + N;  // step A: exp(2 pi i q2 o / n), o < N
  const int c = threadIdx.x % kCW, t = threadIdx.x / kCW;
  const int p0 = cg.ox + blockIdx.x * kCW;
  const int cols = min(kCW, cg.ox + cg.nx - p0);  // even
  const int q = blockIdx.y;
  const int s0 = blockIdx.z * per, ns = min(per, npp - s0);
  auto row = [&](int r) { return A ? cg.N2 * r + q : N * q + r; };
  // mask word of lane i's row (i < M): the input t + T i, or output i, of this warp
  const int mine = A ? row(t + T * c) : q + cg.N1 * (t + T * (c % (M / T)) + M * (c / (M / T)));
  const uint32_t *word = cg.mask + (int64_t)cg.b0 * cg.ntv + (c < M ? mine / cg.T : 0);
  auto used = [&](int s) {
    const uint32_t w = s < ns && c < M ? word[(int64_t)((s0 + s) / cg.NP) * cg.ntv] : 0u;
    return __ballot_sync(0xffffffffu, w != 0);
  };
  const int part = 2 * (c % 16), half = c / 16;  // the lane's columns and row of a copied pair
  auto load = [&](int s, uint32_t rows) {
    if (s < ns && part < cols) {
      const float2 *src = grid + (int64_t)(s0 + s) * cg.plane + p0 + part;
      float2 *dst = smem + (s % S) * N * kCW + part;
#pragma unroll
      for (int i = 0; i < M / 2; ++i) {
        const int m = 2 * i + half, r = m * T + t;
        if (!A || (rows >> m & 1))
          cp_async16(dst + r * kCW, src + (int64_t)row(r) * cg.ngx);
        else
          *reinterpret_cast<float4 *>(dst + r * kCW) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < S - 1; ++s) load(s, A ? used(s) : 0u);
  load_twiddles<N, A ? 1 : -1>(tw, twn, cg.n);
  if (A)
    for (int o = threadIdx.x; o < N; o += blockDim.x) st[o] = twn[q * o];
  __syncthreads();
  for (int s = 0; s < ns; ++s) {
    const uint32_t rows = used(A ? s + S - 1 : s);
    float2 *cur = smem + (s % S) * N * kCW;
    cp_async_wait<S - 2>();
    __syncwarp();
    float2 x[M];
#pragma unroll
    for (int m = 0; m < M; ++m) x[m] = cur[(m * T + t) * kCW + c];
    col_dft_in<N, A ? 1 : -1>(x, cur, tw, t, c);
    __syncthreads();  // exchange complete; tile s - 1 consumed
    load(s + S - 1, rows);
    float2 *plane = grid + (int64_t)(s0 + s) * cg.plane + p0 + c;
#pragma unroll
    for (int ii = 0; ii < M / T; ++ii) {
      float2 y[T];
      col_dft_out<N, A ? 1 : -1>(cur, t, c, ii, y);
#pragma unroll
      for (int k2 = 0; k2 < T; ++k2) {
        const int o = t + T * ii + M * k2;
        if (c < cols && (A || (rows >> (ii + M / T * k2) & 1)))
          plane[(int64_t)row(o) * cg.ngx] = A ? cmul(y[k2], st[o]) : y[k2];
      }
    }
  }
}

// invert step B + w-screen + accumulate: one CTA per (column tile, k1).
// The batch's nb x NP plane-pols stream through two shared-memory tile
// buffers filled by TMA (one 2-D box of N2 rows x 32 columns per tile,
// completion on an mbarrier), so the next tile is in flight while this one
// is transformed; the kept outputs accumulate in per-thread shared-memory
// slots.  A wait that runs past its iteration limit records kErrTmaTimeout
// in *status, drains the other buffer (bounded) and returns.
template <int N2, int NP>
__global__ void __launch_bounds__(ColShape<N2>::THREADS, N2 >= 256 ? 1 : 2)
    k_cols_b_inv(const __grid_constant__ CUtensorMap tmap, const ColGeom cg,
                 const float2 *__restrict__ twn, const ulonglong2 *__restrict__ screen, int do_w,
                 int b0, int nb, float *__restrict__ acc, int first,
                 uint32_t *__restrict__ status) {
  using CS = ColShape<N2>;
  constexpr int T = CS::T, M = CS::M, MT = M / T, KL = T / 4, KK = T / 2;
  constexpr int NK = MT * KK;  // kept outputs per thread
  constexpr unsigned kTileBytes = N2 * kCW * sizeof(float2);
  // dynamic shared memory only (TMA destinations at 128-byte offsets):
  // two tiles | twiddles | accumulators | 2 mbarriers | abort flag
  extern __shared__ __align__(128) float2 smem[];
  auto buf = [&](int s) { return smem + (s & 1) * (N2 * kCW); };
  float2 *tw = smem + 2 * N2 * kCW;
  float *sacc = reinterpret_cast<float *>(tw + N2);  // [NP][NK][T][kCW]
  uint64_t *bar = reinterpret_cast<uint64_t *>(sacc + NP * NK * T * kCW);
  int &s_abort = *reinterpret_cast<int *>(bar + 2);
  const int c = threadIdx.x % kCW, t = threadIdx.x / kCW;
  const int p0 = cg.ox + blockIdx.x * kCW;
  const int p = p0 + c;
  const bool ok = p < cg.ox + cg.nx;
  const int ix = p - cg.ox;
  const int k1o = blockIdx.y;
  const int64_t npix = (int64_t)cg.nx * cg.ny;
  const int iters = nb * NP;
  // tile s = plane-pol s of the batch buffer: rows s ngy + N2 k1o + [0, N2)
  auto issue = [&](int s) {
    fence_proxy_async();  // earlier generic writes to the buffer before the async copy
    mbar_expect_tx(&bar[s & 1], kTileBytes);
    tma_load_2d(buf(s), &tmap, p0, s * cg.n + cg.N2 * k1o, &bar[s & 1]);
  };
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    s_abort = 0;
    fence_mbarrier_init();
  }
  load_twiddles<N2, 1>(tw, twn, cg.n);
  __syncthreads();
  if (threadIdx.x == 0) issue(0);
  // kept output e = ii KK + kk: o = t + T ii + M (KL + kk), image row k1o + N1 o - oy
  auto pixel = [&](int e) {
    const int ii = e / KK, kk = e - ii * KK;
    const int o = t + T * ii + M * (KL + kk);
    return (int64_t)(k1o + cg.N1 * o - cg.oy) * cg.nx + ix;
  };
  auto slot = [&](int pol, int e) { return ((pol * NK + e) * T + t) * kCW + c; };
#pragma unroll 1
  for (int pol = 0; pol < NP; ++pol)
#pragma unroll
    for (int e = 0; e < NK; ++e)
      sacc[slot(pol, e)] = (first || !ok) ? 0.f : acc[pol * npix + pixel(e)];
  int s = 0;
  ScreenRot scr[NK];
#pragma unroll
  for (int e = 0; e < NK; ++e) {
    if (do_w && ok)
      scr[e].start(screen[pixel(e)], b0);
    else
      scr[e].unit();
  }
  for (int j = 0; j < nb; ++j) {
    if (j > 0) {
#pragma unroll
      for (int e = 0; e < NK; ++e) scr[e].next();
    }
#pragma unroll 1
    for (int pol = 0; pol < NP; ++pol, ++s) {
      if (threadIdx.x == 0 && s + 1 < iters) issue(s + 1);
      float2 *cur = buf(s);
      if (!mbar_wait(&bar[s & 1], (s >> 1) & 1)) s_abort = 1;
      float2 x[M];
#pragma unroll
      for (int m = 0; m < M; ++m) x[m] = cur[(m * T + t) * kCW + c];
      float2 y[MT][T];
      col_dft<N2, 1>(x, cur, tw, t, c, y);
#pragma unroll
      for (int e = 0; e < NK; ++e) {
        const float2 v = y[e / KK][KL + e % KK];
        sacc[slot(pol, e)] += v.x * scr[e].cs + v.y * scr[e].sn;  // Re(v exp(-i theta))
      }
      __syncthreads();  // tile s consumed before its buffer is refilled
      if (s_abort) {
        if (threadIdx.x == 0) {
          atomicOr(status, kErrTmaTimeout);
          if (s + 1 < iters) mbar_wait(&bar[(s + 1) & 1], ((s + 1) >> 1) & 1);
        }
        return;
      }
    }
  }
  if (ok) {
#pragma unroll 1
    for (int pol = 0; pol < NP; ++pol)
#pragma unroll
      for (int e = 0; e < NK; ++e) acc[pol * npix + pixel(e)] = sacc[slot(pol, e)];
  }
}

// predict step A from the corrected image: one CTA per (column tile, q2);
// loops over the batch's planes and the pols.  The screens of the CTA's pixels
// (inputs m in [M/4, 3M/4) of each thread) sit in registers, those of the
// batch's later planes from the first by rotation (ScreenRot); the image
// values sit in per-thread shared-memory slots.  Two exchange buffers, so that
// a tile needs one barrier.
// Bound by its stores to HBM and, at N = 128, by instructions: with the
// screens in shared memory, one buffer and 2 CTAs 8.7 ms at 8192 x 4096 columns
// (N = 64), 42 planes of 4 pols, and 16.4 ms at 16384 x 8192 (N = 128), 14
// planes; so 7.2 and 15.2.  4 CTAs at N = 64 spill: 7.5.
template <int N> struct ColPredA {
  static constexpr int CTAS = N <= 32 ? 6 : N == 64 ? 3 : 2;  // per SM
};
template <int N1, int NP>
__global__ void __launch_bounds__(ColShape<N1>::THREADS, ColPredA<N1>::CTAS)
    k_cols_a_pred(const ColGeom cg, const float2 *__restrict__ twn, const float *__restrict__ img,
                  const ulonglong2 *__restrict__ screen, int do_w, int b0, int nb,
                  float2 *__restrict__ grid) {
  using CS = ColShape<N1>;
  constexpr int T = CS::T, M = CS::M, ML = M / 4, MK = M / 2;
  extern __shared__ float2 smem[];
  float2 *tw = smem + 2 * N1 * kCW;
  float2 *st = tw + N1;                             // exp(-2 pi i q2 o / n), o < N1
  float *sv = reinterpret_cast<float *>(st + N1);   // [NP][MK][T][kCW]
  const int c = threadIdx.x % kCW, t = threadIdx.x / kCW;
  const int p = cg.ox + blockIdx.x * kCW + c;
  const bool ok = p < cg.ox + cg.nx;
  const int ix = p - cg.ox;
  const int q2 = blockIdx.y;
  const int64_t npix = (int64_t)cg.nx * cg.ny;
  load_twiddles<N1, -1>(tw, twn, cg.n);
  for (int o = threadIdx.x; o < N1; o += blockDim.x) st[o] = conjf2(twn[q2 * o]);
  // image input mm: row N2 (t + T (ML + mm)) + q2 of the grid, minus oy
  auto pixel = [&](int mm) {
    const int q = cg.N2 * (t + T * (ML + mm)) + q2;
    return (int64_t)(q - cg.oy) * cg.nx + ix;
  };
  auto slot = [&](int pol, int mm) { return ((pol * MK + mm) * T + t) * kCW + c; };
#pragma unroll 1
  for (int pol = 0; pol < NP; ++pol)
#pragma unroll
    for (int mm = 0; mm < MK; ++mm)
      sv[slot(pol, mm)] = ok ? img[pol * npix + pixel(mm)] : 0.f;
  ScreenRot scr[MK];
#pragma unroll
  for (int mm = 0; mm < MK; ++mm) {
    if (do_w && ok)
      scr[mm].start(screen[pixel(mm)], b0);
    else
      scr[mm].unit();
  }
  __syncthreads();  // twiddles
  float2 *plane = grid + p;
  int k = 0;
#pragma unroll 1
  for (int j = 0; j < nb; ++j) {
#pragma unroll 1
    for (int pol = 0; pol < NP; ++pol, ++k, plane += cg.plane) {
      float2 *cur = smem + (k & 1) * (N1 * kCW);
      float2 x[M];
#pragma unroll
      for (int m = 0; m < M; ++m) x[m] = make_float2(0.f, 0.f);
#pragma unroll
      for (int mm = 0; mm < MK; ++mm) {
        const float v = sv[slot(pol, mm)];
        x[ML + mm] = make_float2(v * scr[mm].cs, v * scr[mm].sn);
      }
      col_dft_in<N1, -1>(x, cur, tw, t, c);
      __syncthreads();
#pragma unroll
      for (int ii = 0; ii < M / T; ++ii) {
        float2 y[T];
        col_dft_out<N1, -1>(cur, t, c, ii, y);
#pragma unroll
        for (int k2 = 0; k2 < T; ++k2) {
          const int o = t + T * ii + M * k2;
          if (ok) plane[(int64_t)(cg.N2 * o + q2) * cg.ngx] = cmul(y[k2], st[o]);
        }
      }
    }
#pragma unroll
    for (int mm = 0; mm < MK; ++mm) scr[mm].next();
  }
}

// ----------------------------------------------------------------------
// host side

static int ilog2(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}

bool column_split(int n, int &N1, int &N2) {
  if (n < 256 || n > 32768 || (n & (n - 1))) return false;
  const int lg = ilog2(n);
  const int l1 = lg / 2;  // N1 <= N2
  N1 = 1 << l1;
  N2 = 1 << (lg - l1);
  return N1 >= 16 && N1 <= 128 && N2 <= 256;
}

ColGeom col_geom(const Geom &g) {
  ColGeom cg;
  cg.mask = nullptr;
  cg.b0 = 0;
  cg.NP = g.NP;
  cg.T = g.T;
  cg.ntv = g.ntv;
  cg.n = g.ngy;
  column_split(g.ngy, cg.N1, cg.N2);
  cg.ox = (g.ngx - g.nx) / 2;
  cg.oy = (g.ngy - g.ny) / 2;
  cg.nx = g.nx;
  cg.ny = g.ny;
  cg.plane = (int64_t)g.ngx * g.ngy;
  cg.ngx = g.ngx;
  return cg;
}

RowPerm row_perm(const gb_plan *p) {
  RowPerm rp;
  rp.s1 = -1;
  rp.s2 = 0;
  if (p->col_fft) {
    const ColGeom cg = col_geom(p->g);
    rp.s1 = ilog2(cg.N1);
    rp.s2 = ilog2(cg.N2);
  }
  return rp;
}


// tiles + twiddles + step A's outer twiddles
template <int N> constexpr size_t smem_inplace() {
  return sizeof(float2) * ((size_t)ColPipe<N>::S * N * kCW + 2 * N);
}
// two exchange buffers + twiddles + image slots (N/2 inputs per column)
template <int N, int NP> constexpr size_t smem_a_pred() {
  return sizeof(float2) * ((size_t)2 * N * kCW + 2 * N) + sizeof(float) * NP * (size_t)(N / 2) * kCW;
}
// two tile buffers + twiddles + accumulator slots (N/2 kept outputs per column)
template <int N, int NP> constexpr size_t smem_b_inv() {
  return sizeof(float2) * ((size_t)2 * N * kCW + N) + sizeof(float) * NP * (size_t)(N / 2) * kCW +
         2 * sizeof(uint64_t) + 16;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// link against the driver library).
static PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  return fn;
}

// 2-D map over the batch buffer viewed as rows of ngx 8-byte cells
// (B NP ngy rows); box = 32 cells x box_rows rows.
static int make_tile_map(CUtensorMap *map, const gb_plan *p, const float2 *grid, int box_rows) {
  const Geom &g = p->g;
  PFN_cuTensorMapEncodeTiled_v12000 fn = encode_tiled();
  if (!fn) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return GB_ERR_CUDA;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)g.ngx, (cuuint64_t)g.B * g.NP * (cuuint64_t)g.ngy};
  const cuuint64_t strides[1] = {(cuuint64_t)g.ngx * sizeof(float2)};
  const cuuint32_t box[2] = {(cuuint32_t)kCW, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<float2 *>(grid), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d) for a %d x %lld grid batch", (int)r, g.ngx,
              (long long)dims[1]);
    return GB_ERR_CUDA;
  }
  return GB_OK;
}

// Kernels whose shared memory exceeds the 48 KB default need the opt-in.
template <int NP>
static int setup_np() {
#define GB_ATTR(K, B) \
  GB_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(B)))
  GB_ATTR((k_cols_b_inv<16, NP>), (smem_b_inv<16, NP>()));
  GB_ATTR((k_cols_b_inv<32, NP>), (smem_b_inv<32, NP>()));
  GB_ATTR((k_cols_b_inv<64, NP>), (smem_b_inv<64, NP>()));
  GB_ATTR((k_cols_b_inv<128, NP>), (smem_b_inv<128, NP>()));
  GB_ATTR((k_cols_b_inv<256, NP>), (smem_b_inv<256, NP>()));
  GB_ATTR((k_cols_inplace<64, true>), smem_inplace<64>());
  GB_ATTR((k_cols_inplace<128, true>), smem_inplace<128>());
  GB_ATTR((k_cols_inplace<64, false>), smem_inplace<64>());
  GB_ATTR((k_cols_inplace<128, false>), smem_inplace<128>());
  GB_ATTR((k_cols_inplace<256, false>), smem_inplace<256>());
  GB_ATTR((k_cols_a_pred<16, NP>), (smem_a_pred<16, NP>()));
  GB_ATTR((k_cols_a_pred<32, NP>), (smem_a_pred<32, NP>()));
  GB_ATTR((k_cols_a_pred<64, NP>), (smem_a_pred<64, NP>()));
  GB_ATTR((k_cols_a_pred<128, NP>), (smem_a_pred<128, NP>()));
#undef GB_ATTR
  return GB_OK;
}

int setup_col_kernels(gb_plan *p) {
  if (!p->col_fft) return GB_OK;
  switch (p->g.NP) {
    case 1: return setup_np<1>();
    case 2: return setup_np<2>();
    default: return setup_np<4>();
  }
}

// Invert step A or predict step B of npp plane-pols.  A CTA takes up to 8 of
// them, fewer where that would leave less than about eight CTAs per SM.
template <bool A>
static int run_inplace(gb_plan *p, const ColGeom &cg, const float2 *twn, float2 *grid, int npp,
                       unsigned tiles, cudaStream_t s) {
  const int rows = A ? cg.N2 : cg.N1;
  int per = 8;
  while (per > 1 && (int64_t)tiles * rows * ((npp + per - 1) / per) < (int64_t)8 * p->num_sms)
    per /= 2;
  const dim3 grd(tiles, rows, (npp + per - 1) / per);
#define GB_COL(N) \
  k_cols_inplace<N, A><<<grd, ColShape<N>::THREADS, smem_inplace<N>(), s>>>(cg, twn, grid, npp, per)
  switch (A ? cg.N1 : cg.N2) {
    case 16: GB_COL(16); break;
    case 32: GB_COL(32); break;
    case 64: GB_COL(64); break;
    case 128: GB_COL(128); break;
    default:
      if constexpr (!A) GB_COL(256);
      break;
  }
#undef GB_COL
  GB_LAUNCH_CHECK("k_cols_inplace");
  return GB_OK;
}

template <int NP>
static int cols_invert_np(gb_plan *p, float2 *grid, int b0, int nb, float *acc, int first,
                          cudaStream_t s) {
  const Geom &g = p->g;
  ColGeom cg = col_geom(g);
  cg.mask = p->at<uint32_t>(p->off_rowmask);
  cg.b0 = b0;
  const unsigned tiles = (unsigned)((g.nx + kCW - 1) / kCW);
  const float2 *twn = p->at<float2>(p->off_twn);
  const ulonglong2 *screen = g.do_w ? p->at<ulonglong2>(p->off_screen) : nullptr;
  const double cols = (double)nb * NP * cg.n * g.nx * sizeof(float2);  // image columns
  const double npix = (double)g.nx * g.ny;
  {
    ProfScope ps(kProfColInvA, s, (p->used_rows(b0, nb) + 1.0) * cols);  // used rows in, all out
    const int rc = run_inplace<true>(p, cg, twn, grid, nb * NP, tiles, s);
    if (rc) return rc;
  }
  {
    ProfScope ps(kProfColInvB, s,
                 cols + (first ? 1.0 : 2.0) * sizeof(float) * NP * npix +
                     (g.do_w ? 16.0 * npix : 0.0));
    const dim3 grd(tiles, cg.N1);
    CUtensorMap map;
    int rc = make_tile_map(&map, p, grid, cg.N2);
    if (rc) return rc;
    uint32_t *status = p->status_word();
#define GB_COLB(N)                                                                 \
  k_cols_b_inv<N, NP><<<grd, ColShape<N>::THREADS, smem_b_inv<N, NP>(), s>>>(       \
      map, cg, twn, screen, g.do_w, b0, nb, acc, first, status)
    switch (cg.N2) {
      case 16: GB_COLB(16); break;
      case 32: GB_COLB(32); break;
      case 64: GB_COLB(64); break;
      case 128: GB_COLB(128); break;
      default: GB_COLB(256); break;
    }
#undef GB_COLB
    GB_LAUNCH_CHECK("k_cols_b_inv");
  }
  return GB_OK;
}

template <int NP>
static int cols_predict_np(gb_plan *p, const float *img, int b0, int nb, float2 *grid,
                           cudaStream_t s) {
  const Geom &g = p->g;
  ColGeom cg = col_geom(g);
  cg.mask = p->at<uint32_t>(p->off_rowmask);
  cg.b0 = b0;
  const unsigned tiles = (unsigned)((g.nx + kCW - 1) / kCW);
  const float2 *twn = p->at<float2>(p->off_twn);
  const ulonglong2 *screen = g.do_w ? p->at<ulonglong2>(p->off_screen) : nullptr;
  const double cols = (double)nb * NP * cg.n * g.nx * sizeof(float2);
  const double npix = (double)g.nx * g.ny;
  {
    ProfScope ps(kProfColPredA, s,
                 cols + sizeof(float) * NP * npix + (g.do_w ? 16.0 * npix : 0.0));
    const dim3 grd(tiles, cg.N2);
#define GB_COLA(N)                                                                   \
  k_cols_a_pred<N, NP><<<grd, ColShape<N>::THREADS, smem_a_pred<N, NP>(), s>>>(cg, twn, img, \
                                                                        screen, g.do_w, b0, nb, grid)
    switch (cg.N1) {
      case 16: GB_COLA(16); break;
      case 32: GB_COLA(32); break;
      case 64: GB_COLA(64); break;
      default: GB_COLA(128); break;
    }
#undef GB_COLA
    GB_LAUNCH_CHECK("k_cols_a_pred");
  }
  {
    ProfScope ps(kProfColPredB, s, (1.0 + p->used_rows(b0, nb)) * cols);  // all in, used rows out
    const int rc = run_inplace<false>(p, cg, twn, grid, nb * NP, tiles, s);
    if (rc) return rc;
  }
  if (!p->row_fft) {
    // zero the columns outside the image: [0, ox) and [ox + nx, ngx) of every row
    // (k_rows reads only the image columns, so it needs no zeros there)
    const size_t rows = (size_t)nb * NP * g.ngy, pitch = sizeof(float2) * g.ngx;
    const size_t left = sizeof(float2) * cg.ox, right = sizeof(float2) * (g.ngx - cg.ox - g.nx);
    ProfScope ps(kProfZeroMargins, s, (double)rows * (left + right));
    if (left) GB_CUDA(cudaMemset2DAsync(grid, pitch, 0, left, rows, s));
    if (right) GB_CUDA(cudaMemset2DAsync(grid + cg.ox + g.nx, pitch, 0, right, rows, s));
  }
  return GB_OK;
}

int run_cols_invert(gb_plan *p, void *grid, int b0, int nb, float *acc, int first,
                    cudaStream_t s) {
  switch (p->g.NP) {
    case 1: return cols_invert_np<1>(p, (float2 *)grid, b0, nb, acc, first, s);
    case 2: return cols_invert_np<2>(p, (float2 *)grid, b0, nb, acc, first, s);
    default: return cols_invert_np<4>(p, (float2 *)grid, b0, nb, acc, first, s);
  }
}

int run_cols_predict(gb_plan *p, const float *img, int b0, int nb, void *grid, cudaStream_t s) {
  switch (p->g.NP) {
    case 1: return cols_predict_np<1>(p, img, b0, nb, (float2 *)grid, s);
    case 2: return cols_predict_np<2>(p, img, b0, nb, (float2 *)grid, s);
    default: return cols_predict_np<4>(p, img, b0, nb, (float2 *)grid, s);
  }
}

}  // namespace gb
