// Row transforms of the FP32 form (k_rows) and the zeroing of the rows that
// the gridder writes (k_zero_rows).
//
// Both follow the occupancy mask of a plan: per (w-plane, row tile) a word
// whose bit b says that some visibility reaches cells [b bw, (b + 1) bw) of
// the tile's rows, bw = N / 32.  A w-plane of an interferometer's uv coverage
// is mostly empty (2 % to 20 % of the cells are in occupied bins where 20 % to
// 95 % of the rows are in occupied tiles), so
//   k_zero_rows  zeroes the occupied bins only,
//   invert       reads the occupied bins of a row (zero elsewhere) and stores
//                the image columns,
//   predict      reads the image columns and stores the occupied bins (the
//                degridder reads no others),
// and rows without any are skipped.
//
// A row of N = 32 R2 R3 cells is held by TN = R2 R3 threads and transformed by
// two nested four-step splits, in registers with two exchanges through shared
// memory:
//   pass 1  thread t holds x[t + TN m], m < 32: 32-point DFT, times w_N^(t k1);
//   pass 2  unit (k1, s), s < R3, holds the pass-1 outputs k1 of threads
//           s + R3 m: R2-point DFT over m, times w_TN^(s k');
//   pass 3  unit (k1, k') holds the pass-2 outputs k' of units (k1, s): R3-point
//           DFT over s, giving X[k1 + 32 k' + 32 R2 k2].
//
// Butterflies run on packed pairs (C2): two complex numbers whose real parts
// share one 64-bit register pair and whose imaginary parts share another, so an
// addition, multiplication or multiply-add of both is one f32x2 instruction.
// Pass 1 pairs the halves of its 32-point DFT: lane x of pair m is
// x[m] + x[m + 16] (even outputs), lane y (x[m] - x[m + 16]) w_32^m (odd ones);
// its outputs are pairs (2 k, 2 k + 1), which passes 2 and 3 carry through, two
// units at a time with equal twiddles, to 16-byte stores of adjacent cells.
// The kernel was bound by instruction issue and latency in scalar arithmetic;
// pairs halve the floating-point instructions, 16-byte exchange slots the shared
// accesses.  Measured, invert / predict: 8192-cell rows of 168 plane-pols (59 % of
// the rows, 15 % of the cells occupied) 19.5 / 20.7 -> 15.9 / 14.3 ms; 16384-cell
// rows of 56 plane-pols (46 %, 14 %) 27.1 / 29.6 -> 19.0 / 16.9 ms; zeroing the same
// 8.8 -> 2.1 and 10.7 -> 2.5 ms.  What is left is issue (1.9 per cycle) and the
// latency of the exchanges with 16 warps per SM.
//
// From 4096 cells, the next row's input (occupied bins, up to 16, or the image
// columns) streams into a shared-memory stage by bulk copies (mbarrier
// completion) while passes 2 and 3 of this one run.  A wait past its limit
// records kErrTmaTimeout in *status, waits once more (bounded) for the copies in
// flight and returns.
#include "gb_async.cuh"
#include "gb_dft.cuh"
#include "gb_fft.cuh"

namespace gb {

// Two complex numbers: (r.x, i.x) and (r.y, i.y).
struct C2 {
  float2 r, i;
};
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ C2 padd(C2 a, C2 b) {
  return C2{__fadd2_rn(a.r, b.r), __fadd2_rn(a.i, b.i)};
}
__device__ __forceinline__ C2 psub(C2 a, C2 b) {
  return C2{__fadd2_rn(a.r, neg2(b.r)), __fadd2_rn(a.i, neg2(b.i))};
}
// shared-memory exchange slots of 16 bytes
__device__ __forceinline__ void put(float4 *p, C2 a) {
  *p = make_float4(a.r.x, a.r.y, a.i.x, a.i.y);
}
__device__ __forceinline__ C2 get(const float4 *p) {
  const float4 v = *p;
  return C2{make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
// times s i
template <int S> __device__ __forceinline__ C2 pmul_si(C2 a) {
  return S > 0 ? C2{neg2(a.i), a.r} : C2{a.i, neg2(a.r)};
}
// times (wr.x + i wi.x, wr.y + i wi.y)
__device__ __forceinline__ C2 pmul(C2 a, float2 wr, float2 wi) {
  return C2{__ffma2_rn(a.r, wr, __fmul2_rn(neg2(a.i), wi)),
            __ffma2_rn(a.r, wi, __fmul2_rn(a.i, wr))};
}
__device__ __forceinline__ C2 pmulc(C2 a, float c, float s) {
  return pmul(a, make_float2(c, c), make_float2(s, s));
}

template <int S> __device__ __forceinline__ void pdft4(C2 *a) {
  const C2 s02 = padd(a[0], a[2]), d02 = psub(a[0], a[2]);
  const C2 s13 = padd(a[1], a[3]), d13 = pmul_si<S>(psub(a[1], a[3]));
  a[0] = padd(s02, s13);
  a[2] = psub(s02, s13);
  a[1] = padd(d02, d13);
  a[3] = psub(d02, d13);
}

template <int S> __device__ __forceinline__ void pdft8(C2 *a) {
  C2 e[4] = {a[0], a[2], a[4], a[6]};
  C2 o[4] = {a[1], a[3], a[5], a[7]};
  pdft4<S>(e);
  pdft4<S>(o);
  const C2 t[4] = {o[0], pmulc(o[1], kR2, S * kR2), pmul_si<S>(o[2]), pmulc(o[3], -kR2, S * kR2)};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    a[k] = padd(e[k], t[k]);
    a[k + 4] = psub(e[k], t[k]);
  }
}

// 16 = 4 x 4: n = 4 n1 + n2, k = k1 + 4 k2.
template <int S> __device__ __forceinline__ void pdft16(C2 *a) {
  C2 y[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    C2 b[4] = {a[n2], a[4 + n2], a[8 + n2], a[12 + n2]};
    pdft4<S>(b);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) y[n2][k1] = b[k1];
  }
  y[1][1] = pmulc(y[1][1], kC8, S * kS8);
  y[1][2] = pmulc(y[1][2], kR2, S * kR2);
  y[1][3] = pmulc(y[1][3], kS8, S * kC8);
  y[2][1] = pmulc(y[2][1], kR2, S * kR2);
  y[2][2] = pmul_si<S>(y[2][2]);
  y[2][3] = pmulc(y[2][3], -kR2, S * kR2);
  y[3][1] = pmulc(y[3][1], kS8, S * kC8);
  y[3][2] = pmulc(y[3][2], -kR2, S * kR2);
  y[3][3] = pmulc(y[3][3], -kC8, -S * kS8);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    C2 b[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
    pdft4<S>(b);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) a[k1 + 4 * k2] = b[k2];
  }
}

template <int L, int S> __device__ __forceinline__ void pdft(C2 *a) {
  if constexpr (L == 4) pdft4<S>(a);
  else if constexpr (L == 8) pdft8<S>(a);
  else pdft16<S>(a);
}

// Pair m of a 32-point DFT from elements m and m + 16: (a + b, (a - b) w_32^m).
template <int S> __device__ __forceinline__ C2 pair32(float2 a, float2 b, int m) {
  const float2 d = cmulc(csub(a, b), kCos32[m], S * kSin32[m]);
  return C2{make_float2(a.x + b.x, d.x), make_float2(a.y + b.y, d.y)};
}
// the same with b = 0 (first != 0) or a = 0
template <int S> __device__ __forceinline__ C2 pair32_one(float2 v, int m, bool first) {
  const float f = first ? 1.f : -1.f;
  const float2 d = cmulc(v, f * kCos32[m], f * S * kSin32[m]);
  return C2{make_float2(v.x, d.x), make_float2(v.y, d.y)};
}

// Threads per CTA: one row's, at least a warp (two rows of 512 cells).  CTAs
// per SM: what registers and shared memory allow.
template <int N> struct RowShape;
template <> struct RowShape<512> { static constexpr int R2 = 4, R3 = 4, MINB = 16; };
template <> struct RowShape<1024> { static constexpr int R2 = 8, R3 = 4, MINB = 16; };
template <> struct RowShape<2048> { static constexpr int R2 = 8, R3 = 8, MINB = 8; };
template <> struct RowShape<4096> { static constexpr int R2 = 16, R3 = 8, MINB = 4; };
template <> struct RowShape<8192> { static constexpr int R2 = 16, R3 = 16, MINB = 2; };
template <> struct RowShape<16384> { static constexpr int R2 = 16, R3 = 32, MINB = 1; };

template <int N> struct RowLayout {
  static constexpr int R2 = RowShape<N>::R2, R3 = RowShape<N>::R3;
  static constexpr int TN = R2 * R3;                   // threads per row
  static constexpr int TH = TN < 32 ? 32 : TN;         // threads per CTA
  static constexpr int ROWS = TH / TN;                 // rows per CTA
  static constexpr bool STAGE = N >= 4096;             // bulk-copied input
  static constexpr int CAP = 16;                       // bins the stage holds
  static constexpr int X1 = 16 * (TN + 1);             // pairs of one exchange half
  // pass 2 -> 3 with R3 = 32: scalars, rows of 34 (pairs s, s + 16 adjacent)
  static constexpr int X2 = R3 == 32 ? R2 * 32 * 34 / 2 : 16 * TN;
  static constexpr int X = X1 > X2 ? X1 : X2;          // exchange: X pairs of 16 bytes
  static constexpr int NA = N / 128;  // two-level twiddles: w^m = ta[m >> 7] tb[m & 127]
  static constexpr size_t SMEM =
      sizeof(float4) * ((size_t)X * ROWS + TN) + sizeof(float2) * ((STAGE ? N / 2 : 0) + NA + 128);
};

struct RowArgs {
  float2 *grid;              // batch buffer: rows of ngx cells
  const uint32_t *mask;      // [nplanes][ntv] occupied bins
  const float2 *twx;         // exp(+2 pi i m / ngx), m < ngx
  uint32_t nrows;            // nb NP ngy rows in this batch
  int lgy, lnp;              // log2 of ngy and NP
  int b0, T, tshift, ntv;    // tshift: log2 T, or -1
  RowPerm rp;                // physical row of a logical row (predict)
  int lo, hi;                // image columns, inside [N/4, 3N/4)
  uint32_t *status;          // kErrTmaTimeout when a staging wait runs past its limit
};

template <int N, int S>
__global__ void __launch_bounds__(RowLayout<N>::TH, RowShape<N>::MINB) k_rows(const RowArgs ra) {
  using L = RowLayout<N>;
  constexpr int R2 = L::R2, R3 = L::R3, TN = L::TN, TH = L::TH, ROWS = L::ROWS, NA = L::NA;
  extern __shared__ __align__(16) float2 smem[];
  float4 *t2 = reinterpret_cast<float4 *>(smem);     // [TN] w_TN^m as (re, re, im, im)
  float4 *ex = t2 + TN;                               // exchange, [ROWS][X] pairs
  float2 *stg = reinterpret_cast<float2 *>(ex + L::X * ROWS);  // [N/2]: the next row's input
  float2 *ta = stg + (L::STAGE ? N / 2 : 0);
  float2 *tb = ta + NA;
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ int s_abort;
  const int t = threadIdx.x % TN, sub = threadIdx.x / TN, lane = threadIdx.x & 31;
  float4 *xb = ex + sub * L::X;
  const bool whole = ra.lo == N / 4 && ra.hi == 3 * (N / 4);  // image = middle half
  if (threadIdx.x == 0) {
    mbar_init(&s_bar, 1);
    s_abort = 0;
    fence_mbarrier_init();
  }
  for (int i = threadIdx.x; i < NA + 128; i += TH) {
    const float2 w = ra.twx[i < NA ? i * 128 : i - NA];
    (i < NA ? ta[i] : tb[i - NA]) = S > 0 ? w : conjf2(w);
  }
  for (int i = threadIdx.x; i < TN; i += TH) {
    const float2 w = ra.twx[i * 32];
    const float im = S > 0 ? w.y : -w.y;
    t2[i] = make_float4(w.x, w.x, im, im);
  }
  __syncthreads();  // tables and the barrier's initialisation
  auto sync = [] {
    if constexpr (TH == 32)
      __syncwarp();
    else
      __syncthreads();
  };
  auto tw = [&](int m) { return cmul(ta[m >> 7], tb[m & 127]); };
  // logical row l (plane-pol-major): its occupied bins and its cells
  auto bins = [&](uint32_t l) {
    const uint32_t sp = l >> ra.lgy, q = l & ((1u << ra.lgy) - 1);
    const uint32_t tile = ra.tshift >= 0 ? q >> ra.tshift : q / (uint32_t)ra.T;
    return __ldg(ra.mask + (size_t)(ra.b0 + (sp >> ra.lnp)) * ra.ntv + tile);
  };
  auto cells = [&](uint32_t l) {
    const int q = (int)(l & ((1u << ra.lgy) - 1));
    const uint32_t row = S > 0 ? l : (l - (uint32_t)q) + (uint32_t)ra.rp.row(q);
    return ra.grid + (size_t)row * N;
  };
  // the first group of ROWS rows from g on, in this CTA's stride, that holds an
  // occupied bin: 32 candidates per step, one per lane
  const uint32_t ngroups = ra.nrows / ROWS;
  auto next_used = [&](uint32_t g) {
    for (; g < ngroups; g += 32 * gridDim.x) {
      const uint32_t c = g + lane * gridDim.x;
      uint32_t b = 0;
      if (c < ngroups) {
        b = bins(c * ROWS);
        if constexpr (ROWS > 1) b |= bins(c * ROWS + 1);
      }
      const unsigned hit = __ballot_sync(0xffffffffu, b != 0);
      if (hit) return g + (__ffs(hit) - 1) * gridDim.x;
    }
    return ngroups;
  };
  // the staged input of a row (thread 0; earlier generic reads of the stage are
  // ordered before the copies by the barrier and the proxy fence)
  auto stage_row = [&](uint32_t l) {
    if constexpr (L::STAGE) {
      const float2 *src = cells(l);
      fence_proxy_async();
      if (S < 0) {
        if (whole) {
          mbar_expect_tx(&s_bar, N / 2 * (unsigned)sizeof(float2));
          bulk_load(stg, src + N / 4, N / 2 * (unsigned)sizeof(float2), &s_bar);
        }
        return;
      }
      uint32_t b = bins(l);
      mbar_expect_tx(&s_bar, min(__popc(b), L::CAP) * TN * (unsigned)sizeof(float2));
      for (int slot = 0; b && slot < L::CAP; ++slot, b &= b - 1)
        bulk_load(stg + slot * TN, src + (__ffs(b) - 1) * TN, TN * (unsigned)sizeof(float2),
                  &s_bar);
    }
  };
  const bool staged = L::STAGE && (S > 0 || whole);
  const float2 w1 = tw(t), w8 = tw(8 * t);
  uint32_t g = next_used(blockIdx.x);
  if (threadIdx.x == 0 && g < ngroups) stage_row(g);
  unsigned phase = 0;
  while (g < ngroups) {
    const uint32_t next = next_used(g + gridDim.x);
    const uint32_t l = g * ROWS + sub;
    const uint32_t occ = bins(l);
    float2 *rp = cells(l);
    if (staged) {
      if (!mbar_wait(&s_bar, phase)) s_abort = 1;
      phase ^= 1u;
    }
    // pass 1
    C2 x[16];
    if constexpr (S > 0) {
      const float2 none = make_float2(0.f, 0.f);
      if (L::STAGE && __popc(occ) <= L::CAP) {  // (block-uniform) the whole input is staged
        const float2 *pa = stg + t, *pb = pa + __popc(occ & 0xffffu) * TN;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
          float2 a = none, b = none;
          if (occ >> m & 1u) {
            a = *pa;
            pa += TN;
          }
          if (occ >> (m + 16) & 1u) {
            b = *pb;
            pb += TN;
          }
          x[m] = pair32<S>(a, b, m);
        }
      } else {
        int sa = 0, sb = __popc(occ & 0xffffu);
        auto in = [&](int m, int &slot) {
          float2 v = none;
          if (occ >> m & 1u) {
            v = L::STAGE && slot < L::CAP ? stg[slot * TN + t] : rp[t + TN * m];
            ++slot;
          }
          return v;
        };
#pragma unroll
        for (int m = 0; m < 16; ++m) {
          const float2 a = in(m, sa), b = in(m + 16, sb);
          x[m] = pair32<S>(a, b, m);
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int mm = m < 8 ? m + 16 : m;  // the one of m, m + 16 in [8, 24)
        const int col = t + TN * mm;
        float2 v;
        if (staged)
          v = stg[t + TN * (mm - 8)];
        else
          v = whole || (col >= ra.lo && col < ra.hi) ? rp[col] : make_float2(0.f, 0.f);
        x[m] = pair32_one<S>(v, m, m >= 8);
      }
    }
    pdft16<S>(x);
    {
      // w^(t k1) for the pair k1 = 2 (4 a + b) + {0, 1}: w^(8 a t), table values (as
      // powers of w^(8 t) they raised a predict's rounding error by up to 5 %), times
      // the pair (w^(2 b t), w^((2 b + 1) t)), powers of w^t
      const float2 w2 = cmul(w1, w1);
      C2 wb = C2{make_float2(1.f, w1.x), make_float2(0.f, w1.y)};
      const float2 w16 = tw(16 * t), w24 = tw(24 * t);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        if (b) wb = pmulc(wb, w2.x, w2.y);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          C2 v = pmul(x[4 * a + b], wb.r, wb.i);
          if (a == 1) v = pmulc(v, w8.x, w8.y);
          if (a == 2) v = pmulc(v, w16.x, w16.y);
          if (a == 3) v = pmulc(v, w24.x, w24.y);
          put(xb + (4 * a + b) * (TN + 1) + t, v);
        }
      }
    }
    sync();  // pass-1 exchange written; the stage read by every thread
    if constexpr (L::STAGE) {
      if (s_abort) {
        if (threadIdx.x == 0) {
          atomicOr(ra.status, kErrTmaTimeout);
          mbar_wait(&s_bar, phase ^ 1u);  // (bounded) the copies still in flight
        }
        return;
      }
      if (threadIdx.x == 0 && next < ngroups) stage_row(next);
    }
    // pass 2: unit pairs u = k + 16 s (k1 = 2 k, 2 k + 1); with R3 = 32 a warp's
    // halves hold s and s + 16 (conflict-free scalar stores below)
    constexpr int U2 = 16 / R2;
    auto unit_s = [](int u) { return R3 == 32 ? (u >> 5) + 16 * ((u >> 4) & 1) : u / 16; };
    C2 y[U2][R2];
#pragma unroll
    for (int i = 0; i < U2; ++i) {
      const int u = t + TN * i, k = u % 16, s = unit_s(u);
#pragma unroll
      for (int m = 0; m < R2; ++m) {
        y[i][m] = get(xb + k * (TN + 1) + s + R3 * m);
      }
      pdft<R2, S>(y[i]);
#pragma unroll
      for (int kp = 1; kp < R2; ++kp) {
        const float4 w = t2[s * kp];
        y[i][kp] = pmul(y[i][kp], make_float2(w.x, w.y), make_float2(w.z, w.w));
      }
    }
    sync();
    if constexpr (R3 < 32) {
#pragma unroll
      for (int i = 0; i < U2; ++i) {
        const int u = t + TN * i, k = u % 16, s = unit_s(u);
#pragma unroll
        for (int kp = 0; kp < R2; ++kp) put(xb + (kp * R3 + s) * 16 + k, y[i][kp]);
      }
      sync();
      // pass 3: unit pairs u = k + 16 k'
      constexpr int U3 = 16 / R3;
#pragma unroll
      for (int i = 0; i < U3; ++i) {
        const int u = t + TN * i, k = u % 16, kp = u / 16;
        C2 z[R3];
#pragma unroll
        for (int s = 0; s < R3; ++s) z[s] = get(xb + (kp * R3 + s) * 16 + k);
        pdft<R3, S>(z);
        const int o0 = 2 * k + 32 * kp, b0 = o0 / TN;
#pragma unroll
        for (int k2 = S > 0 ? R3 / 4 : 0; k2 < (S > 0 ? 3 * R3 / 4 : R3); ++k2) {
          const int o = o0 + 32 * R2 * k2;
          const bool on = S > 0 ? whole || (o >= ra.lo && o < ra.hi)
                                : (occ >> (b0 + k2 * (32 / R3)) & 1u) != 0;
          if (on)
            *reinterpret_cast<float4 *>(rp + o) =
                make_float4(z[k2].r.x, z[k2].i.x, z[k2].r.y, z[k2].i.y);
        }
      }
    } else {
      // k1 = 2 k + {0, 1} at row k + 16 {0, 1}, element s at 2 (s % 16) + s / 16
      float *yr = reinterpret_cast<float *>(xb), *yi = yr + 2 * L::X;
      {
        const int k = t % 16, s = unit_s(t), at = k * 34 + 2 * (s % 16) + s / 16;
#pragma unroll
        for (int kp = 0; kp < R2; ++kp) {
          yr[kp * 32 * 34 + at] = y[0][kp].r.x;
          yr[(kp * 32 + 16) * 34 + at] = y[0][kp].r.y;
          yi[kp * 32 * 34 + at] = y[0][kp].i.x;
          yi[(kp * 32 + 16) * 34 + at] = y[0][kp].i.y;
        }
      }
      sync();
      // pass 3: thread (row, k') holds all 32 elements of one k1
      const int row = t % 32, kp = t / 32;
      const float2 *zr = reinterpret_cast<const float2 *>(yr + (kp * 32 + row) * 34);
      const float2 *zi = reinterpret_cast<const float2 *>(yi + (kp * 32 + row) * 34);
      C2 z[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float2 r = zr[j], im = zi[j];
        z[j] = pair32<S>(make_float2(r.x, im.x), make_float2(r.y, im.y), j);
      }
      pdft16<S>(z);
      const int o0 = (row % 16) * 2 + row / 16 + 32 * kp, b0 = o0 / TN;
#pragma unroll
      for (int c = S > 0 ? R3 / 8 : 0; c < (S > 0 ? 3 * R3 / 8 : R3 / 2); ++c) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k2 = 2 * c + h, o = o0 + 32 * R2 * k2;
          const bool on = S > 0 ? whole || (o >= ra.lo && o < ra.hi)
                                : (occ >> (b0 + k2 * (32 / R3)) & 1u) != 0;
          if (on) rp[o] = h ? make_float2(z[c].r.y, z[c].i.y) : make_float2(z[c].r.x, z[c].i.x);
        }
      }
    }
    sync();  // exchange slots free for the next row
    g = next;
  }
}

// Zero the occupied bins of `bw` 16-byte units (whole rows of occupied tiles when
// bw is 0) of nrows = nb NP ngy rows of `width` units: a warp per row.
__global__ void k_zero_rows(float4 *__restrict__ grid, const uint32_t *__restrict__ mask,
                            int64_t nrows, int width, int ngy, int NP, int b0, int T, int ntv,
                            int bw) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; row < nrows;
       row += stride) {
    const int sp = (int)(row / ngy), r = (int)(row - (int64_t)sp * ngy);
    uint32_t occ = mask[(int64_t)(b0 + sp / NP) * ntv + r / T];
    float4 *dst = grid + row * width;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bw == 0) {
      if (occ)
        for (int i = lane; i < width; i += 32) dst[i] = zero;
      continue;
    }
    for (; occ; occ &= occ - 1) {
      float4 *p = dst + (__ffs(occ) - 1) * bw;
      for (int i = lane; i < bw; i += 32) p[i] = zero;
    }
  }
}

int run_zero_rows(gb_plan *p, void *grid, int b0, int nb, cudaStream_t s) {
  const Geom &g = p->g;
  const int64_t nrows = (int64_t)nb * g.NP * g.ngy;
  const unsigned blocks =
      (unsigned)std::min<int64_t>((nrows + kWarps - 1) / kWarps, (int64_t)p->num_sms * 8);
  // the row kernels read the occupied bins only; cuFFT rows read whole rows
  const int width = p->fft64 ? g.ngx : g.ngx / 2;
  k_zero_rows<<<blocks, kThreads, 0, s>>>(
      reinterpret_cast<float4 *>(grid), p->at<uint32_t>(p->off_rowmask), nrows, width, g.ngy,
      g.NP, b0, g.T, g.ntv, p->row_fft || p->fft64 ? width / 32 : 0);
  GB_LAUNCH_CHECK("k_zero_rows");
  return GB_OK;
}

bool row_kernel_fits(int n, int nx) {
  return n >= 512 && n <= 16384 && (n & (n - 1)) == 0 && 2 * nx <= n;
}

// f(RowLayout<N>, k_rows<N, 1>, k_rows<N, -1>) for the plan's width.
template <typename F>
static int rows_instance(int n, F &&f) {
#define GB_ROWS(N) \
  case N: return f(RowLayout<N>(), k_rows<N, 1>, k_rows<N, -1>);
  switch (n) {
    GB_ROWS(512)
    GB_ROWS(1024)
    GB_ROWS(2048)
    GB_ROWS(4096)
    GB_ROWS(8192)
    default: GB_ROWS(16384)
  }
#undef GB_ROWS
}

int setup_row_kernels(gb_plan *p) {
  if (!p->row_fft) return GB_OK;
  return rows_instance(p->g.ngx, [&](auto L, auto inv, auto pred) {
    int per_sm = 1 << 30;
    for (auto k : {inv, pred}) {
      int n = 0;
      GB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.SMEM));
      GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, L.TH, L.SMEM));
      per_sm = std::min(per_sm, n);
    }
    if (per_sm < 1) {
      set_error("k_rows cannot launch for rows of %d cells", p->g.ngx);
      return (int)GB_ERR_INVALID_ARG;
    }
    p->row_blocks = per_sm * p->num_sms;
    return (int)GB_OK;
  });
}

int run_rows(gb_plan *p, void *grid, int b0, int nb, int dir, cudaStream_t s) {
  const Geom &g = p->g;
  RowArgs ra;
  ra.grid = reinterpret_cast<float2 *>(grid);
  ra.mask = p->at<uint32_t>(p->off_rowmask);
  ra.twx = p->at<float2>(p->off_twx);
  const int64_t nrows = (int64_t)nb * g.NP * g.ngy;
  if (nrows >= (int64_t)1 << 31) {
    set_error("a batch of %d planes x %d pols x %d rows exceeds 2^31 rows", nb, g.NP, g.ngy);
    return GB_ERR_INVALID_ARG;
  }
  ra.nrows = (uint32_t)nrows;
  const auto log2_of = [](int n) {
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
  };
  ra.lgy = log2_of(g.ngy);
  ra.lnp = log2_of(g.NP);
  ra.b0 = b0;
  ra.T = g.T;
  ra.tshift = (g.T & (g.T - 1)) == 0 ? log2_of(g.T) : -1;
  ra.ntv = g.ntv;
  ra.rp = row_perm(p);
  ra.lo = (g.ngx - g.nx) / 2;
  ra.hi = ra.lo + g.nx;
  ra.status = p->status_word();
  return rows_instance(g.ngx, [&](auto L, auto inv, auto pred) {
    const unsigned blocks = std::min<unsigned>(p->row_blocks, ra.nrows / L.ROWS);
    (dir > 0 ? inv : pred)<<<blocks, L.TH, L.SMEM, s>>>(ra);
    GB_LAUNCH_CHECK("k_rows");
    return (int)GB_OK;
  });
}

}  // namespace gb
