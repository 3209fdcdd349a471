// Transforms of the FP64 form for power-of-two grids (k_fft64): rows and columns
// of the w-planes, pruned to what holds data.
//
// An FP64 instruction takes an SM's FP64 pipe 16 cycles per warp on this part, so
// an FP64 transform is bound by its arithmetic, not by memory (a 1024-point line
// costs about 33 instructions a cell, whatever its layout), and what pays is
// not transforming what is zero or dropped:
//   invert   rows: only rows that visibilities reach (occupancy mask), only
//            their occupied bins read, only the image columns kept; then the
//            image columns only (half of the grid's at oversampling 2), rows
//            without visibilities taken as zero, only the image rows kept;
//   predict  the image columns from the image rows (the rest is zero and its
//            first butterflies are left out), only rows that visibilities reach
//            stored; then those rows from their image columns, only occupied
//            bins stored.
// A 2-D transform then costs half of a full one or less: 128 plane-pols of
// 1024^2 inverted in 7.2 ms (54 % of the rows occupied; cuFFT on the 972^2 grids
// that 486^2 images had before: 27.2 ms), 20 planes of 2048^2 predicted in 3.6 ms
// (cuFFT 13.4 ms).
//
// A CTA holds 4096 cells: CB = 4096 / N lines of N = 16 R2 R3, TN = N / 16 threads a
// line, 16 cells a thread, by two nested four-step splits in registers with
// exchanges through shared memory (as k_rows): 16-point DFTs over
// x[t + TN m], times w_N^(t k1); R2-point over s + R3 m, times w_TN^(s k'); R3-point
// over s, giving X[k1 + 16 k' + 16 R2 k2].  Lines are rows (threads along the line)
// or columns (threads across the lines, then along).  The exchange's pitches
// keep 8 lanes of a 16-byte access in distinct banks.
#include "gb_fft.cuh"
#include "gb_plan.cuh"

namespace gb {

__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 cmulc(double2 a, double c, double s) {
  return make_double2(a.x * c - a.y * s, a.x * s + a.y * c);
}
// a * (s i)
template <int S> __device__ __forceinline__ double2 mul_si(double2 a) {
  return S > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

constexpr double kD2 = 0.70710678118654752440;  // cos(pi/4)
constexpr double kDC8 = 0.92387953251128675613; // cos(pi/8)
constexpr double kDS8 = 0.38268343236508977173; // sin(pi/8)

// a * exp(s i pi / 4): two additions and two products
template <int S> __device__ __forceinline__ double2 rot45(double2 a) {
  return S > 0 ? make_double2((a.x - a.y) * kD2, (a.x + a.y) * kD2)
               : make_double2((a.x + a.y) * kD2, (a.y - a.x) * kD2);
}

template <int S> __device__ __forceinline__ void ddft4(double2 *a) {
  const double2 s02 = cadd(a[0], a[2]), d02 = csub(a[0], a[2]);
  const double2 s13 = cadd(a[1], a[3]), d13 = mul_si<S>(csub(a[1], a[3]));
  a[0] = cadd(s02, s13);
  a[2] = csub(s02, s13);
  a[1] = cadd(d02, d13);
  a[3] = csub(d02, d13);
}
// the same for a[0] = a[3] = 0
template <int S> __device__ __forceinline__ void ddft4_mid(double2 *a) {
  const double2 b = a[1], c = a[2], ib = mul_si<S>(b);
  a[0] = cadd(c, b);
  a[2] = csub(c, b);
  a[1] = csub(ib, c);
  a[3] = make_double2(-ib.x - c.x, -ib.y - c.y);
}

template <int S> __device__ __forceinline__ void ddft8(double2 *a) {
  double2 e[4] = {a[0], a[2], a[4], a[6]};
  double2 o[4] = {a[1], a[3], a[5], a[7]};
  ddft4<S>(e);
  ddft4<S>(o);
  const double2 t[4] = {o[0], rot45<S>(o[1]), mul_si<S>(o[2]), rot45<S>(mul_si<S>(o[3]))};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    a[k] = cadd(e[k], t[k]);
    a[k + 4] = csub(e[k], t[k]);
  }
}

// 16 = 4 x 4: n = 4 n1 + n2, k = k1 + 4 k2.  MID: a[0..3] = a[12..15] = 0.
template <int S, bool MID> __device__ __forceinline__ void ddft16(double2 *a) {
  double2 y[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    double2 b[4] = {a[n2], a[4 + n2], a[8 + n2], a[12 + n2]};
    if constexpr (MID)
      ddft4_mid<S>(b);
    else
      ddft4<S>(b);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) y[n2][k1] = b[k1];
  }
  y[1][1] = cmulc(y[1][1], kDC8, S * kDS8);
  y[1][2] = rot45<S>(y[1][2]);
  y[1][3] = cmulc(y[1][3], kDS8, S * kDC8);
  y[2][1] = rot45<S>(y[2][1]);
  y[2][2] = mul_si<S>(y[2][2]);
  y[2][3] = rot45<S>(mul_si<S>(y[2][3]));
  y[3][1] = cmulc(y[3][1], kDS8, S * kDC8);
  y[3][2] = rot45<S>(mul_si<S>(y[3][2]));
  y[3][3] = cmulc(y[3][3], -kDC8, -S * kDS8);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    double2 b[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
    ddft4<S>(b);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) a[k1 + 4 * k2] = b[k2];
  }
}

template <int L, int S> __device__ __forceinline__ void ddft(double2 *a) {
  if constexpr (L == 4) ddft4<S>(a);
  else if constexpr (L == 8) ddft8<S>(a);
  else if constexpr (L == 16) ddft16<S, false>(a);
}

template <int N> struct Shape64;
template <> struct Shape64<128> { static constexpr int R2 = 8, R3 = 1; };
template <> struct Shape64<256> { static constexpr int R2 = 16, R3 = 1; };
template <> struct Shape64<512> { static constexpr int R2 = 8, R3 = 4; };
template <> struct Shape64<1024> { static constexpr int R2 = 8, R3 = 8; };
template <> struct Shape64<2048> { static constexpr int R2 = 16, R3 = 8; };
template <> struct Shape64<4096> { static constexpr int R2 = 16, R3 = 16; };

template <int N> struct Layout64 {
  static constexpr int R2 = Shape64<N>::R2, R3 = Shape64<N>::R3;
  static constexpr int TN = N / 16, CB = 4096 / N;  // threads per line, lines per CTA
  static constexpr int PITCH = TN + 1;              // exchange 1: [16][PITCH]
  // line stride: 16 PITCH raised to 8 / CB (mod 8), or 1 from 8 lines
  static constexpr int WANT = CB >= 8 ? 1 : 8 / CB;
  static constexpr int LS = 16 * PITCH + (WANT & 7);
  static constexpr size_t SMEM = sizeof(double2) * (size_t)CB * LS;
};

struct Fft64Args {
  double2 *grid;           // batch buffer
  const double2 *tw;       // exp(+2 pi i m / N), m < N
  const uint32_t *mask;    // [nplanes][ntv] occupied bins
  int ngx, ngy, NP, b0, T, ntv;
  int lo, n;               // image range [lo, lo + n) along the line
  int olo, on;             // image range across the lines (columns)
};

template <int N, int S, bool ROWS>
__global__ void __launch_bounds__(256, 2) k_fft64(const Fft64Args fa) {
  using L = Layout64<N>;
  constexpr int R2 = L::R2, R3 = L::R3, TN = L::TN, CB = L::CB, BW = N / 32;
  extern __shared__ __align__(16) double2 smem64[];
  const int c = ROWS ? threadIdx.x / TN : threadIdx.x % CB;
  const int t = ROWS ? threadIdx.x % TN : threadIdx.x / CB;
  double2 *ex = smem64 + c * L::LS;
  const uint32_t *pmask;  // this plane's mask
  double2 *line;
  size_t step;            // between a line's cells
  uint32_t bits = 0;      // rows: this row's occupied bins
  bool ok = true;
  if constexpr (ROWS) {
    const uint32_t l = blockIdx.x * CB + c, sp = l / (uint32_t)fa.ngy, q = l - sp * fa.ngy;
    pmask = fa.mask + (size_t)(fa.b0 + sp / fa.NP) * fa.ntv;
    bits = pmask[q / (uint32_t)fa.T];
    if (!__syncthreads_or(bits != 0)) return;  // no row of this CTA holds any
    ok = bits != 0;
    line = fa.grid + (size_t)l * N;
    step = 1;
  } else {
    const int col = blockIdx.x * CB + c;
    ok = col < fa.on;
    pmask = fa.mask + (size_t)(fa.b0 + (int)blockIdx.y / fa.NP) * fa.ntv;
    line = fa.grid + (size_t)blockIdx.y * fa.ngx * N + fa.olo + col;
    step = fa.ngx;
  }
  const auto row_used = [&](int q) { return pmask[(uint32_t)q / (uint32_t)fa.T] != 0; };
  const auto in_image = [&](int i) { return i >= fa.lo && i < fa.lo + fa.n; };
  double2 x[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    x[m] = make_double2(0.0, 0.0);
    if (S < 0 && (m < 4 || m >= 12)) continue;  // outside the image's half
    const int i = t + TN * m;
    bool on;
    if constexpr (S > 0)
      on = ROWS ? (bits >> (i / BW) & 1u) != 0 : ok && row_used(i);
    else
      on = ok && in_image(i);
    if (on) x[m] = line[i * step];
  }
  ddft16<S, S < 0>(x);
  const auto twiddle = [&](double2 v, int m) {
    const double2 w = __ldg(fa.tw + m);
    return cmulc(v, w.x, S > 0 ? w.y : -w.y);
  };
#pragma unroll
  for (int k = 0; k < 16; ++k) ex[k * L::PITCH + t] = k ? twiddle(x[k], t * k) : x[0];
  __syncthreads();
  // stores output o of this line
  const auto put = [&](int o, double2 v) {
    bool on;
    if constexpr (S > 0)
      on = ok && in_image(o);
    else
      on = ROWS ? (bits >> (o / BW) & 1u) != 0 : ok && row_used(o);
    if (on) line[o * step] = v;
  };
  // kept output index range of the last pass (of R)
  const auto kept = [](int k, int R) { return S < 0 || (k >= R / 4 && k < 3 * R / 4); };
  constexpr int U2 = 16 / R2;
  double2 y[U2][R2];
#pragma unroll
  for (int i = 0; i < U2; ++i) {
    const int u = t + TN * i, k1 = u % 16, s = u / 16;
#pragma unroll
    for (int m = 0; m < R2; ++m) y[i][m] = ex[k1 * L::PITCH + s + R3 * m];
    ddft<R2, S>(y[i]);
    if constexpr (R3 == 1) {
#pragma unroll
      for (int k = 0; k < R2; ++k)
        if (kept(k, R2)) put(k1 + 16 * k, y[i][k]);
    } else {
#pragma unroll
      for (int k = 1; k < R2; ++k) y[i][k] = twiddle(y[i][k], 16 * s * k);
    }
  }
  if constexpr (R3 > 1) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < U2; ++i) {
      const int u = t + TN * i, k1 = u % 16, s = u / 16;
#pragma unroll
      for (int k = 0; k < R2; ++k) ex[(k * R3 + s) * 16 + k1] = y[i][k];
    }
    __syncthreads();
    constexpr int U3 = 16 / R3;
#pragma unroll
    for (int i = 0; i < U3; ++i) {
      const int u = t + TN * i, k1 = u % 16, kp = u / 16;
      double2 z[R3];
#pragma unroll
      for (int s = 0; s < R3; ++s) z[s] = ex[(kp * R3 + s) * 16 + k1];
      ddft<R3, S>(z);
#pragma unroll
      for (int k2 = 0; k2 < R3; ++k2)
        if (kept(k2, R3)) put(k1 + 16 * kp + 16 * R2 * k2, z[k2]);
    }
  }
}

// exp(+2 pi i m / n), m < n.
__global__ void k_twiddles64(int n, double2 *__restrict__ tw) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < n) sincospi(2.0 * (double)m / (double)n, &tw[m].y, &tw[m].x);
}

bool fft64_fits(int ng, int n) {
  return ng >= 128 && ng <= 4096 && (ng & (ng - 1)) == 0 && 2 * n <= ng;
}

template <int N, int S, bool ROWS>
static int launch64(const Fft64Args &fa, dim3 grid, cudaStream_t s) {
  k_fft64<N, S, ROWS><<<grid, 256, Layout64<N>::SMEM, s>>>(fa);
  GB_LAUNCH_CHECK("k_fft64");
  return GB_OK;
}

template <bool ROWS>
static int lines64(const Fft64Args &fa, int len, int nlines, int npp, int dir, cudaStream_t s) {
  const unsigned cb = 4096u / (unsigned)len;
  const dim3 grid = ROWS ? dim3((unsigned)nlines / cb * (unsigned)npp)
                         : dim3(((unsigned)nlines + cb - 1) / cb, (unsigned)npp);
#define GB_F64(N) \
  case N: return dir > 0 ? launch64<N, 1, ROWS>(fa, grid, s) : launch64<N, -1, ROWS>(fa, grid, s);
  switch (len) {
    GB_F64(128)
    GB_F64(256)
    GB_F64(512)
    GB_F64(1024)
    GB_F64(2048)
    default: GB_F64(4096)
  }
#undef GB_F64
}

// Twiddle tables (bind).
int init_fft64(gb_plan *p, cudaStream_t s) {
  const int n[2] = {p->g.ngx, p->g.ngy};
  const size_t off[2] = {p->off_twx, p->off_twn};
  for (int i = 0; i < 2; ++i) {
    k_twiddles64<<<(n[i] + kThreads - 1) / kThreads, kThreads, 0, s>>>(n[i],
                                                                      p->at<double2>(off[i]));
    GB_LAUNCH_CHECK("k_twiddles64");
  }
  return GB_OK;
}

int run_fft64(gb_plan *p, int b0, int nb, void *grid, int dir, cudaStream_t s) {
  const Geom &g = p->g;
  Fft64Args rows, cols;
  rows.grid = reinterpret_cast<double2 *>(grid);
  rows.mask = p->at<uint32_t>(p->off_rowmask);
  rows.ngx = g.ngx;
  rows.ngy = g.ngy;
  rows.NP = g.NP;
  rows.b0 = b0;
  rows.T = g.T;
  rows.ntv = g.ntv;
  cols = rows;
  rows.tw = p->at<double2>(p->off_twx);
  cols.tw = p->at<double2>(p->off_twn);
  rows.lo = cols.olo = (g.ngx - g.nx) / 2;
  rows.n = cols.on = g.nx;
  cols.lo = rows.olo = (g.ngy - g.ny) / 2;
  cols.n = rows.on = g.ny;
  const int npp = nb * g.NP;
  // plane-pols are the second dimension of the columns' launch (at most 65535)
  for (int pass = 0; pass < 2; ++pass) {
    int rc = GB_OK;
    if ((dir > 0) == (pass == 0)) {
      rc = lines64<true>(rows, g.ngx, g.ngy, npp, dir, s);
    } else {
      for (int q0 = 0; !rc && q0 < npp; q0 += 65532) {  // a multiple of every NP
        Fft64Args part = cols;
        part.grid += (size_t)q0 * g.ngx * g.ngy;
        part.b0 += q0 / g.NP;
        rc = lines64<false>(part, g.ngy, g.nx, std::min(npp - q0, 65532), dir, s);
      }
    }
    if (rc) return rc;
  }
  return GB_OK;
}

template <int N> static int setup64() {
  for (auto k : {k_fft64<N, 1, true>, k_fft64<N, -1, true>, k_fft64<N, 1, false>,
                 k_fft64<N, -1, false>}) {
    const int rc = allow_shared_memory(k);
    if (rc) return rc;
  }
  return GB_OK;
}

int setup_fft64(gb_plan *p) {
  if (!p->fft64) return GB_OK;
  for (int n : {p->g.ngx, p->g.ngy}) {
    int rc;
    switch (n) {
      case 128: rc = setup64<128>(); break;
      case 256: rc = setup64<256>(); break;
      case 512: rc = setup64<512>(); break;
      case 1024: rc = setup64<1024>(); break;
      case 2048: rc = setup64<2048>(); break;
      default: rc = setup64<4096>(); break;
    }
    if (rc) return rc;
  }
  return GB_OK;
}

}  // namespace gb
