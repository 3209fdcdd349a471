// Tile kernels of the FP64 form (k_grid64, k_degrid64).
//
// An FP64 instruction occupies an SM's FP64 pipe for 16 cycles per warp on
// this part (1/64 of the FP32 rate), so both kernels are built around how few
// of them an item and plane need.  Both evaluate every item's 3 W kernel
// values once (an exp and a square root each, about 35 FP64 instructions),
// not per item and plane.
#include <cfloat>

#include "gb_fft.cuh"
#include "gb_plan.cuh"

namespace gb {

// ---------------------------------------------------------------------
// Fixed point.  Kernel values are in Q62 (K = round(k 2^62), 1 saturating at
// 2^62 - 1); a chunk's visibilities are int64 at a power-of-two scale with
// the sum of their magnitudes below 2^61, so a cell's sum cannot overflow.
// A product keeps the high part: with c = ch 2^31 + cl, k = kh 2^31 + kl (kh, kl,
// cl in [0, 2^31)), c k 2^-62 = ch kh + (ch kl + cl kh) 2^-31 + (cl kl) 2^-62, the
// last term below one unit and left out: three 32 x 32 -> 64 bit
// multiply-adds.  A unit is 2^-62 of the largest kernel value and 2^-61 of the
// chunk's sum, against 2^-53 of a double product.
__device__ __forceinline__ long long mul_q62(long long c, long long k) {
  const int ch = (int)(c >> 31), cl = (int)c & 0x7fffffff;
  const int kh = (int)(k >> 31), kl = (int)k & 0x7fffffff;
  long long mid = (long long)ch * kl + 0x40000000LL;
  mid += (long long)cl * kh;
  return (long long)ch * kh + (mid >> 31);
}

__device__ __forceinline__ long long kernel_q62(double k) {
  const long long q = __double2ll_rn(k * 4611686018427387904.0);
  return min(q, 4611686018427387903LL);
}

// Slab range [s_lo, s_hi] whose items reach planes [b0, b0 + nb).
__device__ __forceinline__ void batch_chunks(const Geom &g, const uint32_t *chunk_off, int b0,
                                             int nb, uint32_t &c_begin, uint32_t &c_end) {
  const int ntiles = g.ntu * g.ntv;
  const int wk = g.do_w ? g.W : 1;
  const int lo = b0 - (g.S + wk - 2);
  const int s_lo = lo <= 0 ? 0 : (lo + g.S - 1) / g.S;
  const int s_hi = min(g.nslabs - 1, (b0 + nb - 1) / g.S);
  c_begin = chunk_off[(int64_t)s_lo * ntiles];
  c_end = chunk_off[(int64_t)(s_hi + 1) * ntiles];
}

// Support-normalised ES kernel value r of an item: r in [0, W) the u values,
// [W, 2W) v, [2W, 3W) w (1 on its only plane without w-stacking).
__device__ __forceinline__ double item_kernel(const Geom &g, const ItemD &it, int r) {
  const int dim = r / g.W, a = r - dim * g.W;
  if (dim == 2 && !g.do_w) return 1.0;
  const double d = dim == 0 ? it.du : (dim == 1 ? it.dv : it.dwf);
  return es_kernel(((double)a - d) * (2.0 / (double)g.W), g.beta);
}

// FP64 gridder.  A CTA takes one chunk (up to kChunkItems64 items of one
// (w-slab, uv tile) bucket), caches the items' kernel values and values in
// fixed point, and per w-plane accumulates the chunk's cells in shared
// memory: thread (tx, ty) of the 16 x 16 block owns every sub-grid cell with
// x = tx and y = ty modulo 16.  A support of W <= 16 cells meets each owner
// at most once, so the owners add without atomics and without a barrier
// between items, and a 16-lane row falls in distinct banks for any pitch.
// The plane is then flushed to the grid (touched cells only, inside the
// chunk's bounding box) and the sub-grid left zeroed.  All products are
// integer multiply-adds (mul_q62); FP64 instructions are left to the kernel
// values, the values' conversion and the flush.  Measured on 145,152 items x 4
// pols, W = 13, 972^2 grid: 26.5 ms with a warp per item, kernel values
// evaluated per item and plane and 64-bit shared atomics, 5.0 ms like this.
template <int NP>
__global__ void __launch_bounds__(kThreads)
    k_grid64(const Geom g, const ItemD *__restrict__ items, const double *__restrict__ cvis,
             const Chunk *__restrict__ chunks, const uint32_t *__restrict__ chunk_off, int b0,
             int nb, double2 *__restrict__ grid, uint32_t *__restrict__ counter) {
  constexpr int NC = 2 * NP;  // components: re, im of each pol
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int W = g.W, T = g.T, SW = T + W - 1, SW2 = SW * SW, W3 = 3 * W;
  long long *acc = reinterpret_cast<long long *>(smem_raw);  // [NC][SW][SW]
  long long *kq = acc + NC * SW2;                             // [kChunkItems64][3 W]
  long long *cq = kq + kChunkItems64 * W3;                    // [kChunkItems64][NC]
  __shared__ uint32_t s_loc[kChunkItems64];
  __shared__ int s_first[kMaxSlab + 1];
  __shared__ int s_box[4];  // x_lo, x_hi, y_lo, y_hi (first support cells)
  __shared__ double s_sum[2];
  __shared__ uint32_t s_bad, s_ci;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int ntiles = g.ntu * g.ntv;
  const size_t plane = (size_t)g.ngx * g.ngy;
  uint32_t c_begin, c_end;
  batch_chunks(g, chunk_off, b0, nb, c_begin, c_end);
  for (int i = threadIdx.x; i < NC * SW2; i += kThreads) acc[i] = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      s_ci = c_begin + atomicAdd(counter, 1u);
      s_box[0] = s_box[2] = kMaxTile;
      s_box[1] = s_box[3] = 0;
      s_bad = 0;
    }
    __syncthreads();
    const uint32_t ci = s_ci;
    if (ci >= c_end) break;
    const Chunk ch = chunks[ci];
    const int slab = (int)(ch.bucket / (uint32_t)ntiles);
    const int tile = (int)(ch.bucket - (uint32_t)slab * ntiles);
    const int tv = tile / g.ntu, tu = tile - tv * g.ntu;
    const int kbase = slab * g.S;
    const int n = (int)(ch.end - ch.begin);
    // items run in order of first w-plane: the chunk's planes span from its
    // first item's first plane to its last item's last
    const int lk_first = (int)((items[ch.begin].loc >> 16) & 0xffu);
    const int lk_last = (int)((items[ch.end - 1].loc >> 16) & 0xffu);
    const int k_lo = max(kbase + lk_first, b0);
    const int k_hi = min(min(kbase + lk_last + W, g.nplanes), b0 + nb);
    if (k_lo >= k_hi) {  // (block-uniform) no item reaches this batch's planes
      __syncthreads();   // s_ci read by every thread
      continue;
    }
    // the chunk's sum of max |component| (thread j: item j), its tables
    if (warp < kChunkItems64 / 32) {
      double m = 0.0;
      uint32_t bad = 0;  // pols with a non-finite value
      const int j = threadIdx.x;
      if (j < n) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const double v = fabs(cvis[(size_t)(ch.begin + j) * NC + c]);
          if (v <= DBL_MAX)
            m = fmax(m, v);
          else
            bad |= 1u << (c / 2);
        }
        const uint32_t loc = items[ch.begin + j].loc;
        s_loc[j] = loc;
        atomicMin(&s_box[0], (int)(loc & 0xffu));
        atomicMax(&s_box[1], (int)(loc & 0xffu));
        atomicMin(&s_box[2], (int)((loc >> 8) & 0xffu));
        atomicMax(&s_box[3], (int)((loc >> 8) & 0xffu));
        // s_first[l] = the first item with first plane >= l
        const int lk = (int)((loc >> 16) & 0xffu);
        const int lkp = j == 0 ? -1 : (int)((items[ch.begin + j - 1].loc >> 16) & 0xffu);
        for (int q = lkp + 1; q <= lk; ++q) s_first[q] = j;
        if (j == n - 1)
          for (int q = lk + 1; q <= g.S; ++q) s_first[q] = n;
      }
      for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
      if (lane == 0) s_sum[warp] = m;
      if (bad) atomicOr(&s_bad, bad);
    }
    // kernel values in Q62
    for (int i = threadIdx.x; i < n * W3; i += kThreads) {
      const int jj = i / W3;
      kq[i] = kernel_q62(item_kernel(g, items[ch.begin + jj], i - jj * W3));
    }
    __syncthreads();
    // scale 2^(61 - e) with S < 2^e (S clamped to where the scale is normal)
    const double S = fmax(s_sum[0] + s_sum[1], 0x1p-900);
    const int e = min(((__double2hiint(S) >> 20) & 0x7ff) - 1022, 1023);
    const double scale = __hiloint2double((61 - e + 1023) << 20, 0);
    const double inv = __hiloint2double((e - 61 + 1023) << 20, 0);
    for (int i = threadIdx.x; i < n * NC; i += kThreads) {
      const double v = cvis[(size_t)ch.begin * NC + i];
      // a non-finite value reaches the image through the NaN added below
      cq[i] = fabs(v) <= DBL_MAX ? __double2ll_rn(v * scale) : 0;
    }
    const int x_lo = s_box[0], y_lo = s_box[2];
    const int bw = s_box[1] - x_lo + W, bh = s_box[3] - y_lo + W;
    const uint32_t bad = S <= DBL_MAX ? s_bad : 0xfu;
    if (threadIdx.x == 0 && bad) {
      // a cell of the chunk's own: the transforms read no bin that no item reaches
      int p = tu * T + x_lo, q = tv * T + y_lo;
      while (p >= g.ngx) p -= g.ngx;
      while (q >= g.ngy) q -= g.ngy;
      double2 *cell = grid + (size_t)(k_lo - b0) * NP * plane + (size_t)q * g.ngx + p;
      for (int pol = 0; pol < NP; ++pol)
        if (bad >> pol & 1u)
          atomicAdd(&cell[pol * plane].x, __longlong_as_double(0x7ff8000000000000LL));
    }
    __syncthreads();
    for (int k = k_lo; k < k_hi; ++k) {
      double2 *gplane = grid + (size_t)(k - b0) * NP * plane;
      const int lk_lo = max(0, k - kbase - W + 1), lk_hi = min(g.S - 1, k - kbase);
      const int j_lo = s_first[lk_lo];
      const int j_hi = lk_lo <= lk_hi ? s_first[lk_hi + 1] : j_lo;
      for (int jj = j_lo; jj < j_hi; ++jj) {
        const uint32_t loc = s_loc[jj];
        const int lu = (int)(loc & 0xffu), lv = (int)((loc >> 8) & 0xffu);
        const int a = (tx - lu) & 15, b = (ty - lv) & 15;
        if (a < W && b < W) {
          const long long *kj = kq + jj * W3;
          const int aw = k - (kbase + (int)((loc >> 16) & 0xffu));  // in [0, W) here
          const long long kk = mul_q62(mul_q62(kj[a], kj[W + b]), kj[2 * W + aw]);
          long long *cell = acc + (lv + b) * SW + lu + a;
          const long long *cj = cq + jj * NC;
#pragma unroll
          for (int c = 0; c < NC; ++c) cell[c * SW2] += mul_q62(cj[c], kk);
        }
      }
      __syncthreads();
      for (int i = threadIdx.x; i < bw * bh; i += kThreads) {
        const int by = i / bw, x = x_lo + i - by * bw, y = y_lo + by;
        int p = tu * T + x;
        while (p >= g.ngx) p -= g.ngx;
        int q = tv * T + y;
        while (q >= g.ngy) q -= g.ngy;
        const double sgn = ((p + q) & 1) ? -inv : inv;  // checkerboard
        long long *cell = acc + y * SW + x;
        double2 *dst = gplane + (size_t)q * g.ngx + p;
#pragma unroll
        for (int pol = 0; pol < NP; ++pol) {
          const long long re = cell[2 * pol * SW2], im = cell[(2 * pol + 1) * SW2];
          if ((re | im) != 0) {
            cell[2 * pol * SW2] = 0;
            cell[(2 * pol + 1) * SW2] = 0;
            atomicAdd(&dst[pol * plane].x, sgn * (double)re);
            atomicAdd(&dst[pol * plane].y, sgn * (double)im);
          }
        }
      }
      __syncthreads();
    }
  }
}

size_t grid64_smem_bytes(const Geom &g) {
  const size_t SW = (size_t)g.T + g.W - 1;
  return 8 * (2 * (size_t)g.NP * SW * SW + (size_t)kChunkItems64 * (3 * g.W + 2 * g.NP));
}

// ---------------------------------------------------------------------
// FP64 degridder: warp per item, no block barriers.  A warp takes half a
// chunk (up to 32 items) from the work counter, evaluates the kernel values
// of kDegridGroup items at a time (32 lanes busy) into its own shared memory,
// and then per item: the W x W support cells are dealt to the lanes, lane +
// 32 i being one of NI cells a lane holds; a cell's weight (u times v value,
// checkerboard sign) and grid offset are formed once and reused for the
// item's W planes, whose cells are read straight from the grid (L1 / L2:
// neighbouring items share them).  A plane costs 2 NI + 2 FP64 instructions
// per pol, the W x W x 2 multiply-adds of the sum spread over 32 lanes, and
// the lanes are summed once per item, not once per plane.  The epilogue
// (lane i, item i) rotates back by exp(+2 pi i w tc), conjugates mirrored
// items, applies the pol-frame matrix and weights and writes (the item's
// first batch) or accumulates (later batches).  Measured on 520,192 items x 1
// pol, W = 11, 2048^2 grid: 43.7 ms with each plane's sub-grid staged in
// shared memory and kernel values evaluated per item and plane, 4.9 ms like
// this (FP64 pipe: 1.9 ms of it are the multiply-adds).
constexpr int kDegridGroup = 8;

template <int NP, int NI>
__global__ void __launch_bounds__(kThreads)
    k_degrid64(const Geom g, const ItemD *__restrict__ items, const Chunk *__restrict__ chunks,
               const uint32_t *__restrict__ chunk_off, int b0, int nb,
               const double2 *__restrict__ grid, double2 *__restrict__ vis, int npv,
               const double *__restrict__ wgt, const PolMat pm, const RowPerm rp,
               uint32_t *__restrict__ counter) {
  __shared__ double s_k[kWarps][kDegridGroup * 3 * kMaxSupport];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int W = g.W, T = g.T, W3 = 3 * W;
  const int ntiles = g.ntu * g.ntv;
  const int64_t plane = (int64_t)g.ngx * g.ngy;
  const int wk = g.do_w ? W : 1;
  double *kv = s_k[warp];
  constexpr int kParts = kChunkItems64 / 32;
  uint32_t c_begin, c_end;
  batch_chunks(g, chunk_off, b0, nb, c_begin, c_end);
  // this lane's support cells: (b << 8) | a.  Beyond W x W the last cell, at weight
  // 0: only cells of a support are sure to be written (0 times a NaN is a NaN)
  int ab[NI];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int cell = min(lane + 32 * i, W * W - 1), b = cell / W;
    ab[i] = (b << 8) | (cell - b * W);
  }
  for (;;) {
    uint32_t u = 0;
    if (lane == 0) u = atomicAdd(counter, 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
    const uint32_t ci = c_begin + u / kParts;
    if (ci >= c_end) break;
    const Chunk ch = chunks[ci];
    const uint32_t begin = ch.begin + 32 * (u % kParts);
    if (begin >= ch.end) continue;
    const int n = (int)min(ch.end - begin, 32u);
    const int slab = (int)(ch.bucket / (uint32_t)ntiles);
    const int tile = (int)(ch.bucket - (uint32_t)slab * ntiles);
    const int tv = tile / g.ntu, tu = tile - tv * g.ntu;
    const int kbase = slab * g.S;
    ItemD mine;  // lane i: item i
    mine.idx = 0;
    mine.loc = 0;
    if (lane < n) mine = items[begin + lane];
    double vr[NP], vi[NP];  // lane i: item i's sums
#pragma unroll
    for (int p = 0; p < NP; ++p) vr[p] = vi[p] = 0.0;
    for (int j0 = 0; j0 < n; j0 += kDegridGroup) {
      const int ng = min(kDegridGroup, n - j0);
      __syncwarp();
      for (int i = lane; i < ng * W3; i += 32) {
        const int jj = i / W3;
        kv[i] = item_kernel(g, items[begin + j0 + jj], i - jj * W3);
      }
      __syncwarp();
      for (int jj = 0; jj < ng; ++jj) {
        const uint32_t loc = __shfl_sync(0xffffffffu, mine.loc, j0 + jj);
        const int lu = (int)(loc & 0xffu), lv = (int)((loc >> 8) & 0xffu);
        const int k0 = kbase + (int)((loc >> 16) & 0xffu);
        const int k_lo = max(k0, b0), k_hi = min(k0 + wk, b0 + nb);
        if (k_lo >= k_hi) continue;  // warp-uniform
        const double *kj = kv + jj * W3;
        double w[NI];
        int64_t off[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          const int a = ab[i] & 0xff, b = ab[i] >> 8;
          int p = tu * T + lu + a;
          while (p >= g.ngx) p -= g.ngx;
          int q = tv * T + lv + b;
          while (q >= g.ngy) q -= g.ngy;
          const double k2 = lane + 32 * i < W * W ? kj[a] * kj[W + b] : 0.0;
          w[i] = ((p + q) & 1) ? -k2 : k2;
          off[i] = (int64_t)rp.row(q) * g.ngx + p;
        }
        double ar[NP], ai[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) ar[p] = ai[p] = 0.0;
        for (int k = k_lo; k < k_hi; ++k) {
          const double2 *gp = grid + (int64_t)(k - b0) * NP * plane;
          const double kw = kj[2 * W + k - k0];
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            double2 v[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i) v[i] = __ldg(gp + p * plane + off[i]);
            double sr = w[0] * v[0].x, si = w[0] * v[0].y;
#pragma unroll
            for (int i = 1; i < NI; ++i) {
              sr = fma(w[i], v[i].x, sr);
              si = fma(w[i], v[i].y, si);
            }
            ar[p] = fma(kw, sr, ar[p]);
            ai[p] = fma(kw, si, ai[p]);
          }
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            ar[p] += __shfl_xor_sync(0xffffffffu, ar[p], o);
            ai[p] += __shfl_xor_sync(0xffffffffu, ai[p], o);
          }
          if (lane == j0 + jj) {
            vr[p] = ar[p];
            vi[p] = ai[p];
          }
        }
      }
    }
    const int k0 = kbase + (int)((mine.loc >> 16) & 0xffu);
    if (lane < n && k0 + wk > b0 && k0 < b0 + nb) {
      double2 v[NP];
      // a mirrored item (at -uvw) predicts the conjugate
      const double conj_sign = (mine.loc & kLocFlip) ? -1.0 : 1.0;
#pragma unroll
      for (int p = 0; p < NP; ++p) {  // multiply by conj(ph) = exp(+2 pi i w tc)
        v[p].x = vr[p] * mine.ph.x + vi[p] * mine.ph.y;
        v[p].y = (vi[p] * mine.ph.x - vr[p] * mine.ph.y) * conj_sign;
      }
      const size_t base = (size_t)mine.idx * npv;
      const bool first = k0 >= b0;
      for (int q = 0; q < npv; ++q) {
        double2 o = v[0];
        if (pm.identity) {
#pragma unroll
          for (int p = 1; p < NP; ++p)
            if (p == (q < NP ? q : NP - 1)) o = v[p];
        } else {
          double re = 0.0, im = 0.0;
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const double mr = pm.re[q * pm.nin + p], mi = pm.im[q * pm.nin + p];
            re += mr * v[p].x - mi * v[p].y;
            im += mr * v[p].y + mi * v[p].x;
          }
          o = make_double2(re, im);
        }
        if (wgt) {
          const double x = wgt[base + q];
          o.x *= x;
          o.y *= x;
        }
        if (!first) {
          const double2 prev = vis[base + q];
          o.x += prev.x;
          o.y += prev.y;
        }
        vis[base + q] = o;
      }
    }
  }
}

// ---------------------------------------------------------------------
// host side

template <int NP>
static int launch_grid64_np(gb_plan *p, int b0, int nb, const void *cvis, void *grid,
                            uint32_t *counter, cudaStream_t s) {
  k_grid64<NP><<<p->grid_blocks, kThreads, grid64_smem_bytes(p->g), s>>>(
      p->g, p->at<ItemD>(p->off_items), reinterpret_cast<const double *>(cvis),
      p->at<Chunk>(p->off_chunks), p->at<uint32_t>(p->off_chunk_off), b0, nb,
      reinterpret_cast<double2 *>(grid), counter);
  GB_LAUNCH_CHECK("k_grid64");
  return GB_OK;
}

int launch_grid64(gb_plan *p, int b0, int nb, const void *cvis, void *grid, uint32_t *counter,
                  cudaStream_t s) {
  switch (p->g.NP) {
    case 1: return launch_grid64_np<1>(p, b0, nb, cvis, grid, counter, s);
    case 2: return launch_grid64_np<2>(p, b0, nb, cvis, grid, counter, s);
    default: return launch_grid64_np<4>(p, b0, nb, cvis, grid, counter, s);
  }
}

// Cells per lane of a W x W support (25 .. 256 cells over 32 lanes), rounded
// up to even: one instance per two support widths.
static int degrid64_cells(int W) { return (W * W + 63) / 64 * 2; }

template <int NP, typename F>
static int degrid64_instance(int cells, F &&f) {
  switch (cells) {
    case 2: return f(k_degrid64<NP, 2>);
    case 4: return f(k_degrid64<NP, 4>);
    case 6: return f(k_degrid64<NP, 6>);
    default: return f(k_degrid64<NP, 8>);
  }
}

int launch_degrid64(gb_plan *p, int b0, int nb, const void *grid, const void *wgt,
                    const PolMat &pm, int npv, void *vis, uint32_t *counter, cudaStream_t s) {
  const auto launch = [&](auto k) {
    k<<<p->degrid_blocks, kThreads, 0, s>>>(
        p->g, p->at<ItemD>(p->off_items), p->at<Chunk>(p->off_chunks),
        p->at<uint32_t>(p->off_chunk_off), b0, nb, reinterpret_cast<const double2 *>(grid),
        reinterpret_cast<double2 *>(vis), npv, reinterpret_cast<const double *>(wgt), pm,
        row_perm(p), counter);
    GB_LAUNCH_CHECK("k_degrid64");
    return (int)GB_OK;
  };
  const int cells = degrid64_cells(p->g.W);
  switch (p->g.NP) {
    case 1: return degrid64_instance<1>(cells, launch);
    case 2: return degrid64_instance<2>(cells, launch);
    default: return degrid64_instance<4>(cells, launch);
  }
}

template <int NP>
static int setup_np(gb_plan *p) {
  const size_t smem = grid64_smem_bytes(p->g);
  const int rc = allow_shared_memory(k_grid64<NP>);
  if (rc) return rc;
  int per_sm = 0;
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_grid64<NP>, kThreads, smem));
  if (per_sm < 1) {
    set_error("k_grid64 cannot launch with %zu bytes of shared memory", smem);
    return GB_ERR_INVALID_ARG;
  }
  p->grid_blocks = per_sm * p->num_sms;
  return degrid64_instance<NP>(degrid64_cells(p->g.W), [&](auto k) {
    int blocks = 0;
    GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, kThreads, 0));
    p->degrid_blocks = std::max(blocks, 1) * p->num_sms;
    return (int)GB_OK;
  });
}

int setup_tile_kernels64(gb_plan *p) {
  switch (p->g.NP) {
    case 1: return setup_np<1>(p);
    case 2: return setup_np<2>(p);
    default: return setup_np<4>(p);
  }
}

}  // namespace gb
