// Predict (dirty2ms): model image -> visibilities.
//
// Per call:   k_prep_image  image * correction, into [pol][y][x] order.
// Per batch of w-planes, one of
//             columns, rows (FP32 form, gb_fft.cu and gb_rows.cu) the screens
//                           image * exp(+2 pi i w_k (n-1-tc)) fused into the
//                           columns' first step; occupied bins written;
//             k_screen_block, k_fft64 (FP64 form, gb_fft64.cu) the screened
//                           image, then its transform; occupied bins written;
//             k_screen_pad, cuFFT every grid cell of every plane written once,
//                           the central block screened, the rest 0 (no separate
//                           memset pass); 2-D c2c, e^{-2 pi i}.
//             Then
//             k_degrid_warp one CTA per work chunk (FP32 form): every item's
//                           kernel values cached once per chunk; supports
//                           of up to 7 cells from planes staged in shared
//                           memory, a few at a time (degrid_staged_chunk);
//                           wider ones a warp per item straight from the
//                           grid (a lane group's eight lanes read one
//                           64-byte row segment), weighted and summed over
//                           the lanes with shuffles.  k_degrid64 (FP64 form) is in
//                           gb_fp64.cu.  The
//                           epilogue rotates back by exp(+2 pi i w tc),
//                           conjugates mirrored items, applies the pol-frame
//                           matrix and weights and writes (first batch of
//                           the item) or accumulates (later batches) in place.
#include <cufft.h>

#include "gb_async.cuh"
#include "gb_fft.cuh"
#include "gb_plan.cuh"

namespace gb {

int run_fft(gb_plan *p, int nb, void *data, int dir, cudaStream_t s);
int setup_grid_kernels(gb_plan *p);

template <typename R>
__global__ void k_prep_image(const Geom g, const R *__restrict__ dirty, int layout,
                             const R *__restrict__ corr, R *__restrict__ img) {
  __shared__ R tile[32][33];
  const int64_t npix = (int64_t)g.nx * g.ny;
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32, p = blockIdx.z;
  if (layout == GB_LAYOUT_XY) {
    // read dirty[p][x][y] rows (y fastest) into the tile
    for (int j = threadIdx.y; j < 32; j += 8) {
      const int ix = bx + j, iy = by + threadIdx.x;
      if (ix < g.nx && iy < g.ny) tile[threadIdx.x][j] = dirty[p * npix + (int64_t)ix * g.ny + iy];
    }
    __syncthreads();
  }
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int iy = by + j, ix = bx + threadIdx.x;
    if (iy < g.ny && ix < g.nx) {
      const int64_t i = (int64_t)iy * g.nx + ix;
      const R v = layout == GB_LAYOUT_XY ? tile[j][threadIdx.x] : dirty[p * npix + i];
      img[p * npix + i] = v * corr[i];
    }
  }
}

// The screened image into the image block of every plane (k_fft64 reads nothing
// else of it).
template <typename R, int NP>
__global__ void __launch_bounds__(kThreads)
    k_screen_block(const Geom g, const R *__restrict__ img, const double *__restrict__ tprime,
                   int b0, int nb, typename Traits<R>::C *__restrict__ grid) {
  using C = typename Traits<R>::C;
  const int64_t npix = (int64_t)g.nx * g.ny, plane = (int64_t)g.ngx * g.ngy;
  const int ox = (g.ngx - g.nx) / 2, oy = (g.ngy - g.ny) / 2;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const double2 *tab = g.do_w ? screen_table<R>() : nullptr;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npix; i += stride) {
    const int iy = (int)(i / g.nx), ix = (int)(i - (int64_t)iy * g.nx);
    C *dst = grid + (int64_t)(iy + oy) * g.ngx + ix + ox;
    R v[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) v[p] = img[p * npix + i];
    PlaneScreen<R> ps(tab);
    if (g.do_w) ps.start(g, b0, tprime[i]);
    for (int j = 0; j < nb; ++j) {
      if (g.do_w) {
        ps.plane(j);
      } else {
        ps.c = (R)1;
        ps.s = (R)0;
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        C z;
        z.x = v[p] * ps.c;
        z.y = v[p] * ps.s;
        dst[((int64_t)j * NP + p) * plane] = z;
      }
    }
  }
}

template <typename R, int NP>
__global__ void __launch_bounds__(kThreads)
    k_screen_pad(const Geom g, const R *__restrict__ img, const double *__restrict__ tprime,
                 int b0, int nb, typename Traits<R>::C *__restrict__ grid) {
  using C = typename Traits<R>::C;
  const int64_t npix = (int64_t)g.nx * g.ny;
  const int ox = (g.ngx - g.nx) / 2, oy = (g.ngy - g.ny) / 2;
  const int64_t plane = (int64_t)g.ngx * g.ngy;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const double2 *tab = g.do_w ? screen_table<R>() : nullptr;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < plane; i += stride) {
    const int my = (int)(i / g.ngx), mx = (int)(i - (int64_t)my * g.ngx);
    const int ix = mx - ox, iy = my - oy;
    if (ix >= 0 && ix < g.nx && iy >= 0 && iy < g.ny) {
      const int64_t pi = (int64_t)iy * g.nx + ix;
      R v[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) v[p] = img[p * npix + pi];
      if (g.do_w) {
        PlaneScreen<R> ps(tab);
        ps.start(g, b0, tprime[pi]);
        for (int j = 0; j < nb; ++j) {
          ps.plane(j);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            C z;
            z.x = v[p] * ps.c;
            z.y = v[p] * ps.s;
            grid[((int64_t)j * NP + p) * plane + i] = z;
          }
        }
      } else {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          C z;
          z.x = v[p];
          z.y = (R)0;
          grid[(int64_t)p * plane + i] = z;
        }
      }
    } else {
      C z;
      z.x = (R)0;
      z.y = (R)0;
      for (int j = 0; j < nb; ++j)
#pragma unroll
        for (int p = 0; p < NP; ++p) grid[((int64_t)j * NP + p) * plane + i] = z;
    }
  }
}

// The end of a chunk's degridding (thread i, item i, NT threads): the item's sums
// rotated back by exp(+2 pi i w tc), conjugated if it is mirrored, through the
// pol-frame matrix and weights, written (the item's first batch of w-planes) or
// accumulated (later batches).  Every thread's sums in sacc are complete.
template <int NP, int NT>
__device__ __forceinline__ void degrid_epilogue(const Geom &g, const ItemF *__restrict__ items,
                                                const Chunk &ch, int kbase, int b0, int nb,
                                                float2 *__restrict__ vis, int npv,
                                                const float *__restrict__ wgt, const PolMat &pm,
                                                const float2 *sacc) {
  const int n = (int)(ch.end - ch.begin), wk = g.do_w ? g.W : 1;
  for (int jj = threadIdx.x; jj < n; jj += NT) {
    const ItemF it = items[ch.begin + jj];
    const int k0 = kbase + (int)((it.loc >> 16) & 0xffu);
    if (!(k0 + wk > b0 && k0 < b0 + nb)) continue;
    float2 v[NP];
    // a mirrored item (at -uvw) predicts the conjugate
    const float conj_sign = (it.loc & kLocFlip) ? -1.f : 1.f;
#pragma unroll
    for (int p = 0; p < NP; ++p) {  // multiply by conj(ph) = exp(+2 pi i w tc)
      const float2 a = sacc[jj * NP + p];
      v[p].x = a.x * it.ph.x + a.y * it.ph.y;
      v[p].y = (a.y * it.ph.x - a.x * it.ph.y) * conj_sign;
    }
    const size_t vbase = (size_t)it.idx * npv;
    const bool first = k0 >= b0;
    for (int q = 0; q < npv; ++q) {
      float2 o = v[0];
      if (pm.identity) {
#pragma unroll
        for (int p = 1; p < NP; ++p)
          if (p == (q < NP ? q : NP - 1)) o = v[p];
      } else {
        float re = 0.f, im = 0.f;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const float mr = pm.fre[q * pm.nin + p], mi = pm.fim[q * pm.nin + p];
          re += mr * v[p].x - mi * v[p].y;
          im += mr * v[p].y + mi * v[p].x;
        }
        o = make_float2(re, im);
      }
      if (wgt) {
        const float w = wgt[vbase + q];
        o.x *= w;
        o.y *= w;
      }
      if (first) {
        vis[vbase + q] = o;
      } else {
        float2 prev = vis[vbase + q];
        prev.x += o.x;
        prev.y += o.y;
        vis[vbase + q] = prev;
      }
    }
  }
}

// FP32 degridder, warp per item, reading the grid directly (no staging
// pass).  A CTA takes a work chunk (up to kChunkItems items of one (w-slab,
// uv tile) bucket).  Once per chunk it caches in shared memory every item's
// kernel values -- the u and v values with the checkerboard sign (-1)^(p+q)
// folded in, and the w values -- and the chunk's grid rows (wrapped, in the
// grid's row order, times the row length) and columns.  Then per w-plane k
// each warp takes the items reaching k whose chunk index is congruent to the
// warp modulo the warp count (an item always meets the same warp, so its
// running sums need no barrier between planes), two items at a time: lane
// (g, a) reads column a of the item's support rows of its pols straight
// from the grid -- the eight lanes of a group read eight adjacent cells of
// one row, one 64-byte segment -- weights them by the v values, folds in its
// u value, and the lanes of a group are summed by shuffles.  The tile's
// cells of one plane stay in L1 while the chunk's items pass over them.
// Per item-plane: W reads and 2 W FMAs per lane and one shuffle reduction,
// with no shared-memory staging and no per-plane barrier.  For supports of 8 to
// 16 cells and tiles that cannot be staged.
template <int NP, int AW>
__device__ __forceinline__ void degrid_warp_chunk(
    const Geom &g, const ItemF *__restrict__ items, const Chunk ch, int b0, int nb,
    const float2 *__restrict__ grid, float2 *__restrict__ vis, int npv,
    const float *__restrict__ wgt, const PolMat &pm, const RowPerm &rp, float *kc, float2 *sacc,
    int *s_first, int *s_rowoff, int *s_col) {
  using LM = LaneMap<NP, AW>;
  constexpr int KS = kcache_stride(AW);
  constexpr int kMaxRows = (AW + LM::RS - 1) / LM::RS;
  const int W = g.W, T = g.T, SW = T + W - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LM lm(lane);
  const bool lane_in = lm.a < W;
  const float scale_u = 2.f / (float)W;
  const float beta = (float)g.beta;
  const int ntiles = g.ntu * g.ntv;
  const int64_t plane = (int64_t)g.ngx * g.ngy;
  const int wk = g.do_w ? W : 1;
  const int slab = (int)(ch.bucket / (uint32_t)ntiles);
  const int tile = (int)(ch.bucket - (uint32_t)slab * ntiles);
  const int tv = tile / g.ntu, tu = tile - tv * g.ntu;
  const int kbase = slab * g.S;
  // a chunk's items run in order of first w-plane (sort_key): its planes
  // span from its first item's first plane to its last item's last
  const int lk_first = (int)((items[ch.begin].loc >> 16) & 0xffu);
  const int lk_last = (int)((items[ch.end - 1].loc >> 16) & 0xffu);
  const int k_lo = max(kbase + lk_first, b0);
  const int k_hi = min(min(kbase + lk_last + wk, g.nplanes), b0 + nb);
  if (k_lo >= k_hi) return;  // (block-uniform) no item reaches this batch's planes
  const int n = (int)(ch.end - ch.begin);
  for (int i = threadIdx.x; i < 2 * SW; i += kThreads) {
    if (i < SW) {
      int q = tv * T + i;
      while (q >= g.ngy) q -= g.ngy;
      s_rowoff[i] = rp.row(q) * g.ngx;
    } else {
      int pc = tu * T + (i - SW);
      while (pc >= g.ngx) pc -= g.ngx;
      s_col[i - SW] = pc;
    }
  }
  const int tpar = ((tu + tv) * T) & 1;  // checkerboard parity of the tile origin
  for (int jj = threadIdx.x; jj < n; jj += kThreads) {
    const ItemF it = items[ch.begin + jj];
    float *c = kc + jj * KS;
    c[0] = __uint_as_float(it.loc);
    const int lu = (int)(it.loc & 0xffu), lv = (int)((it.loc >> 8) & 0xffu);
#pragma unroll
    for (int a = 0; a < AW; ++a) {
      const bool in = a < W;
      const float x = in ? es_kernel(((float)a - it.du) * scale_u, beta) : 0.f;
      const float y = in ? es_kernel(((float)a - it.dv) * scale_u, beta) : 0.f;
      c[4 + a] = ((lu + a + tpar) & 1) ? -x : x;
      c[4 + AW + a] = ((lv + a) & 1) ? -y : y;
      c[4 + 2 * AW + a] = in ? (g.do_w ? es_kernel(((float)a - it.dwf) * scale_u, beta) : 1.f)
                             : 0.f;
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) sacc[jj * NP + p] = make_float2(0.f, 0.f);
    // s_first[l] = the first item with lk >= l (the items reaching plane k
    // are then one run)
    const int lk = (int)((it.loc >> 16) & 0xffu);
    const int lkp = jj == 0 ? -1 : (int)((items[ch.begin + jj - 1].loc >> 16) & 0xffu);
    for (int q = lkp + 1; q <= lk; ++q) s_first[q] = jj;
    if (jj == n - 1)
      for (int q = lk + 1; q <= g.S; ++q) s_first[q] = n;
  }
  __syncthreads();
  for (int k = k_lo; k < k_hi; ++k) {
    const float2 *gplane = grid + (int64_t)(k - b0) * NP * plane;
    const int lk_lo = max(0, k - kbase - wk + 1), lk_hi = min(g.S - 1, k - kbase);
    if (lk_lo > lk_hi) continue;
    const int jlo = s_first[lk_lo], jhi = s_first[lk_hi + 1];
    // this warp's items: index congruent to the warp
    for (int j0 = jlo + ((warp - jlo) % kWarps + kWarps) % kWarps; j0 < jhi;
         j0 += 2 * kWarps) {
      const bool two = j0 + kWarps < jhi;  // warp-uniform
      float sr[2][LM::NPL], si[2][LM::NPL], kf[2];
      float kv[2][LM::RS == 1 ? AW : 1];
      const float2 *base[2][LM::NPL];
      const float *kjs[2];
      int lvs[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int jj = (u == 1 && two) ? j0 + kWarps : j0;
        const float *kj = kc + jj * KS;
        kjs[u] = kj;
        const uint32_t loc = __float_as_uint(kj[0]);
        const int lu = (int)(loc & 0xffu);
        lvs[u] = (int)((loc >> 8) & 0xffu);
        const int aw = k - (kbase + (int)((loc >> 16) & 0xffu));  // in [0, wk) here
        kf[u] = kj[4 + 2 * AW + aw] * kj[4 + lm.a];               // kw(aw) ku(a), signed
        if constexpr (LM::RS == 1) {
#pragma unroll
          for (int q = 0; q < AW; q += 4) {
            const float4 t = *reinterpret_cast<const float4 *>(kj + 4 + AW + q);
            kv[u][q] = t.x;
            kv[u][q + 1] = t.y;
            kv[u][q + 2] = t.z;
            kv[u][q + 3] = t.w;
          }
        }
        const int col = s_col[lu + (lane_in ? lm.a : 0)];
#pragma unroll
        for (int i = 0; i < LM::NPL; ++i) {
          base[u][i] = gplane + lm.pol(i) * plane + col;
          sr[u][i] = 0.f;
          si[u][i] = 0.f;
        }
      }
#pragma unroll
      for (int r = 0; r < kMaxRows; ++r) {
        if (LM::RS == 1 && r >= W) break;  // warp-uniform
        const int b = lm.r0 + r * LM::RS;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (u == 1 && !two) break;  // warp-uniform
          if (b < W && lane_in) {
            float kvb;
            if constexpr (LM::RS == 1)
              kvb = kv[u][r];
            else
              kvb = kjs[u][4 + AW + b];
            const int ro = s_rowoff[lvs[u] + b];
#pragma unroll
            for (int i = 0; i < LM::NPL; ++i) {
              const float2 v = __ldg(base[u][i] + ro);
              sr[u][i] += kvb * v.x;
              si[u][i] += kvb * v.y;
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (u == 1 && !two) break;  // warp-uniform
        const int jj = u == 1 ? j0 + kWarps : j0;
#pragma unroll
        for (int i = 0; i < LM::NPL; ++i) {
          float xr = sr[u][i] * kf[u], xi = si[u][i] * kf[u];
#pragma unroll
          for (int o = 1; o < AW; o <<= 1) {
            xr += __shfl_xor_sync(0xffffffffu, xr, o);
            xi += __shfl_xor_sync(0xffffffffu, xi, o);
          }
          if (NP < LM::G) {  // groups sharing a pol hold different rows
#pragma unroll
            for (int o = AW * NP; o < 32; o <<= 1) {
              xr += __shfl_xor_sync(0xffffffffu, xr, o);
              xi += __shfl_xor_sync(0xffffffffu, xi, o);
            }
          }
          if (lm.a == 0 && lm.r0 == 0) {  // only this warp touches item jj
            float2 &s = sacc[jj * NP + lm.pol(i)];
            s.x += xr;
            s.y += xi;
          }
        }
      }
    }
  }
  __syncthreads();  // every item's sums complete
  degrid_epilogue<NP, kThreads>(g, items, ch, kbase, b0, nb, vis, npv, wgt, pm, sacc);
}

// FP32 degridder for supports of up to 7 cells, from staged planes.  A CTA of 16
// warps takes a work chunk and stages, window by window of P = 8 / NP w-planes,
// the tile's sub-grid (SW x SW cells of each plane and pol: 8 sheets) in shared
// memory by 16-byte cp.async, the next window's copies in flight while this
// one's items are summed.  Eight lanes per item, four items per warp: lane (par,
// seg) takes the cell pair 2 seg, 2 seg + 1 (counted from the item's first cell
// rounded down to even) of rows par, par + 2, par + 4, par + 6, so a sheet's
// W x W support is four 16-byte shared loads and eight packed multiply-adds for
// four items.  A quarter-warp reads two adjacent rows of 64 bytes; rows are pitched to
// 64 bytes modulo 128, so its lanes fall in distinct banks.  Weights (u times v
// value, checkerboard sign folded in) are formed once per item and window, and
// its lanes summed once, by a transposing reduction.  What bounds it is the
// shared-memory pipe: 16 wavefronts of cells per item and plane (NP = 4), where
// reading the grid through L1 cost a wavefront per (row, pol) line plus the item's
// constants per plane, about 64 cycles.  Measured: 33.5M items x 4 pols, 42 planes of
// 8192^2, 51.5 -> 27.6 ms; 9.9M items x 4 pols in smaller chunks, 18.5 -> 12.8; 4.2M
// items x 1 pol, 2.74 -> 1.18 ms.
constexpr int kStageSheets = 8;                 // sheets (plane x pol) of one window
constexpr int kStageWarps = 16;
constexpr int kStageMaxW = 7;
constexpr int kStageItem = 25;                  // cached floats: loc, 0, ku[8], kv[8], kw[7]
// Buckets of fewer items are read through L1 / L2: a window's copies cost about as
// much as 20 items' sums.
constexpr int kStageMinItems = 24;

__device__ __forceinline__ bool alone_in_bucket(const Chunk &ch, const uint32_t *chunk_off) {
  return chunk_off[(int64_t)ch.bucket + 1] - chunk_off[ch.bucket] == 1;
}

// Cells per staged row: SW raised to 64 bytes modulo 128.
inline __host__ __device__ int stage_pitch(int SW) { return (SW + 7) / 16 * 16 + 8; }

inline __host__ __device__ size_t stage_bytes(int SW) {
  return (size_t)2 * kStageSheets * SW * stage_pitch(SW) * sizeof(float2);
}

// v[0 .. NV) summed over groups of eight lanes; the sum of value idx lands in v[0]
// of the group's lanes l with l / (8 / NV) = idx.
template <int NV> __device__ __forceinline__ void reduce8(float *v, int lane) {
  int off = 4;
#pragma unroll
  for (int h = NV / 2; h > 0; h /= 2, off /= 2) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const float send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
#pragma unroll
  for (int o = 4 / NV; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

// Chunks of few items, supports of up to 7 cells, with w-stacking (as every staged
// plan): a warp per item over all its planes, the cells of a 7 x 7 frame dealt to the lanes (two each), their weights
// and offsets formed once and the planes' cells read straight from the grid with
// no wait between planes; one reduction per item.
template <int NP>
__device__ __forceinline__ void degrid_sparse_chunk(
    const Geom &g, const ItemF *__restrict__ items, const Chunk &ch, int b0, int nb,
    const float2 *__restrict__ grid, float2 *__restrict__ vis, int npv,
    const float *__restrict__ wgt, const PolMat &pm, const RowPerm &rp, float2 *sacc) {
  constexpr int NV = 2 * NP;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int W = g.W, T = g.T, n = (int)(ch.end - ch.begin);
  const int ntiles = g.ntu * g.ntv;
  const int64_t plane = (int64_t)g.ngx * g.ngy;
  const int slab = (int)(ch.bucket / (uint32_t)ntiles);
  const int tile = (int)(ch.bucket - (uint32_t)slab * ntiles);
  const int tv = tile / g.ntu, tu = tile - tv * g.ntu, kbase = slab * g.S;
  const int dim = lane / 7, a_k = lane - 7 * dim;  // lanes 0 .. 20: the kernel values
  for (int jj = warp; jj < n; jj += kStageWarps) {
    const ItemF it = items[ch.begin + jj];
    const int lu = (int)(it.loc & 0xffu), lv = (int)((it.loc >> 8) & 0xffu);
    const int k0 = kbase + (int)((it.loc >> 16) & 0xffu);
    const int k_lo = max(k0, b0), k_hi = min(k0 + W, b0 + nb);
    const float d = dim == 0 ? it.du : (dim == 1 ? it.dv : it.dwf);
    float val = 0.f;
    if (dim < 3 && a_k < W) val = es_kernel(((float)a_k - d) * (2.f / (float)W), (float)g.beta);
    float2 w[2];
    int64_t off[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = min(lane + 32 * i, 48), b = c / 7, a = c - 7 * b;
      const float ku = __shfl_sync(0xffffffffu, val, a), kv = __shfl_sync(0xffffffffu, val, 7 + b);
      // cells past the support (and the second cells past 49): weight 0, any
      // cell of the support
      int p = tu * T + lu + min(a, W - 1), q = tv * T + lv + min(b, W - 1);
      while (p >= g.ngx) p -= g.ngx;
      while (q >= g.ngy) q -= g.ngy;
      float f = lane + 32 * i < 49 ? ku * kv : 0.f;
      if ((p + q) & 1) f = -f;
      w[i] = make_float2(f, f);
      off[i] = (int64_t)rp.row(q) * g.ngx + p;
    }
    float2 acc[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) acc[p] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int k = k_lo; k < k_hi; ++k) {
      const float2 *gp = grid + (int64_t)(k - b0) * NP * plane;
      const float kw = __shfl_sync(0xffffffffu, val, 14 + k - k0);
      const float2 kw2 = make_float2(kw, kw);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const float2 s = __fmul2_rn(__ldg(gp + p * plane + off[0]), w[0]);
        acc[p] = __ffma2_rn(__ffma2_rn(__ldg(gp + p * plane + off[1]), w[1], s), kw2, acc[p]);
      }
    }
    float sum[NV];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      sum[2 * p] = acc[p].x;
      sum[2 * p + 1] = acc[p].y;
    }
    reduce8<NV>(sum, lane);
    sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 8);
    sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 16);
    if (lane < 8 && lane % (8 / NV) == 0)
      reinterpret_cast<float *>(sacc + jj * NP)[lane / (8 / NV)] = sum[0];
  }
  __syncthreads();  // every item's sums complete
  degrid_epilogue<NP, 32 * kStageWarps>(g, items, ch, kbase, b0, nb, vis, npv, wgt, pm, sacc);
}

template <int NP>
__device__ __forceinline__ void degrid_staged_chunk(
    const Geom &g, const ItemF *__restrict__ items, const Chunk ch, int b0, int nb,
    const float2 *__restrict__ grid, float2 *__restrict__ vis, int npv,
    const float *__restrict__ wgt, const PolMat &pm, const RowPerm &rp, bool alone,
    unsigned char *smem, int *s_first, int *s_rowoff) {
  constexpr int P = kStageSheets / NP, NV = 2 * NP, NT = 32 * kStageWarps;
  const int W = g.W, T = g.T, SW = T + W - 1, pitch = stage_pitch(SW), hp = pitch / 2;
  float4 *sheets = reinterpret_cast<float4 *>(smem);  // [2][kStageSheets][SW][hp] cell pairs
  float *kc = reinterpret_cast<float *>(smem + stage_bytes(SW));
  float2 *sacc = reinterpret_cast<float2 *>(kc + kChunkItems * kStageItem);
  const int n = (int)(ch.end - ch.begin);
  // by the size of the bucket, not of a full bucket's last chunk: which items fall
  // in that one varies from bind to bind, the order of an item's sum must not
  if (alone && n < kStageMinItems) {  // block-uniform
    degrid_sparse_chunk<NP>(g, items, ch, b0, nb, grid, vis, npv, wgt, pm, rp, sacc);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float scale_u = 2.f / (float)W, beta = (float)g.beta;
  const int ntiles = g.ntu * g.ntv;
  const int64_t plane = (int64_t)g.ngx * g.ngy;
  const int slab = (int)(ch.bucket / (uint32_t)ntiles);
  const int tile = (int)(ch.bucket - (uint32_t)slab * ntiles);
  const int tv = tile / g.ntu, tu = tile - tv * g.ntu;
  const int kbase = slab * g.S;
  // items run in order of first w-plane: the chunk's planes span from its
  // first item's first plane to its last item's last
  const int lk_first = (int)((items[ch.begin].loc >> 16) & 0xffu);
  const int lk_last = (int)((items[ch.end - 1].loc >> 16) & 0xffu);
  const int k_lo = max(kbase + lk_first, b0);
  const int k_hi = min(min(kbase + lk_last + W, g.nplanes), b0 + nb);
  if (k_lo >= k_hi) return;  // (block-uniform) no item reaches this batch's planes
  for (int i = threadIdx.x; i < SW; i += NT) {
    int q = tv * T + i;
    while (q >= g.ngy) q -= g.ngy;
    s_rowoff[i] = rp.row(q) * g.ngx;
  }
  __syncthreads();
  // Windows start at multiples of P planes of the batch, whatever the chunk's
  // first plane, so an item's sum is formed in the same order in every chunk.
  const auto window_end = [&](int k) { return min(b0 + ((k - b0) / P + 1) * P, k_hi); };
  // The copies of the window from plane k, 16 bytes each, the cell pairs of all sheets'
  // rows dealt to the threads in order (thread i takes pairs i, i + NT, ...).  An
  // odd SW takes one cell more, which the transforms have written (the mask
  // rounds up to pairs).  (One bulk copy per 304-byte row was slower: 300 issues a
  // window from one warp held the others up, 36.6 -> 54 ms.)
  const int pairs = (SW + 1) / 2, step_row = NT / pairs, step_pair = NT - step_row * pairs;
  const int row_0 = threadIdx.x / pairs, pair_0 = threadIdx.x - row_0 * pairs;
  const auto stage = [&](int k, int buf) {
    const int rows = (window_end(k) - k) * NP * SW;
    const float2 *src = grid + (int64_t)(k - b0) * NP * plane;
    float4 *dst = sheets + (size_t)buf * kStageSheets * SW * hp;
    int pair = pair_0, row = row_0;  // row inside the sheet `src` points to
    for (int r = row_0; r < rows;) {
      while (row >= SW) {
        row -= SW;
        src += plane;
      }
      int col = tu * T + 2 * pair;
      if (col >= g.ngx) col -= g.ngx;
      cp_async16(dst + r * hp + pair, src + s_rowoff[row] + col);
      pair += step_pair;
      const int carry = pair >= pairs;
      pair -= carry ? pairs : 0;
      r += step_row + carry;
      row += step_row + carry;
    }
    cp_async_commit();
  };
  stage(k_lo, 0);
  const int tpar = ((tu + tv) * T) & 1;  // checkerboard parity of the tile origin
  for (int i = threadIdx.x; i < 3 * n; i += NT) {  // thread (item, dimension)
    const int dim = i / n, jj = i - dim * n;
    const ItemF it = items[ch.begin + jj];
    float *c = kc + jj * kStageItem;
    const int first = dim == 0 ? (int)(it.loc & 0xffu) + tpar : (int)((it.loc >> 8) & 0xffu);
    const float d = dim == 0 ? it.du : (dim == 1 ? it.dv : it.dwf);
    float *k = c + 2 + 8 * dim;
#pragma unroll
    for (int a = 0; a < 7; ++a) {
      const float x = a < W ? es_kernel(((float)a - d) * scale_u, beta) : 0.f;
      k[a] = dim < 2 && ((first + a) & 1) ? -x : x;
    }
    if (dim < 2) k[7] = 0.f;
    if (dim == 0) {
      c[0] = __uint_as_float(it.loc);
      c[1] = 0.f;
      // s_first[l] = the first item with lk >= l (the items reaching plane k
      // are then one run)
      const int lk = (int)((it.loc >> 16) & 0xffu);
      const int lkp = jj == 0 ? -1 : (int)((items[ch.begin + jj - 1].loc >> 16) & 0xffu);
      for (int q = lkp + 1; q <= lk; ++q) s_first[q] = jj;
      if (jj == n - 1)
        for (int q = lk + 1; q <= g.S; ++q) s_first[q] = n;
    }
    if (dim == 1)
#pragma unroll
      for (int p = 0; p < NP; ++p) sacc[jj * NP + p] = make_float2(0.f, 0.f);
  }
  const int l8 = lane & 7, par = l8 >> 2, seg = l8 & 3;
  // this lane's cell pair of its four rows (rows past the support: any finite
  // cells, weight 0; so is a pair past it, whatever the parity of the first cell)
  int off[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) off[i] = min(par + 2 * i, W - 1) * hp + (2 * seg > W ? 0 : seg);
  int buf = 0;
  for (int k = k_lo, k_next; k < k_hi; k = k_next, buf ^= 1) {
    k_next = window_end(k);
    if (k_next < k_hi) {
      stage(k_next, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();  // window staged (and, first, the item cache written)
    const int np = k_next - k;
    // items whose support reaches a plane of the window
    const int lk_lo = max(0, k - kbase - W + 1), lk_hi = min(g.S - 1, k + np - 1 - kbase);
    const int jlo = s_first[min(lk_lo, g.S)], jhi = lk_lo <= lk_hi ? s_first[lk_hi + 1] : jlo;
    const float4 *win = sheets + (size_t)buf * kStageSheets * SW * hp;
    for (int j0 = jlo + 4 * warp; j0 < jhi; j0 += 4 * kStageWarps) {
      const int j = j0 + (lane >> 3), jj = min(j, jhi - 1);
      const float *kj = kc + jj * kStageItem;
      const uint32_t loc = __float_as_uint(kj[0]);
      const int lu = (int)(loc & 0xffu), lv = (int)((loc >> 8) & 0xffu);
      const int aw0 = k - (kbase + (int)((loc >> 16) & 0xffu));
      const float *ku = kj + 2 + 2 * seg - (lu & 1);
      const float ku0 = ku[0], ku1 = ku[1];
      float2 w0[4], w1[4];  // weights of the pair's cells, duplicated for re and im
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float kv = kj[10 + par + 2 * i];
        w0[i] = make_float2(kv * ku0, kv * ku0);
        w1[i] = make_float2(kv * ku1, kv * ku1);
      }
      const float4 *cell = win + lv * hp + (lu >> 1);
      float2 acc[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) acc[p] = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < P; ++q) {
        if (q < np) {  // block-uniform
          // a plane of the chunk that this item does not reach weighs 0
          const int aw = aw0 + q;
          const float kw = aw >= 0 && aw < W ? kj[18 + aw] : 0.f;
          const float2 kw2 = make_float2(kw, kw);
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            float2 s = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 v = cell[(q * NP + p) * SW * hp + off[i]];
              s = __ffma2_rn(make_float2(v.x, v.y), w0[i], s);
              s = __ffma2_rn(make_float2(v.z, v.w), w1[i], s);
            }
            acc[p] = __ffma2_rn(s, kw2, acc[p]);
          }
        }
      }
      float sum[NV];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        sum[2 * p] = acc[p].x;
        sum[2 * p + 1] = acc[p].y;
      }
      reduce8<NV>(sum, lane);
      if (j < jhi && l8 % (8 / NV) == 0)  // only these lanes touch the item in this window
        reinterpret_cast<float *>(sacc + jj * NP)[l8 / (8 / NV)] += sum[0];
    }
    __syncthreads();  // window consumed before its buffer is refilled; sums complete
  }
  degrid_epilogue<NP, NT>(g, items, ch, kbase, b0, nb, vis, npv, wgt, pm, sacc);
}

// The degridding kernels: AW = 8 or 16, the lane width of the warp degridder; AW = 0
// (kStaged), staged planes.  CTAs per SM the warp degridders are compiled for:
// few enough that the CTAs' tiles of one plane fit L1 beside their shared memory.
constexpr int kStaged = 0, kDegridWarpBlocks = 3;
constexpr int degrid_threads(int AW) { return AW == kStaged ? 32 * kStageWarps : kThreads; }
constexpr int degrid_ctas(int AW) { return AW == kStaged ? 1 : kDegridWarpBlocks; }

// Dynamic shared memory of the warp degridder: the item cache, then the
// per-item sums.
__host__ __device__ constexpr size_t degrid_warp_smem(int AW, int NP) {
  return (size_t)kChunkItems * (kcache_stride(AW) * sizeof(float) + NP * sizeof(float2));
}

template <int NP, int AW>
__global__ void __launch_bounds__(degrid_threads(AW), degrid_ctas(AW))
    k_degrid_warp(const Geom g, const ItemF *__restrict__ items, const Chunk *__restrict__ chunks,
                  const uint32_t *__restrict__ chunk_off, int b0, int nb,
                  const float2 *__restrict__ grid, float2 *__restrict__ vis, int npv,
                  const float *__restrict__ wgt, const PolMat pm, const RowPerm rp,
                  uint32_t *__restrict__ counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *kc = reinterpret_cast<float *>(smem_raw);                               // item cache
  float2 *sacc = reinterpret_cast<float2 *>(kc + kChunkItems * kcache_stride(AW));  // sums
  __shared__ int s_first[kMaxSlab + 1], s_rowoff[kMaxSubSide], s_col[kMaxSubSide];
  __shared__ uint32_t s_ci;
  const int ntiles = g.ntu * g.ntv;
  const int wk = g.do_w ? g.W : 1;
  const int lo = b0 - (g.S + wk - 2);
  const int s_lo = lo <= 0 ? 0 : (lo + g.S - 1) / g.S;
  const int s_hi = min(g.nslabs - 1, (b0 + nb - 1) / g.S);
  const uint32_t c_begin = chunk_off[(int64_t)s_lo * ntiles];
  const uint32_t c_end = chunk_off[(int64_t)(s_hi + 1) * ntiles];
  for (;;) {
    if (threadIdx.x == 0) s_ci = c_begin + atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t ci = s_ci;
    __syncthreads();  // every thread has read s_ci (and the last chunk's tables)
    if (ci >= c_end) break;
    if constexpr (AW == kStaged)
      degrid_staged_chunk<NP>(g, items, chunks[ci], b0, nb, grid, vis, npv, wgt, pm, rp,
                              alone_in_bucket(chunks[ci], chunk_off), smem_raw, s_first, s_rowoff);
    else
      degrid_warp_chunk<NP, AW>(g, items, chunks[ci], b0, nb, grid, vis, npv, wgt, pm, rp, kc,
                                sacc, s_first, s_rowoff, s_col);
  }
}

// Many plans' degridding in one persistent launch (FP32 form, one lane
// width): the work queue is the concatenation of every job's chunk range,
// as in k_grid_jobs; each CTA takes the next index from one atomic counter
// and degrids that chunk of its job into the job's visibilities.
template <int NP, int AW>
__global__ void __launch_bounds__(degrid_threads(AW), degrid_ctas(AW))
    k_degrid_warp_jobs(const __grid_constant__ GridJobs jobs, const PolMat pm,
                       uint32_t *__restrict__ counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *kc = reinterpret_cast<float *>(smem_raw);
  float2 *sacc = reinterpret_cast<float2 *>(kc + kChunkItems * kcache_stride(AW));
  __shared__ int s_first[kMaxSlab + 1], s_rowoff[kMaxSubSide], s_col[kMaxSubSide];
  __shared__ uint32_t s_wbeg[kMaxJobs + 1], s_cbeg[kMaxJobs];
  __shared__ uint32_t s_w;
  __shared__ int s_j;
  if (threadIdx.x == 0) {
    uint32_t w = 0;
    for (int j = 0; j < jobs.n; ++j) {
      const GridJob &jb = jobs.job[j];
      const Geom &g = jb.g;
      const int ntiles = g.ntu * g.ntv;
      const int wk = g.do_w ? g.W : 1;
      const int lo = jb.b0 - (g.S + wk - 2);
      const int s_lo = lo <= 0 ? 0 : (lo + g.S - 1) / g.S;
      const int s_hi = min(g.nslabs - 1, (jb.b0 + jb.nb - 1) / g.S);
      const uint32_t c0 = jb.chunk_off[(int64_t)s_lo * ntiles];
      const uint32_t c1 = jb.chunk_off[(int64_t)(s_hi + 1) * ntiles];
      s_wbeg[j] = w;
      s_cbeg[j] = c0;
      w += c1 > c0 ? c1 - c0 : 0u;
    }
    s_wbeg[jobs.n] = w;
  }
  __syncthreads();
  const uint32_t total = s_wbeg[jobs.n];
  for (;;) {
    if (threadIdx.x == 0) {
      const uint32_t w = atomicAdd(counter, 1u);
      int j = 0;
      while (j + 1 < jobs.n && s_wbeg[j + 1] <= w) ++j;
      s_w = w;
      s_j = j;
    }
    __syncthreads();
    const uint32_t w = s_w;
    const int j = s_j;
    __syncthreads();  // every thread has read s_w, s_j
    if (w >= total) break;
    const GridJob &jb = jobs.job[j];
    const uint32_t ci = s_cbeg[j] + (w - s_wbeg[j]);
    const ItemF *items = reinterpret_cast<const ItemF *>(jb.items);
    const float2 *grid = reinterpret_cast<const float2 *>(jb.grid);
    float2 *vis = reinterpret_cast<float2 *>(jb.vis);
    if constexpr (AW == kStaged)
      degrid_staged_chunk<NP>(jb.g, items, jb.chunks[ci], jb.b0, jb.nb, grid, vis, jb.npv, jb.wgt,
                              pm, jb.rp, alone_in_bucket(jb.chunks[ci], jb.chunk_off), smem_raw,
                              s_first, s_rowoff);
    else
      degrid_warp_chunk<NP, AW>(jb.g, items, jb.chunks[ci], jb.b0, jb.nb, grid, vis, jb.npv,
                                jb.wgt, pm, jb.rp, kc, sacc, s_first, s_rowoff, s_col);
  }
}

// Dynamic shared memory of the staged degridder for a plan's tile.
static size_t degrid_staged_smem(const Geom &g) {
  return stage_bytes(g.T + g.W - 1) +
         (size_t)kChunkItems * (kStageItem * sizeof(float) + g.NP * sizeof(float2));
}

// The staged degridder's tiles: supports of up to 7 cells (four cell pairs a
// row), even tile sides (16-byte copies) no wider than the grid, two windows in an
// SM's shared memory (32-cell tiles and smaller).  Others, supports of 8 to 16
// cells, and plans without w-stacking take the warp degridder: a window of one
// plane holds 1, 2 or 4 of the 8 sheets that share an item's weights and its
// reduction (6.7M items, 256^2 to 4096^2 pixels: 0.78-1.21 ms by warps, 1.10-1.71
// staged at 1 pol; 1.29-2.93 and 1.56-3.16 at 4).
static int degrid_width(const Geom &g) {
  const int SW = g.T + g.W - 1;
  const bool staged = g.do_w && g.W <= kStageMaxW && g.T % 2 == 0 && SW + 1 <= g.ngx &&
                      degrid_staged_smem(g) + 3072 <= 227 * 1024;
  return staged ? kStaged : group_lanes(g.W);
}

static size_t degrid_smem(const Geom &g, int AW) {
  return AW == kStaged ? degrid_staged_smem(g) : degrid_warp_smem(AW, g.NP);
}

// Shared-memory carveout (percent of the SM's maximum) that holds `per_sm`
// CTAs of `smem` bytes and leaves the rest of the unified array to L1.
static int degrid_carveout(size_t smem, int per_sm) {
  int dev = 0, max_smem = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (max_smem <= 0) return -1;
  const size_t need = (size_t)per_sm * (smem + 3072);  // + static and reserved shared memory
  const int pct = (int)((need * 100 + max_smem - 1) / max_smem);
  return pct > 100 ? 100 : pct;
}

// Opt-in, carveout and CTAs per SM of a degridding kernel of lane width AW.
template <typename K> static int degrid_prepare(K k, int AW, size_t smem, int *per_sm) {
  const int rc = allow_shared_memory(k);
  if (rc) return rc;
  const int pct = AW == kStaged ? 100 : degrid_carveout(smem, kDegridWarpBlocks);
  if (pct > 0) GB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
  GB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k, degrid_threads(AW), smem));
  if (*per_sm < 1) {
    set_error("a degridding kernel cannot launch with %zu bytes of shared memory", smem);
    return GB_ERR_INVALID_ARG;
  }
  return GB_OK;
}

template <int NP>
static int setup_degrid_warp(gb_plan *p) {
  const int AW = degrid_width(p->g);
  const size_t smem = degrid_smem(p->g, AW);
  int per_sm = 0;
  const int rc = AW == kStaged ? degrid_prepare(k_degrid_warp<NP, kStaged>, AW, smem, &per_sm)
                 : AW == 8     ? degrid_prepare(k_degrid_warp<NP, 8>, AW, smem, &per_sm)
                               : degrid_prepare(k_degrid_warp<NP, 16>, AW, smem, &per_sm);
  if (rc) return rc;
  p->degrid_blocks = per_sm * p->num_sms;
  return GB_OK;
}

// The predict driver in steps (gb_batch.cu interleaves them across plans):
// begin (corrected image), then per w-plane batch bi: transform (screens +
// 2-D transform into the batch buffer), degrid.
template <typename R, int NP>
static int pred_begin_impl(gb_plan *p, const void *dirty, int layout, cudaStream_t s) {
  const Geom &g = p->g;
  R *img = reinterpret_cast<R *>(p->ws + p->off_temp + p->c_img);
  uint32_t *counters = p->at<uint32_t>(p->off_counters) + p->nbatches;
  GB_CUDA(cudaMemsetAsync(counters, 0, 4 * (size_t)p->nbatches, s));
  dim3 fb((g.nx + 31) / 32, (g.ny + 31) / 32, NP);
  const double npix = (double)g.nx * g.ny;
  ProfScope ps(kProfPrepImage, s, 3.0 * sizeof(R) * NP * npix);
  k_prep_image<R><<<fb, dim3(32, 8), 0, s>>>(g, reinterpret_cast<const R *>(dirty), layout,
                                             p->at<R>(p->off_corr), img);
  GB_LAUNCH_CHECK("k_prep_image");
  return GB_OK;
}

template <typename R, int NP>
static int pred_transform_impl(gb_plan *p, int bi, cudaStream_t s) {
  using C = typename Traits<R>::C;
  const Geom &g = p->g;
  char *tmp = p->ws + p->off_temp;
  C *grid = reinterpret_cast<C *>(tmp + p->c_grid);
  R *img = reinterpret_cast<R *>(tmp + p->c_img);
  const int b0 = bi * g.B, nb = std::min(g.B, g.nplanes - b0);
  const int64_t plane = (int64_t)g.ngx * g.ngy;
  const double gbytes = (double)sizeof(C) * nb * NP * (double)plane;
  const double npix = (double)g.nx * g.ny;
  bool cols = false;
  if constexpr (std::is_same<R, float>::value) {
    if (p->col_fft) {  // screen + columns now, rows below
      const int rc = run_cols_predict(p, img, b0, nb, grid, s);
      if (rc) return rc;
      cols = true;
    }
  }
  if (p->fft64) {
    if constexpr (std::is_same<R, double>::value) {
      {
        const unsigned pix_blocks = (unsigned)std::min<int64_t>(
            ((int64_t)npix + kThreads - 1) / kThreads, (int64_t)p->num_sms * 32);
        ProfScope ps(kProfScreenPad, s, 0.25 * gbytes + sizeof(R) * NP * npix);
        k_screen_block<R, NP><<<pix_blocks, kThreads, 0, s>>>(
            g, img, p->at<double>(p->off_tprime), b0, nb, grid);
        GB_LAUNCH_CHECK("k_screen_block");
      }
      // the image, then the image columns of the used rows, read; those
      // columns, then the occupied bins, written
      ProfScope ps(kProfFftFwd, s,
                   (p->used_cells(b0, nb) + p->used_rows(b0, nb) + 0.25) * gbytes);
      return run_fft64(p, b0, nb, grid, -1, s);
    }
  }
  if (!cols) {
    const unsigned cell_blocks = (unsigned)std::min<int64_t>((plane + kThreads - 1) / kThreads,
                                                             (int64_t)p->num_sms * 32);
    ProfScope ps(kProfScreenPad, s, gbytes + sizeof(R) * NP * npix);
    k_screen_pad<R, NP><<<cell_blocks, kThreads, 0, s>>>(g, img, p->at<double>(p->off_tprime),
                                                         b0, nb, grid);
    GB_LAUNCH_CHECK("k_screen_pad");
  }
  if (p->row_fft) {
    // image half in, occupied bins out
    ProfScope ps(kProfRowsFwd, s,
                 (p->used_cells(b0, nb) + 0.5 * p->used_rows(b0, nb)) * gbytes);
    return run_rows(p, grid, b0, nb, -1, s);
  }
  ProfScope ps(kProfFftFwd, s, 2.0 * gbytes);
  return run_fft(p, nb, grid, CUFFT_FORWARD, s);
}

// Algorithmic bytes and updates of degridding batch bi (profiling): items
// read, their vis written once; the grid cells they reach read once (the
// cells of the (plane, tile) pairs reached, else the rows).
template <typename R, int NP>
static void degrid_counts(const gb_plan *p, int bi, int npv, bool wgt, double *bytes,
                          double *updates) {
  using C = typename Traits<R>::C;
  using Item = typename Traits<R>::Item;
  const Geom &g = p->g;
  const int b0 = bi * g.B, nb = std::min(g.B, g.nplanes - b0);
  const double gbytes = (double)sizeof(C) * nb * NP * (double)g.ngx * g.ngy;
  const double cells = p->touched_cells(b0, nb);
  const double gread = cells > 0.0 ? cells * NP * sizeof(C) : p->used_rows(b0, nb) * gbytes;
  *bytes = (double)p->batch_items(b0, nb) *
               (sizeof(Item) + npv * sizeof(C) + (wgt ? npv * sizeof(R) : 0.0)) + gread;
  *updates = p->item_planes(b0, nb) * g.W * g.W * NP;
}

template <typename R, int NP>
static int pred_degrid_impl(gb_plan *p, int bi, const void *wgt, const PolMat &pm, int npv,
                            void *vis, cudaStream_t s) {
  using C = typename Traits<R>::C;
  const Geom &g = p->g;
  C *grid = reinterpret_cast<C *>(p->ws + p->off_temp + p->c_grid);
  uint32_t *counters = p->at<uint32_t>(p->off_counters) + p->nbatches;
  const int b0 = bi * g.B, nb = std::min(g.B, g.nplanes - b0);
  double bytes = 0.0, updates = 0.0;
  if (prof_on()) degrid_counts<R, NP>(p, bi, npv, wgt != nullptr, &bytes, &updates);
  ProfScope ps(kProfDegrid, s, bytes, updates);
  if constexpr (std::is_same<R, float>::value) {
    const ItemF *items = p->at<ItemF>(p->off_items);
    const Chunk *chunks = p->at<Chunk>(p->off_chunks);
    const uint32_t *chunk_off = p->at<uint32_t>(p->off_chunk_off);
    const RowPerm rperm = row_perm(p);
    float2 *vis_c = reinterpret_cast<float2 *>(vis);
    const int AW = degrid_width(g);
    const auto launch = [&](auto k) {
      k<<<p->degrid_blocks, degrid_threads(AW), degrid_smem(g, AW), s>>>(
          g, items, chunks, chunk_off, b0, nb, grid, vis_c, npv, reinterpret_cast<const R *>(wgt),
          pm, rperm, counters + bi);
    };
    if (AW == kStaged)
      launch(k_degrid_warp<NP, kStaged>);
    else if (AW == 8)
      launch(k_degrid_warp<NP, 8>);
    else
      launch(k_degrid_warp<NP, 16>);
    GB_LAUNCH_CHECK("k_degrid_warp");
    return GB_OK;
  } else {
    return launch_degrid64(p, b0, nb, grid, wgt, pm, npv, vis, counters + bi, s);
  }
}

template <typename R, int NP>
static int dirty2ms_impl(gb_plan *p, const void *dirty, int layout, const void *wgt,
                         const PolMat &pm, int npv, void *vis, cudaStream_t s) {
  int rc = pred_begin_impl<R, NP>(p, dirty, layout, s);
  for (int bi = 0; !rc && bi < p->nbatches; ++bi) {
    rc = pred_transform_impl<R, NP>(p, bi, s);
    if (!rc) rc = pred_degrid_impl<R, NP>(p, bi, wgt, pm, npv, vis, s);
  }
  return rc;
}

#define GB_PRED_DISPATCH(p, CALL)                    \
  do {                                               \
    if ((p)->precision == GB_FP64) {                 \
      switch ((p)->g.NP) {                           \
        case 1: { using R = double; constexpr int NP = 1; return CALL; } \
        case 2: { using R = double; constexpr int NP = 2; return CALL; } \
        default: { using R = double; constexpr int NP = 4; return CALL; } \
      }                                              \
    }                                                \
    switch ((p)->g.NP) {                             \
      case 1: { using R = float; constexpr int NP = 1; return CALL; } \
      case 2: { using R = float; constexpr int NP = 2; return CALL; } \
      default: { using R = float; constexpr int NP = 4; return CALL; } \
    }                                                \
  } while (0)

int pred_begin(gb_plan *p, const void *dirty, int layout, cudaStream_t s) {
  GB_PRED_DISPATCH(p, (pred_begin_impl<R, NP>(p, dirty, layout, s)));
}
int pred_transform(gb_plan *p, int bi, cudaStream_t s) {
  GB_PRED_DISPATCH(p, (pred_transform_impl<R, NP>(p, bi, s)));
}

// Fill one job of a multi-plan degridding launch from a bound FP32 plan
// whose batch bi has been transformed.
int degrid_job(gb_plan *p, int bi, void *vis, int npv, GridJob &jb) {
  if (p->precision != GB_FP32 || !p->bound || bi < 0 || bi >= p->nbatches) {
    set_error("degrid_job: needs a bound FP32 plan and a batch index in range");
    return GB_ERR_INVALID_ARG;
  }
  char *tmp = p->ws + p->off_temp;
  jb.g = p->g;
  jb.items = p->at<ItemF>(p->off_items);
  jb.cvis = nullptr;
  jb.chunks = p->at<Chunk>(p->off_chunks);
  jb.chunk_off = p->at<uint32_t>(p->off_chunk_off);
  jb.grid = tmp + p->c_grid;
  jb.b0 = bi * p->g.B;
  jb.nb = std::min(p->g.B, p->g.nplanes - jb.b0);
  jb.vis = vis;
  jb.npv = npv;
  jb.pad = 0;
  jb.wgt = nullptr;
  jb.rp = row_perm(p);
  return GB_OK;
}

void degrid_job_counts(const gb_plan *p, int bi, int npv, double *bytes, double *updates) {
  *bytes = 0.0;
  *updates = 0.0;
  if (!prof_on()) return;
  switch (p->g.NP) {
    case 1: degrid_counts<float, 1>(p, bi, npv, false, bytes, updates); break;
    case 2: degrid_counts<float, 2>(p, bi, npv, false, bytes, updates); break;
    default: degrid_counts<float, 4>(p, bi, npv, false, bytes, updates); break;
  }
}

// One launch over `jobs` (all of one NP and support W, unit weights, one pol
// matrix); `counter` must be zero.
int launch_degrid_jobs(const GridJobs &jobs, const PolMat &pm, int num_sms, uint32_t *counter,
                       double bytes, double updates, cudaStream_t s) {
  if (jobs.n < 1 || jobs.n > kMaxJobs) {
    set_error("launch_degrid_jobs: %d jobs (1..%d)", jobs.n, kMaxJobs);
    return GB_ERR_INVALID_ARG;
  }
  const int NP = jobs.job[0].g.NP;
  int AW = kStaged;  // if every job's tile can be staged
  for (int j = 0; j < jobs.n; ++j) {
    const Geom &g = jobs.job[j].g;
    if (g.NP != NP || group_lanes(g.W) != group_lanes(jobs.job[0].g.W)) {
      set_error("launch_degrid_jobs: jobs of one launch share NP and the lane width");
      return GB_ERR_INVALID_ARG;
    }
    if (degrid_width(g) != kStaged) AW = group_lanes(g.W);
  }
  size_t smem = 0;
  for (int j = 0; j < jobs.n; ++j) smem = std::max(smem, degrid_smem(jobs.job[j].g, AW));
  ProfScope ps(kProfDegrid, s, bytes, updates);
  const auto launch = [&](auto k) {
    int per_sm = 0;
    const int rc = degrid_prepare(k, AW, smem, &per_sm);
    if (!rc) k<<<per_sm * num_sms, degrid_threads(AW), smem, s>>>(jobs, pm, counter);
    return rc;
  };
  const auto launch_np = [&](auto np) {
    constexpr int N = decltype(np)::value;
    return AW == kStaged ? launch(k_degrid_warp_jobs<N, kStaged>)
           : AW == 8     ? launch(k_degrid_warp_jobs<N, 8>)
                         : launch(k_degrid_warp_jobs<N, 16>);
  };
  const int rc = NP == 1   ? launch_np(std::integral_constant<int, 1>())
                 : NP == 2 ? launch_np(std::integral_constant<int, 2>())
                           : launch_np(std::integral_constant<int, 4>());
  if (rc) return rc;
  GB_LAUNCH_CHECK("k_degrid_warp_jobs");
  return GB_OK;
}

int run_dirty2ms(gb_plan *p, const void *dirty, int layout, const void *wgt, const PolMat &pm,
                 int npv, void *vis, cudaStream_t s) {
#define GB_CASE(R, NP) return dirty2ms_impl<R, NP>(p, dirty, layout, wgt, pm, npv, vis, s)
  if (p->precision == GB_FP64) {
    switch (p->g.NP) {
      case 1: GB_CASE(double, 1);
      case 2: GB_CASE(double, 2);
      default: GB_CASE(double, 4);
    }
  }
  switch (p->g.NP) {
    case 1: GB_CASE(float, 1);
    case 2: GB_CASE(float, 2);
    default: GB_CASE(float, 4);
  }
#undef GB_CASE
}

int setup_tile_kernels(gb_plan *p) {
  if (p->precision == GB_FP64) return setup_tile_kernels64(p);
  const int rc = setup_grid_kernels(p);
  if (rc) return rc;
  switch (p->g.NP) {
    case 1: return setup_degrid_warp<1>(p);
    case 2: return setup_degrid_warp<2>(p);
    default: return setup_degrid_warp<4>(p);
  }
}

}  // namespace gb
