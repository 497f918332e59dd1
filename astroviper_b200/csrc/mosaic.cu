// Mosaic / A-projection gridding with general convolution functions
// (mosaic_grid.py): each sample's footprint is a window of a 2-D complex
// convolution function chosen by (baseline, channel, polarisation) maps,
// premultiplied by the field's phase gradient.
//
// av_mosaic_grid      mosaic_grid_jit (mosaic_grid.py:307-486): one warp per
//                     (time, baseline, channel) sample, lanes over the
//                     support window, FP64 atomics into the grid; the
//                     window's norm is reduced in the warp for sum_weight.
// av_aperture_grid    aperture_grid_jit (mosaic_grid.py:13-153): every
//                     sample adds its function at the grid centre, so the
//                     weights are first summed per (function baseline,
//                     channel, polarisation) class and each class then adds
//                     its function once.
// av_cf_phase_product conv_kernel x phase_gradient[0] (mosaic_grid.py:384,
//                     :56-58), elementwise without fused multiply-add.
#include <math_constants.h>

#include <algorithm>

#include "plan.cuh"

namespace av {

struct MosaicArgs {
  double2 *grid;
  double *sumw;
  int do_psf;
  const double2 *vis;      // (nt, nb, nchan, npol), NULL for do_psf
  const double *wt;        // (nt, nb, nchan, npol)
  const double *uvw, *freq;
  const int32_t *chan_map, *pol_map, *cfb_map, *cfc_map, *cfp_map;
  const double2 *cf;       // (n_cfb, n_cfc, n_cfp, cu, cv), phase gradient applied
  int64_t n_cfb, n_cfc, n_cfp, cu, cv;
  const int32_t *support;  // (n_cfb, n_cfc, n_cfp, 2)
  int max_support;         // np.max(weight_support)
  int64_t n_u, n_v;
  double dl0, dl1;
  int os_u, os_v;
  int64_t nt, nb, nchan, npol, n_img_chan, n_img_pol;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                      __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}

// Position of a sample (mosaic_grid.py:384-405): centre cell and the offset
// index into the function; false when off the grid or NaN.
__device__ __forceinline__ bool mosaic_pos(const MosaicArgs &a, int64_t tb, int64_t c,
                                           long long &uc, long long &vc, long long &uo,
                                           long long &vo) {
  const double f = a.freq[c];
  const double s0 = __ddiv_rn(-__dmul_rn(__dmul_rn(f, a.dl0), (double)a.n_u), C_LIGHT);
  const double s1 = __ddiv_rn(-__dmul_rn(__dmul_rn(f, a.dl1), (double)a.n_v), C_LIGHT);
  const double u = __dmul_rn(a.uvw[3 * tb], s0), v = __dmul_rn(a.uvw[3 * tb + 1], s1);
  if (isnan(u) || isnan(v)) return false;
  const double up = __dadd_rn(u, (double)(a.n_u / 2)), vp = __dadd_rn(v, (double)(a.n_v / 2));
  uc = trunc_ll(__dadd_rn(up, 0.5));
  vc = trunc_ll(__dadd_rn(vp, 0.5));
  const long long ms = a.max_support;
  if (!(uc + ms < a.n_u && vc + ms < a.n_v && uc - ms >= 0 && vc - ms >= 0)) return false;
  uo = (long long)floor(__dadd_rn(__dmul_rn(__dsub_rn((double)uc, up), (double)a.os_u), 0.5)) +
       a.cu / 2;
  vo = (long long)floor(__dadd_rn(__dmul_rn(__dsub_rn((double)vc, vp), (double)a.os_v), 0.5)) +
       a.cv / 2;
  return true;
}

constexpr int MG_THREADS = 256;

__global__ void __launch_bounds__(MG_THREADS) k_mosaic_grid(MosaicArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t n_rows = a.nt * a.nb * a.nchan;
  for (int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; row < n_rows;
       row += n_warps) {
    const int64_t tb = row / a.nchan;
    const int64_t c = row - tb * a.nchan;
    const int64_t b = tb % a.nb;
    long long uc, vc, uo, vo;
    if (!mosaic_pos(a, tb, c, uc, vc, uo, vo)) continue;
    const int cfb = a.cfb_map[b], cfc = a.cfc_map[c], ach = a.chan_map[c];
    if (ach < 0 || ach >= a.n_img_chan || cfb < 0 || cfb >= a.n_cfb || cfc < 0 ||
        cfc >= a.n_cfc)
      continue;
    for (int64_t p = 0; p < a.npol; ++p) {
      const int64_t k = row * a.npol + p;
      const double w = a.wt[k];
      double2 wd;
      if (a.do_psf) wd = make_double2(w, 0.0);
      else {
        const double2 vv = a.vis[k];
        wd = make_double2(__dmul_rn(vv.x, w), __dmul_rn(vv.y, w));
      }
      if (isnan(wd.x) || isnan(wd.y) || (wd.x == 0.0 && wd.y == 0.0)) continue;
      const int cfp = a.cfp_map[p], apol = a.pol_map[p];
      if (cfp < 0 || cfp >= a.n_cfp || apol < 0 || apol >= a.n_img_pol) continue;
      const int64_t fidx = ((int64_t)cfb * a.n_cfc + cfc) * a.n_cfp + cfp;
      const int su = a.support[2 * fidx], sv = a.support[2 * fidx + 1];
      const int su0 = -(su / 2), sv0 = -(sv / 2);
      const double2 *f = a.cf + fidx * a.cu * a.cv;
      double2 *g = a.grid + ((int64_t)ach * a.n_img_pol + apol) * a.n_u * a.n_v;
      double2 norm = make_double2(0.0, 0.0);
      const int n_tap = su * sv;
      for (int t0 = 0; t0 < n_tap; t0 += 32) {
        const int t = t0 + lane;
        if (t >= n_tap) continue;
        const int iv = sv0 + t / su, iu = su0 + t % su;  // v outer, u inner
        const long long fu = (long long)a.os_u * iu + uo, fv = (long long)a.os_v * iv + vo;
        // a window reaching past the function (the reference reads beyond it)
        if (fu < 0 || fu >= a.cu || fv < 0 || fv >= a.cv) continue;
        const double2 conv = f[fu * a.cv + fv];
        const double2 x = cmul(conv, wd);
        double2 *cell = g + (uc + iu) * a.n_v + (vc + iv);
        atomicAdd(&cell->x, x.x);
        atomicAdd(&cell->y, x.y);
        norm.x += conv.x;
        norm.y += conv.y;
      }
      for (int off = 16; off > 0; off >>= 1) {
        norm.x += __shfl_down_sync(0xffffffffu, norm.x, off);
        norm.y += __shfl_down_sync(0xffffffffu, norm.y, off);
      }
      if (lane == 0 && a.sumw) {
        // do_psf: w Re(norm); else w Re(norm^2) (the function enters twice)
        const double re = a.do_psf ? norm.x
                                   : __dsub_rn(__dmul_rn(norm.x, norm.x), __dmul_rn(norm.y, norm.y));
        atomicAdd(&a.sumw[(int64_t)ach * a.n_img_pol + apol], __dmul_rn(w, re));
      }
    }
  }
}

// aperture_grid_jit, pass 1: weight sums per (function baseline, channel,
// polarisation) class over the samples that pass the grid bounds.
__global__ void __launch_bounds__(MG_THREADS) k_aperture_classes(MosaicArgs a, double *cls) {
  const int64_t n_rows = a.nt * a.nb * a.nchan;
  for (int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; row < n_rows;
       row += (int64_t)gridDim.x * blockDim.x) {
    const int64_t tb = row / a.nchan;
    const int64_t c = row - tb * a.nchan;
    const int64_t b = tb % a.nb;
    long long uc, vc, uo, vo;
    if (!mosaic_pos(a, tb, c, uc, vc, uo, vo)) continue;
    const int cfb = a.cfb_map[b];
    if (cfb < 0 || cfb >= a.n_cfb) continue;
    for (int64_t p = 0; p < a.npol; ++p) {
      const double w = a.wt[row * a.npol + p];
      if (isnan(w) || w == 0.0) continue;
      atomicAdd(&cls[((int64_t)cfb * a.nchan + c) * a.npol + p], w);
    }
  }
}

// pass 2: one block per class adds w_class x function window at the grid
// centre and w_class x Re(norm) to sum_weight.
__global__ void __launch_bounds__(MG_THREADS) k_aperture_add(MosaicArgs a, const double *cls) {
  const int64_t cl = blockIdx.x;
  const double w = cls[cl];
  if (w == 0.0) return;
  const int64_t p = cl % a.npol;
  const int64_t c = (cl / a.npol) % a.nchan;
  const int64_t cfb = cl / (a.npol * a.nchan);
  const int cfc = a.cfc_map[c], cfp = a.cfp_map[p], ach = a.chan_map[c], apol = a.pol_map[p];
  if (cfc < 0 || cfc >= a.n_cfc || cfp < 0 || cfp >= a.n_cfp || ach < 0 ||
      ach >= a.n_img_chan || apol < 0 || apol >= a.n_img_pol)
    return;
  const int64_t fidx = (cfb * a.n_cfc + cfc) * a.n_cfp + cfp;
  const int su = a.support[2 * fidx], sv = a.support[2 * fidx + 1];
  const int su0 = -(su / 2), sv0 = -(sv / 2);
  const double2 *f = a.cf + fidx * a.cu * a.cv;
  double2 *g = a.grid + ((int64_t)ach * a.n_img_pol + apol) * a.n_u * a.n_v;
  double2 norm = make_double2(0.0, 0.0);
  const int n_tap = su * sv;
  for (int t0 = 0; t0 < n_tap; t0 += blockDim.x) {
    const int t = t0 + threadIdx.x;
    if (t >= n_tap) continue;
    const int iv = sv0 + t / su, iu = su0 + t % su;
    const long long fu = (long long)a.os_u * iu + a.cu / 2, fv = (long long)a.os_v * iv + a.cv / 2;
    const long long gu = a.n_u / 2 + iu, gv = a.n_v / 2 + iv;
    if (fu < 0 || fu >= a.cu || fv < 0 || fv >= a.cv || gu < 0 || gu >= a.n_u || gv < 0 ||
        gv >= a.n_v)
      continue;
    const double2 conv = f[fu * a.cv + fv];
    double2 *cell = g + gu * a.n_v + gv;
    atomicAdd(&cell->x, __dmul_rn(conv.x, w));
    atomicAdd(&cell->y, __dmul_rn(conv.y, w));
    norm.x += conv.x;
  }
  __shared__ double sh[MG_THREADS / 32];
  double s = norm.x;
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0 && a.sumw) {
    double r = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r += sh[i];
    atomicAdd(&a.sumw[(int64_t)ach * a.n_img_pol + apol], __dmul_rn(w, r));
  }
}

__global__ void k_cf_phase_product(const void *kern, int kern_complex, const double2 *pg,
                                   double2 *out, int64_t n_cf, int64_t n_pix) {
  const int64_t n = n_cf * n_pix;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double2 g = pg[i % n_pix];
    if (kern_complex) {
      out[i] = cmul(((const double2 *)kern)[i], g);
    } else {
      const double r = ((const double *)kern)[i];
      out[i] = make_double2(__dmul_rn(r, g.x), __dmul_rn(r, g.y));
    }
  }
}

// Airy-disk primary beams (make_pb_symmetric.py:1-280), one value per
// thread in the reference's operation order; J1 is CUDA's j1.
struct AiryArgs {
  double *out;
  int64_t n_dish, n_freq, nx, ny, cx, cy, n_pol;
  double cell_x, cell_y;
  int ipower, casa, rorder;
  double dish[16], block[16];
  const double *freq;
};

__global__ void k_airy_pattern(AiryArgs a) {
  const int64_t n = a.n_dish * a.n_freq * a.nx * a.ny;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t iy = t % a.ny;
    const int64_t ix = (t / a.ny) % a.nx;
    const int64_t f = (t / (a.ny * a.nx)) % a.n_freq;
    const int64_t d = t / (a.ny * a.nx * a.n_freq);
    double v = 1.0;
    if (!(ix == a.cx && iy == a.cy)) {
      const double x = __dmul_rn((double)(ix - a.cx), a.cell_x);
      const double y = __dmul_rn((double)(iy - a.cy), a.cell_y);
      const double k = __ddiv_rn(__dmul_rn(2.0 * 3.141592653589793, a.freq[f]), C_LIGHT);
      const double r = __dmul_rn(__dmul_rn(__dsqrt_rn(__dadd_rn(__dmul_rn(x, x),
                                                                 __dmul_rn(y, y))), k),
                                 __ddiv_rn(a.dish[d], 2.0));
      const double dd = a.dish[d], bd = a.block[d];
      if (bd == 0.0) {
        v = __ddiv_rn(__dmul_rn(2.0, j1(r)), r);
      } else if (!a.casa) {
        const double e = __ddiv_rn(bd, dd);
        const double t1 = __ddiv_rn(__dmul_rn(2.0, j1(r)), r);
        const double t2 = __ddiv_rn(__dmul_rn(__dmul_rn(2.0, e), j1(__dmul_rn(r, e))), r);
        v = __ddiv_rn(__dsub_rn(t1, t2), __dsub_rn(1.0, __dmul_rn(e, e)));
      } else {
        const double lr = __ddiv_rn(dd, bd);
        const double ar = __dmul_rn(lr, lr);
        const double t1 = __ddiv_rn(__dmul_rn(__dmul_rn(ar, 2.0), j1(r)), r);
        const double rl = __dmul_rn(r, lr);
        const double t2 = __ddiv_rn(__dmul_rn(2.0, j1(rl)), rl);
        v = __ddiv_rn(__dsub_rn(t1, t2), __dsub_rn(ar, 1.0));
      }
      double p = v;
      for (int i = 1; i < a.ipower; ++i) p = __dmul_rn(p, v);
      v = a.ipower == 0 ? 1.0 : p;
    }
    for (int64_t q = 0; q < a.n_pol; ++q) {
      int64_t o;
      if (a.rorder)  // (dish, freq, pol, x, y)
        o = (((d * a.n_freq + f) * a.n_pol + q) * a.nx + ix) * a.ny + iy;
      else  // (x, y, freq, pol, dish)
        o = (((ix * a.ny + iy) * a.n_freq + f) * a.n_pol + q) * a.n_dish + d;
      a.out[o] = v;
    }
  }
}

// ----------------------------------------------------------------- tiled --
// Binned version of k_mosaic_grid: the gridder's plan (plan.cuh) with a
// footprint window of S = max_support cells and the mosaic's edge margin
// (np.max(weight_support)) holds every kept sample's cell and kernel offset;
// a persistent CTA per SM takes record chunks, keeps an FP64 complex
// sub-grid of (32 + S - 1)^2 x n_img_pol in shared memory per tile segment
// and flushes it once.  A warp takes one record at a time; its lanes cover
// the support window packed as (32 / su) rows of su columns.
constexpr int MT_THREADS = 512;
constexpr int MT_WARPS = MT_THREADS / 32;

// Unsigned 32-bit division by an invariant d (Granlund and Montgomery,
// "Division by invariant integers using multiplication", 1994): with
// l = ceil(log2 d), m = floor(2^32 (2^l - d) / d) + 1, t = mulhi(m, n),
// n / d = (t + ((n - t) >> 1)) >> (l - 1); d = 1 uses m = 0 and no shifts.
struct FastDiv {
  uint32_t m;
  int s1, s2;
};

static FastDiv fast_div(uint32_t d) {
  FastDiv f{0u, 0, 0};
  if (d <= 1) return f;
  int l = 0;
  while ((1ull << l) < d) ++l;
  f.m = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << l) - d)) / d + 1);
  f.s1 = 1;
  f.s2 = l - 1;
  return f;
}

__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv &f) {
  const uint32_t t = __umulhi(f.m, n);
  return (t + ((n - t) >> f.s1)) >> f.s2;
}

struct MosaicTiledArgs {
  MosaicArgs m;
  FastDiv div_nchan, div_nb;  // row -> (time x baseline, channel), -> baseline
  const Rec *recs;
  const uint32_t *tile_start;
  const uint32_t *n_rec;
  uint32_t *sched;
  int64_t n_tiles, ntu, ntv, chunk;
  int S;   // footprint window (max_support)
  int W;   // sub-grid edge, TILE + S - 1
};

__global__ void __launch_bounds__(MT_THREADS, 1) k_mosaic_tiled(MosaicTiledArgs t) {
  const MosaicArgs &a = t.m;
  extern __shared__ __align__(16) unsigned char smem[];
  // real and imaginary planes [apol][W * W]: a warp's 8-byte atomics along a
  // window row fall on consecutive banks
  const int W = t.W, npg = (int)a.n_img_pol;
  const int sub_n = npg * W * W;
  double *sre = (double *)smem;
  double *sim = sre + sub_n;
  __shared__ int s_chunk;
  // lane packing of a window with sv columns: 32 / sv rows per pass, lane
  // ir = lane / sv (sv <= max_support <= 32)
  __shared__ unsigned char s_ir[33][32], s_rp[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n_rec = *t.n_rec;
  const int64_t n_chunks = ((int64_t)n_rec + t.chunk - 1) / t.chunk;
  const uint32_t nchan = (uint32_t)a.nchan, nb = (uint32_t)a.nb;
  for (int i = threadIdx.x; i < 33 * 32; i += MT_THREADS) {
    const int sv = i >> 5, l = i & 31;
    s_ir[sv][l] = (unsigned char)(sv ? l / sv : 0);
    if (l == 0) s_rp[sv] = (unsigned char)(sv ? 32 / sv : 0);
  }
  for (int i0 = 0; i0 < sub_n; i0 += MT_THREADS) {
    const int i = i0 + threadIdx.x;
    if (i < sub_n) {
      sre[i] = 0.0;
      sim[i] = 0.0;
    }
  }
  for (;;) {
    __syncthreads();  // sub-grid clear; previous s_chunk consumed
    if (threadIdx.x == 0)
      s_chunk = chunk_in_turn(atomicAdd(&t.sched[0], 1u), (uint32_t)n_chunks,
                              (uint32_t)(t.n_tiles / (t.ntu * t.ntv)));
    __syncthreads();
    const int64_t ch = s_chunk;
    if (ch >= n_chunks) break;
    const uint32_t r0 = (uint32_t)(ch * t.chunk);
    const uint32_t r1 = (uint32_t)min((int64_t)n_rec, (int64_t)r0 + t.chunk);
    int64_t lo = 0, hi = t.n_tiles;  // tile holding r0
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (t.tile_start[mid] <= r0) lo = mid; else hi = mid;
    }
    int64_t tile = lo;
    uint32_t seg_lo = r0;
    while (seg_lo < r1) {
      const uint32_t t_end = t.tile_start[tile + 1];
      const uint32_t seg_hi = min(r1, t_end);
      if (seg_hi <= seg_lo) {
        ++tile;
        continue;
      }
      const int64_t plane = tile / (t.ntu * t.ntv);
      const int64_t trem = tile - plane * t.ntu * t.ntv;
      const int tu = (int)(trem / t.ntv), tv = (int)(trem - (int64_t)tu * t.ntv);
      double swacc[4] = {0.0, 0.0, 0.0, 0.0};
      // one trip count per block: every warp reaches the barrier converged
      for (uint32_t rb = seg_lo; rb < seg_hi; rb += MT_WARPS) {
        const uint32_t r = rb + warp;
        if (r >= seg_hi) continue;
        const Rec rc = t.recs[r];
        const int64_t row = rc.row;
        const uint32_t tb = fdiv(rc.row, t.div_nchan);  // rows fit 32 bits (the plan checks)
        const uint32_t c = rc.row - tb * nchan;
        const uint32_t b = tb - fdiv(tb, t.div_nb) * nb;
        const int cfb = a.cfb_map[b], cfc = a.cfc_map[c];
        if (cfb < 0 || cfb >= a.n_cfb || cfc < 0 || cfc >= a.n_cfc) continue;
        const long long uo = (long long)rc.ou - 128 + a.cu / 2;
        const long long vo = (long long)rc.ov - 128 + a.cv / 2;
        const int cu0 = rc.du + t.S / 2, cv0 = rc.dv + t.S / 2;  // centre in the sub-grid
        // the window's norm depends on the function only (same sample): kept
        // for the next polarisation that uses the same function
        int64_t norm_fidx = -1;
        double2 norm_prev = make_double2(0.0, 0.0);
        for (int64_t p = 0; p < a.npol; ++p) {
          const int64_t k = row * a.npol + p;
          const double w = a.wt[k];
          double2 wd;
          if (a.do_psf) wd = make_double2(w, 0.0);
          else {
            const double2 vv = a.vis[k];
            wd = make_double2(__dmul_rn(vv.x, w), __dmul_rn(vv.y, w));
          }
          if (isnan(wd.x) || isnan(wd.y) || (wd.x == 0.0 && wd.y == 0.0)) continue;
          const int cfp = a.cfp_map[p], apol = a.pol_map[p];
          if (cfp < 0 || cfp >= a.n_cfp || apol < 0 || apol >= npg) continue;
          const int64_t fidx = ((int64_t)cfb * a.n_cfc + cfc) * a.n_cfp + cfp;
          const int su = a.support[2 * fidx], sv = a.support[2 * fidx + 1];
          // a window larger than the footprint the plan reserved would leave
          // the sub-grid: such functions are skipped (the host passes
          // max_support = np.max(support))
          if (su < 1 || sv < 1 || su > t.S || sv > t.S) continue;
          const double2 *f = a.cf + fidx * a.cu * a.cv;
          double *pre = sre + (size_t)apol * W * W, *pim = sim + (size_t)apol * W * W;
          // lanes along the window's v (contiguous) axis: lane = ir * sv + jv,
          // 32 / sv u-rows per pass
          const int rp = s_rp[sv];
          const int ir = s_ir[sv][lane];
          const int iv = -(sv / 2) + (lane - ir * sv);
          const long long fv = (long long)a.os_v * iv + vo;
          const bool v_ok = ir < rp && fv >= 0 && fv < a.cv;
          double2 norm = make_double2(0.0, 0.0);
          for (int iu0 = 0; iu0 < su; iu0 += rp) {
            const int iui = iu0 + ir;
            if (!v_ok || iui >= su) continue;
            const int iu = -(su / 2) + iui;
            const long long fu = (long long)a.os_u * iu + uo;
            if (fu < 0 || fu >= a.cu) continue;
            const double2 conv = __ldg(f + fu * a.cv + fv);
            const double2 x = cmul(conv, wd);
            const int cell = (cu0 + iu) * W + (cv0 + iv);
            atomicAdd(pre + cell, x.x);
            atomicAdd(pim + cell, x.y);
            norm.x += conv.x;
            norm.y += conv.y;
          }
          if (fidx == norm_fidx) {
            norm = norm_prev;
          } else {
            for (int off = 16; off > 0; off >>= 1) {
              norm.x += __shfl_down_sync(0xffffffffu, norm.x, off);
              norm.y += __shfl_down_sync(0xffffffffu, norm.y, off);
            }
            norm_fidx = fidx;
            norm_prev = norm;
          }
          const double re = a.do_psf ? norm.x
                                     : __dsub_rn(__dmul_rn(norm.x, norm.x),
                                                 __dmul_rn(norm.y, norm.y));
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (q == apol) swacc[q] += __dmul_rn(w, re);
        }
      }
      if (lane == 0 && a.sumw)
        for (int q = 0; q < npg && q < 4; ++q)
          if (swacc[q] != 0.0) atomicAdd(&a.sumw[plane * npg + q], swacc[q]);
      __syncthreads();
      // flush the segment's sub-grid to the global grid and clear it
      for (int i0 = 0; i0 < sub_n; i0 += MT_THREADS) {
        const int i = i0 + threadIdx.x;
        if (i >= sub_n) continue;
        const double vr = sre[i], vi = sim[i];
        if (vr == 0.0 && vi == 0.0) continue;
        const int gp = i / (W * W);
        const int cell = i - gp * W * W;
        const int iu = cell / W, iv = cell - iu * W;
        const int64_t gu = (int64_t)tu * TILE + iu, gv = (int64_t)tv * TILE + iv;
        double2 *gd = a.grid + ((plane * npg + gp) * a.n_u + gu) * a.n_v + gv;
        atomicAdd(&gd->x, vr);
        atomicAdd(&gd->y, vi);
        sre[i] = 0.0;
        sim[i] = 0.0;
      }
      seg_lo = seg_hi;
      if (seg_hi == t_end) ++tile;
    }
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&t.sched[1], 1u) == gridDim.x - 1) {
      t.sched[0] = 0u;
      t.sched[1] = 0u;
      __threadfence();
    }
  }
}

// ------------------------------------------------------------------ runs --
// The same binned gridding for windows of up to MR_MAX_S cells and up to 4
// polarisations, with the footprint in registers: the kernel above spends
// some 640 instructions on a sample (a whole warp per sample and
// polarisation, the sample's indices worked out by every lane, two shared
// FP64 atomics per tap).  Here
//   - the taps of every function and kernel offset are first gathered into
//     contiguous rows of S x S values (k_mosaic_taps), with the row's norm, so
//     a sample's taps are one coalesced read where the oversampled function
//     spreads them over a 32-byte sector each; one more row, of zeros, is for
//     samples without a value to add;
//   - a warp's lanes stage 32 samples at once (weighted values, tap row, sum
//     of weights), the next round's data in flight meanwhile;
//   - lane l owns window cells l, l + 32, ... and keeps their sums for all
//     polarisations while the samples stay in one cell: one tap load and 4
//     NPOL DFMA per sample and owned cell, shared atomics only when the cell
//     changes; two samples' taps are in flight whatever the runs (one where a
//     sample has more than 4 loads per lane).
// Cells past the window hold zero taps and skipped values are zeros, so
// products that the reference does not form are zeros too, unless the other
// factor is not finite: a round with an infinite value or a row that holds a
// tap that is not finite (both rare) goes tap by tap and value by value.
// 1.03M samples x 2 polarisations, supports 5-7: k_mosaic_tiled 1315 us, this
// 178 us (and 45 us of plan): 87M warp instructions, 84 a sample, issued in 47 %
// of the cycles at 16 warps per SM (114 registers), which wait for fixed
// latencies, taps and slots.
constexpr int MR_MAX_S = 11;
constexpr int MR_THREADS = 256;
constexpr int MR_WARPS = MR_THREADS / 32;
constexpr int MR_ROUND = 32;  // samples a warp stages at once

struct MosaicRunsArgs {
  MosaicTiledArgs t;
  const double2 *taps;  // [function][u offset][v offset][S * S], then a row of zeros
  const double2 *norm;  // per row: Re(norm) (PSF) or Re(norm^2); infinite when a
                        // tap is not finite, else 0
  int first, n_off;     // kernel offsets first .. first + n_off - 1
  int zero_row;
};

// Whether tap (iu, iv) counted from the window's corner is one of function
// fidx's at offset (ou, ov), and where it is.
__device__ __forceinline__ bool mosaic_tap(const MosaicArgs &a, int64_t fidx, int S, int ri,
                                           int ci, int ou, int ov, int64_t &at) {
  const int su = a.support[2 * fidx], sv = a.support[2 * fidx + 1];
  const int iu = ri - S / 2, iv = ci - S / 2;
  const int64_t fu = (int64_t)a.os_u * iu + ou + a.cu / 2;
  const int64_t fv = (int64_t)a.os_v * iv + ov + a.cv / 2;
  at = fidx * a.cu * a.cv + fu * a.cv + fv;
  return su >= 1 && sv >= 1 && su <= S && sv <= S && iu >= -(su / 2) && iu < su - su / 2 &&
         iv >= -(sv / 2) && iv < sv - sv / 2 && fu >= 0 && fu < a.cu && fv >= 0 && fv < a.cv;
}

// One block per (function, u offset, v offset), and one for the row of zeros.
__global__ void __launch_bounds__(128) k_mosaic_taps(MosaicArgs a, int S, int first, int n_off,
                                                     double2 *taps, double2 *norm) {
  const int64_t row = blockIdx.x;
  const bool zeros = row == gridDim.x - 1;
  const int ov = first + (int)(row % n_off), ou = first + (int)(row / n_off % n_off);
  const int64_t fidx = row / ((int64_t)n_off * n_off);
  double2 c = make_double2(0.0, 0.0);
  const int i = threadIdx.x;
  if (i < S * S) {
    int64_t at;
    if (!zeros && mosaic_tap(a, fidx, S, i / S, i % S, ou, ov, at)) c = a.cf[at];
    taps[row * (S * S) + i] = c;
  }
  const int bad = __syncthreads_or(!isfinite(c.x) || !isfinite(c.y));
  __shared__ double2 sh[4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c.x += __shfl_down_sync(0xffffffffu, c.x, o);
    c.y += __shfl_down_sync(0xffffffffu, c.y, o);
  }
  if ((i & 31) == 0) sh[i >> 5] = c;
  __syncthreads();
  if (i == 0) {
    const double x = (sh[0].x + sh[1].x) + (sh[2].x + sh[3].x);
    const double y = (sh[0].y + sh[1].y) + (sh[2].y + sh[3].y);
    norm[row] = make_double2(a.do_psf ? x : __dsub_rn(__dmul_rn(x, x), __dmul_rn(y, y)),
                             bad ? CUDART_INF : 0.0);
  }
}

// A sample's record and raw values, in flight until used.
template <int NPOL>
struct MosaicRaw {
  Rec rc;
  bool ok;
  double w[NPOL];
  double2 v[NPOL];
};

template <int NPOL>
__device__ __forceinline__ void mosaic_fetch(MosaicRaw<NPOL> &f, const MosaicArgs &a,
                                             const Rec &rc, bool ok) {
  f.ok = ok;
  if (!ok) return;
  f.rc = rc;
  const int64_t k = (int64_t)rc.row * a.npol;
#pragma unroll
  for (int p = 0; p < NPOL; ++p) {
    f.w[p] = p < a.npol ? __ldg(a.wt + k + p) : 0.0;
    f.v[p] = p < a.npol && !a.do_psf ? __ldg(a.vis + k + p) : make_double2(0.0, 0.0);
  }
}

struct MosaicShape {  // sub-grid strides: odd rows, planes 1 mod 16 doubles
  int W, RS, PS;
  __host__ __device__ explicit MosaicShape(int S)
      : W(TILE + S - 1), RS(W | 1), PS((W * RS + 15) / 16 * 16 + 1) {}
};

template <int NPOL>
__host__ __device__ constexpr size_t mosaic_stage_bytes() {
  return (size_t)MR_WARPS * MR_ROUND * NPOL * (sizeof(double2) + sizeof(int));
}

// Round slots: value [pol][sample], tap row [pol][sample].
template <int CPL, int NPOL, bool MULTI>
struct MosaicLanes {
  double2 acc[CPL][NPOL];
  int cell[CPL];  // offset of the owned cells in the sub-grid
  bool own[CPL];
  int ipm[NPOL];

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int c = 0; c < CPL; ++c)
#pragma unroll
      for (int p = 0; p < NPOL; ++p) acc[c][p] = make_double2(0.0, 0.0);
  }

  __device__ __forceinline__ void add(int c, int p, double2 k, double2 d) {
    double2 &x = acc[c][p];
    x.x = fma(k.x, d.x, x.x);
    x.y = fma(k.x, d.y, x.y);
    x.x = fma(-k.y, d.y, x.x);
    x.y = fma(k.y, d.x, x.y);
  }

  __device__ __forceinline__ void flush(double *sre, double *sim, int key,
                                        const MosaicShape &m) {
    const int base = (key & 255) * m.RS + ((key >> 8) & 255);
#pragma unroll
    for (int c = 0; c < CPL; ++c)
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        const double2 v = acc[c][p];
        if (own[c] && ipm[p] >= 0 && (v.x != 0.0 || v.y != 0.0)) {
          const int e = ipm[p] * m.PS + base + cell[c];
          atomicAdd(sre + e, v.x);
          atomicAdd(sim + e, v.y);
        }
      }
    clear();
  }
};

template <int CPL, int NPOL, bool MULTI>
__global__ void __launch_bounds__(MR_THREADS, CPL *NPOL <= 4 ? 2 : 1)
    k_mosaic_runs(MosaicRunsArgs q) {
  const MosaicTiledArgs &t = q.t;
  const MosaicArgs &a = t.m;
  constexpr int NF = MULTI ? NPOL : 1;  // tap rows per sample
  // samples whose taps are loaded together: two where a sample has up to 4
  // loads per lane (225 us of the 1.03M samples with their chunks in record
  // order; four at a time 256 us, for their registers), else one (up to 16)
  constexpr int AHEAD = NF * CPL <= 4 ? 2 : 1;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int S = t.S, S2 = S * S, npg = (int)a.n_img_pol;
  const MosaicShape m(S);
  double2 *wd = (double2 *)smem + warp * MR_ROUND * NPOL;
  int *tr = (int *)(smem + (size_t)MR_WARPS * MR_ROUND * NPOL * sizeof(double2)) +
            warp * MR_ROUND * NPOL;
  double *sre = (double *)(smem + mosaic_stage_bytes<NPOL>());
  double *sim = sre + (size_t)npg * m.PS;
  __shared__ int s_chunk;

  MosaicLanes<CPL, NPOL, MULTI> lanes;
  int cfp[NPOL];
#pragma unroll
  for (int p = 0; p < NPOL; ++p) {
    const int ap = p < a.npol ? a.pol_map[p] : -1;
    cfp[p] = p < a.npol ? a.cfp_map[p] : -1;
    lanes.ipm[p] = ap >= 0 && ap < npg && cfp[p] >= 0 && cfp[p] < a.n_cfp ? ap : -1;
  }
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    const int i = lane + 32 * c;
    lanes.own[c] = i < S2;
    lanes.cell[c] = (i / S) * m.RS + i % S;
  }
  lanes.clear();
  for (int i0 = 0; i0 < 2 * npg * m.PS; i0 += MR_THREADS) {
    const int i = i0 + threadIdx.x;
    if (i < 2 * npg * m.PS) sre[i] = 0.0;
  }
  const uint32_t n_rec = *t.n_rec;
  const int64_t n_chunks = ((int64_t)n_rec + t.chunk - 1) / t.chunk;
  for (;;) {
    __syncthreads();  // sub-grid clear; previous s_chunk consumed
    if (threadIdx.x == 0)
      s_chunk = chunk_in_turn(atomicAdd(&t.sched[0], 1u), (uint32_t)n_chunks,
                              (uint32_t)(t.n_tiles / (t.ntu * t.ntv)));
    __syncthreads();
    const int64_t ch = s_chunk;
    if (ch >= n_chunks) break;
    const uint32_t r0 = (uint32_t)(ch * t.chunk);
    const uint32_t r1 = (uint32_t)min((int64_t)n_rec, (int64_t)r0 + t.chunk);
    int64_t tile = find_tile_warp(t.tile_start, t.n_tiles, r0);
    uint32_t seg_lo = r0;
    while (seg_lo < r1) {
      const uint32_t t_end = t.tile_start[tile + 1];
      const uint32_t seg_hi = min(r1, t_end);
      if (seg_hi <= seg_lo) {
        ++tile;
        continue;
      }
      const int64_t plane = tile / (t.ntu * t.ntv);
      const int64_t trem = tile - plane * t.ntu * t.ntv;
      const int tu = (int)(trem / t.ntv), tv = (int)(trem - (int64_t)tu * t.ntv);
      const uint32_t seg_n = seg_hi - seg_lo;
      const uint32_t w_lo = seg_lo + (uint32_t)(((uint64_t)seg_n * warp) / MR_WARPS);
      const uint32_t w_hi = seg_lo + (uint32_t)(((uint64_t)seg_n * (warp + 1)) / MR_WARPS);
      const int n_rounds = (int)((w_hi - w_lo + MR_ROUND - 1) / MR_ROUND);
      int cur = -1;
      double sw[NPOL];
#pragma unroll
      for (int p = 0; p < NPOL; ++p) sw[p] = 0.0;
      auto load_rec = [&](int rd) {
        const uint32_t r = w_lo + (uint32_t)rd * MR_ROUND + lane;
        Rec x;
        if (rd < n_rounds && r < w_hi) x = t.recs[r];
        else x.row = 0xffffffffu;
        return x;
      };
      MosaicRaw<NPOL> raw;
      Rec next = load_rec(0);
      mosaic_fetch<NPOL>(raw, a, next, next.row != 0xffffffffu);
      next = load_rec(1);
      for (int rd = 0; rd < n_rounds; ++rd) {
        // ---- stage one sample per lane
        int key = -1;
        bool inf = false;  // a value or a tap of the sample is not finite
        if (raw.ok) {
          const Rec rc = raw.rc;
          const uint32_t tb = fdiv(rc.row, t.div_nchan);
          const uint32_t c = rc.row - tb * (uint32_t)a.nchan;
          const uint32_t b = tb - fdiv(tb, t.div_nb) * (uint32_t)a.nb;
          const int cfb = a.cfb_map[b], cfc = a.cfc_map[c];
          const bool has = cfb >= 0 && cfb < a.n_cfb && cfc >= 0 && cfc < a.n_cfc;
          const int ou = min(max((int)rc.ou - 128 - q.first, 0), q.n_off - 1);
          const int ov = min(max((int)rc.ov - 128 - q.first, 0), q.n_off - 1);
          if (!MULTI) tr[lane] = q.zero_row;
#pragma unroll
          for (int p = 0; p < NPOL; ++p) {
            double2 d;
            if (a.do_psf) d = make_double2(raw.w[p], 0.0);
            else d = make_double2(__dmul_rn(raw.v[p].x, raw.w[p]),
                                  __dmul_rn(raw.v[p].y, raw.w[p]));
            bool ok = has && lanes.ipm[p] >= 0 && !isnan(d.x) && !isnan(d.y) &&
                      (d.x != 0.0 || d.y != 0.0);
            int row = q.zero_row;
            if (ok) {
              const int64_t fidx = ((int64_t)cfb * a.n_cfc + cfc) * a.n_cfp + cfp[p];
              const int su = a.support[2 * fidx], sv = a.support[2 * fidx + 1];
              // a window larger than the plan's footprint (max_support) is skipped
              ok = su >= 1 && sv >= 1 && su <= S && sv <= S;
              if (ok) row = (int)((fidx * q.n_off + ou) * q.n_off + ov);
            }
            wd[p * MR_ROUND + lane] = ok ? d : make_double2(0.0, 0.0);
            if (ok) {
              const double2 nm = __ldg(q.norm + row);
              sw[p] += __dmul_rn(raw.w[p], nm.x);
              inf |= !(fabs(d.x) + fabs(d.y) + nm.y < CUDART_INF);
            }
            if (MULTI || ok) tr[(MULTI ? p : 0) * MR_ROUND + lane] = row;
          }
          key = (int)rc.du | ((int)rc.dv << 8);
        }
        int prev = __shfl_up_sync(0xffffffffu, key, 1);
        if (lane == 0) prev = cur;
        const unsigned starts = __ballot_sync(0xffffffffu, key >= 0 && key != prev);
        const unsigned infs = __ballot_sync(0xffffffffu, inf);
        // ---- the next round's loads, before this one is computed
        mosaic_fetch<NPOL>(raw, a, next, next.row != 0xffffffffu);
        next = load_rec(rd + 2);
        __syncwarp();
        const int jn = (int)min((uint32_t)MR_ROUND, w_hi - (w_lo + (uint32_t)rd * MR_ROUND));
        if (infs == 0u) {
          for (int j0 = 0; j0 < jn; j0 += AHEAD) {
            double2 cv[AHEAD][NF][CPL];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u)
#pragma unroll
              for (int f = 0; f < NF; ++f) {
                const int j = min(j0 + u, jn - 1);
                const double2 *row = q.taps + (int64_t)tr[f * MR_ROUND + j] * S2;
#pragma unroll
                for (int c = 0; c < CPL; ++c)
                  cv[u][f][c] =
                      lanes.own[c] ? __ldg(row + lane + 32 * c) : make_double2(0.0, 0.0);
              }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
              const int j = j0 + u;
              if (j >= jn) break;
              if ((starts >> j) & 1u) {
                if (cur >= 0) lanes.flush(sre, sim, cur, m);
                cur = __shfl_sync(0xffffffffu, key, j);
              }
#pragma unroll
              for (int p = 0; p < NPOL; ++p)
#pragma unroll
                for (int c = 0; c < CPL; ++c)
                  lanes.add(c, p, cv[u][MULTI ? p : 0][c], wd[p * MR_ROUND + j]);
            }
          }
        } else {
          for (int j = 0; j < jn; ++j) {
            if ((starts >> j) & 1u) {
              if (cur >= 0) lanes.flush(sre, sim, cur, m);
              cur = __shfl_sync(0xffffffffu, key, j);
            }
#pragma unroll
            for (int p = 0; p < NPOL; ++p) {
              const double2 d = wd[p * MR_ROUND + j];
              if (d.x == 0.0 && d.y == 0.0) continue;  // skipped: its row may be the zeros
#pragma unroll
              for (int c = 0; c < CPL; ++c) {
                const int row = tr[(MULTI ? p : 0) * MR_ROUND + j], i = lane + 32 * c;
                const int per = q.n_off * q.n_off;
                int64_t at;
                if (lanes.own[c] &&
                    mosaic_tap(a, row / per, S, i / S, i % S, q.first + row / q.n_off % q.n_off,
                               q.first + row % q.n_off, at))
                  lanes.add(c, p, __ldg(a.cf + at), d);
              }
            }
          }
        }
        __syncwarp();
      }
      if (cur >= 0) lanes.flush(sre, sim, cur, m);
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        double v = sw[p];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && a.sumw && lanes.ipm[p] >= 0 && v != 0.0)
          atomicAdd(&a.sumw[plane * npg + lanes.ipm[p]], v);
      }
      __syncthreads();
      // the segment's sub-grid to the global grid, a warp per row, cleared
      for (int rr = warp; rr < npg * m.W; rr += MR_WARPS) {
        const int gp = rr / m.W, iu = rr - gp * m.W;
        double2 *gd = a.grid + ((plane * npg + gp) * a.n_u + (int64_t)tu * TILE + iu) * a.n_v +
                      (int64_t)tv * TILE;
        for (int iv = lane; iv < m.W; iv += 32) {
          const int e = gp * m.PS + iu * m.RS + iv;
          const double vr = sre[e], vi = sim[e];
          if (vr == 0.0 && vi == 0.0) continue;
          atomicAdd(&gd[iv].x, vr);
          atomicAdd(&gd[iv].y, vi);
          sre[e] = 0.0;
          sim[e] = 0.0;
        }
      }
      __syncthreads();
      seg_lo = seg_hi;
      if (seg_hi == t_end) ++tile;
    }
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&t.sched[1], 1u) == gridDim.x - 1) {
      t.sched[0] = 0u;
      t.sched[1] = 0u;
      __threadfence();
    }
  }
}

static int64_t mosaic_tap_rows(int64_t n_cf, int os) { return n_cf * (os + 1) * (os + 1) + 1; }

static size_t mosaic_runs_smem(int S, int64_t n_img_pol, int npol_t) {
  const size_t stage = (size_t)MR_WARPS * MR_ROUND * npol_t * (sizeof(double2) + sizeof(int));
  return stage + (size_t)2 * n_img_pol * MosaicShape(S).PS * sizeof(double);
}

template <int CPL, int NPOL, bool MULTI>
static int launch_mosaic_runs(const MosaicRunsArgs &q, int64_t n_chunks, cudaStream_t st) {
  const size_t smem = mosaic_runs_smem(q.t.S, q.t.m.n_img_pol, NPOL);
  auto kernel = k_mosaic_runs<CPL, NPOL, MULTI>;
  AV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 1;
  AV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, MR_THREADS, smem));
  const int64_t most = (int64_t)sm_count() * std::max(per_sm, 1);
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min(most, n_chunks));
  kernel<<<blocks, MR_THREADS, smem, st>>>(q);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

template <int CPL, int NPOL>
static int launch_mosaic_runs(const MosaicRunsArgs &q, int64_t n_chunks, cudaStream_t st) {
  // one tap row per sample when there is one function per (baseline, channel)
  return q.t.m.n_cfp == 1 ? launch_mosaic_runs<CPL, NPOL, false>(q, n_chunks, st)
                          : launch_mosaic_runs<CPL, NPOL, true>(q, n_chunks, st);
}

template <int CPL>
static int launch_mosaic_runs(const MosaicRunsArgs &q, int64_t n_chunks, cudaStream_t st) {
  if (q.t.m.npol <= 1) return launch_mosaic_runs<CPL, 1>(q, n_chunks, st);
  if (q.t.m.npol <= 2) return launch_mosaic_runs<CPL, 2>(q, n_chunks, st);
  return launch_mosaic_runs<CPL, 4>(q, n_chunks, st);
}

static size_t mosaic_tiled_smem(int S, int64_t n_img_pol) {
  const int W = TILE + S - 1;
  return (size_t)W * W * (size_t)n_img_pol * sizeof(double2);
}

static int mosaic_geom(PlanGeom &g, Plan &p, int64_t n_u, int64_t n_v, int max_support,
                       int os, int64_t nt, int64_t nb, int64_t nchan, int64_t n_img_chan,
                       void *workspace, size_t workspace_bytes, const char *who) {
  AV_CHECK_ARG(max_support >= 1 && max_support <= 32, "%s: max_support must be in [1, 32]",
               who);
  AV_CHECK_ARG(os >= 1 && os <= 254, "%s: oversampling must be in [1, 254]", who);
  AV_CHECK_ARG(n_u > 2 * max_support && n_v > 2 * max_support && n_u < 131072 &&
                   n_v < 131072,
               "%s: grid size out of range", who);
  AV_CHECK_ARG(nt >= 0 && nb >= 0 && nchan >= 0 && n_img_chan >= 1, "%s: bad shape", who);
  AV_CHECK_ARG(workspace && (((uintptr_t)workspace) & 255) == 0,
               "%s: workspace must be 256-byte aligned", who);
  plan_geometry(g, nt, nb, nchan, n_img_chan, n_u, n_v, max_support, os);
  g.margin = max_support;
  g.convention = 0;
  g.chk_x = g.chk_y = 0;
  g.scale0 = g.scale1 = g.offset0 = g.offset1 = 0.0;
  const size_t need = plan_workspace_bytes(g);
  if (workspace_bytes < need) {
    set_error("%s: workspace %zu bytes < %zu needed", who, workspace_bytes, need);
    return AV_ERR_WORKSPACE;
  }
  Workspace ws(workspace, workspace_bytes);
  if (!plan_carve(g, ws, p)) {
    set_error("%s: workspace carve failed", who);
    return AV_ERR_WORKSPACE;
  }
  return AV_OK;
}

static unsigned mg_blocks(int64_t n_items, int per_block) {
  int64_t b = (n_items + per_block - 1) / per_block;
  const int64_t cap = (int64_t)sm_count() * 32;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

static int fill_mosaic(MosaicArgs &a, void *grid, double *sum_weight, int do_psf,
                       const void *vis, const double *weight, const double *uvw,
                       const double *freq, const int32_t *chan_map, const int32_t *pol_map,
                       const int32_t *cfb_map, const int32_t *cfc_map, const int32_t *cfp_map,
                       const void *cf, int64_t n_cfb, int64_t n_cfc, int64_t n_cfp,
                       int64_t conv_u, int64_t conv_v, const int32_t *support,
                       int max_support, int64_t n_u, int64_t n_v, double delta_l,
                       double delta_m, int os_u, int os_v, int64_t nt, int64_t nb,
                       int64_t nchan, int64_t npol, int64_t n_img_chan, int64_t n_img_pol) {
  a.grid = (double2 *)grid;
  a.sumw = sum_weight;
  a.do_psf = do_psf;
  a.vis = (const double2 *)vis;
  a.wt = weight;
  a.uvw = uvw;
  a.freq = freq;
  a.chan_map = chan_map;
  a.pol_map = pol_map;
  a.cfb_map = cfb_map;
  a.cfc_map = cfc_map;
  a.cfp_map = cfp_map;
  a.cf = (const double2 *)cf;
  a.n_cfb = n_cfb;
  a.n_cfc = n_cfc;
  a.n_cfp = n_cfp;
  a.cu = conv_u;
  a.cv = conv_v;
  a.support = support;
  a.max_support = max_support;
  a.n_u = n_u;
  a.n_v = n_v;
  a.dl0 = delta_l;
  a.dl1 = delta_m;
  a.os_u = os_u;
  a.os_v = os_v;
  a.nt = nt;
  a.nb = nb;
  a.nchan = nchan;
  a.npol = npol;
  a.n_img_chan = n_img_chan;
  a.n_img_pol = n_img_pol;
  return AV_OK;
}

}  // namespace av

using namespace av;

extern "C" {

int av_cf_phase_product(const void *conv_kernel, int kernel_dtype, const void *phase_gradient,
                        void *out, int64_t n_cf, int64_t conv_u, int64_t conv_v, void *stream) {
  clear_error();
  AV_CHECK_ARG(conv_kernel && phase_gradient && out, "av_cf_phase_product: null pointer");
  AV_CHECK_ARG(kernel_dtype == AV_F64 || kernel_dtype == AV_C128,
               "av_cf_phase_product: kernel must be float64 or complex128");
  AV_CHECK_ARG(n_cf >= 0 && conv_u >= 1 && conv_v >= 1, "av_cf_phase_product: bad shape");
  if (n_cf == 0) return AV_OK;
  const int64_t n = n_cf * conv_u * conv_v;
  k_cf_phase_product<<<mg_blocks(n, 256), 256, 0, as_stream(stream)>>>(
      conv_kernel, kernel_dtype == AV_C128, (const double2 *)phase_gradient, (double2 *)out,
      n_cf, conv_u * conv_v);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

int av_airy_pattern(double *out, const double *dish_diameters, const double *blockage_diameters,
                    int64_t n_dish, const double *freq, int64_t n_freq, int64_t n_pol,
                    int64_t nx, int64_t ny, int64_t cx, int64_t cy, double cell_x,
                    double cell_y, int ipower, int casa, int rorder, void *stream) {
  clear_error();
  AV_CHECK_ARG(out && dish_diameters && blockage_diameters && freq,
               "av_airy_pattern: null pointer");
  AV_CHECK_ARG(n_dish >= 1 && n_dish <= 16, "av_airy_pattern: 1 to 16 dish types");
  AV_CHECK_ARG(n_freq >= 1 && n_pol >= 1 && nx >= 1 && ny >= 1 && ipower >= 0 && ipower <= 8,
               "av_airy_pattern: bad shape or power");
  AiryArgs a;
  a.out = out;
  a.n_dish = n_dish;
  a.n_freq = n_freq;
  a.nx = nx;
  a.ny = ny;
  a.cx = cx;
  a.cy = cy;
  a.n_pol = n_pol;
  a.cell_x = cell_x;
  a.cell_y = cell_y;
  a.ipower = ipower;
  a.casa = casa;
  a.rorder = rorder;
  a.freq = freq;
  for (int i = 0; i < 16; ++i) {
    a.dish[i] = i < n_dish ? dish_diameters[i] : 0.0;
    a.block[i] = i < n_dish ? blockage_diameters[i] : 0.0;
  }
  const int64_t n = n_dish * n_freq * nx * ny;
  k_airy_pattern<<<mg_blocks(n, 256), 256, 0, as_stream(stream)>>>(a);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

#define AV_MOSAIC_PARAMS                                                                   \
  void *grid, double *sum_weight, int do_psf, const void *vis, const double *weight,       \
      const double *uvw, const double *freq, const int32_t *chan_map,                      \
      const int32_t *pol_map, const int32_t *cf_baseline_map, const int32_t *cf_chan_map,  \
      const int32_t *cf_pol_map, const void *cf, int64_t n_cf_baseline, int64_t n_cf_chan, \
      int64_t n_cf_pol, int64_t conv_u, int64_t conv_v, const int32_t *support,            \
      int max_support, int64_t n_u, int64_t n_v, double delta_l, double delta_m, int os_u, \
      int os_v, int64_t nt, int64_t nb, int64_t nchan, int64_t npol, int64_t n_img_chan,    \
      int64_t n_img_pol

static int check_mosaic(const char *who, AV_MOSAIC_PARAMS) {
  AV_CHECK_ARG(grid && weight && uvw && freq && chan_map && pol_map && cf_baseline_map &&
                   cf_chan_map && cf_pol_map && cf && support,
               "%s: null pointer", who);
  AV_CHECK_ARG(do_psf || vis, "%s: vis is required unless do_psf", who);
  AV_CHECK_ARG(n_cf_baseline >= 1 && n_cf_chan >= 1 && n_cf_pol >= 1 && conv_u >= 1 &&
                   conv_v >= 1,
               "%s: bad convolution-function shape", who);
  AV_CHECK_ARG(n_u >= 1 && n_v >= 1 && os_u >= 1 && os_v >= 1 && max_support >= 0,
               "%s: bad grid or oversampling", who);
  AV_CHECK_ARG(nt >= 0 && nb >= 0 && nchan >= 0 && npol >= 0 && n_img_chan >= 1 &&
                   n_img_pol >= 1,
               "%s: bad shape", who);
  return AV_OK;
}

int av_mosaic_grid(AV_MOSAIC_PARAMS, void *stream) {
  clear_error();
  int rc = check_mosaic("av_mosaic_grid", grid, sum_weight, do_psf, vis, weight, uvw, freq,
                        chan_map, pol_map, cf_baseline_map, cf_chan_map, cf_pol_map, cf,
                        n_cf_baseline, n_cf_chan, n_cf_pol, conv_u, conv_v, support,
                        max_support, n_u, n_v, delta_l, delta_m, os_u, os_v, nt, nb, nchan,
                        npol, n_img_chan, n_img_pol);
  if (rc) return rc;
  const int64_t rows = nt * nb * nchan;
  if (rows == 0 || npol == 0) return AV_OK;
  MosaicArgs a;
  fill_mosaic(a, grid, sum_weight, do_psf, vis, weight, uvw, freq, chan_map, pol_map,
              cf_baseline_map, cf_chan_map, cf_pol_map, cf, n_cf_baseline, n_cf_chan, n_cf_pol,
              conv_u, conv_v, support, max_support, n_u, n_v, delta_l, delta_m, os_u, os_v, nt,
              nb, nchan, npol, n_img_chan, n_img_pol);
  k_mosaic_grid<<<mg_blocks(rows, MG_THREADS / 32), MG_THREADS, 0, as_stream(stream)>>>(a);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

size_t av_mosaic_tiled_workspace_size(int64_t nt, int64_t nb, int64_t nchan, int64_t n_u,
                                      int64_t n_v, int64_t n_img_chan, int max_support) {
  PlanGeom g;
  plan_geometry(g, nt, nb, nchan, n_img_chan, n_u, n_v, max_support < 1 ? 1 : max_support,
                100);
  return plan_workspace_bytes(g);
}

int av_mosaic_tiled_plan(const double *uvw, const double *freq, const int32_t *chan_map,
                         int64_t n_u, int64_t n_v, double delta_l, double delta_m,
                         int max_support, int oversampling, int64_t nt, int64_t nb,
                         int64_t nchan, int64_t n_img_chan, void *workspace,
                         size_t workspace_bytes, void *stream) {
  clear_error();
  AV_CHECK_ARG(uvw && freq && chan_map, "av_mosaic_tiled_plan: null pointer");
  PlanGeom g;
  Plan p;
  int rc = mosaic_geom(g, p, n_u, n_v, max_support, oversampling, nt, nb, nchan, n_img_chan,
                       workspace, workspace_bytes, "av_mosaic_tiled_plan");
  if (rc) return rc;
  return plan_build(g, p, uvw, freq, chan_map, delta_l, delta_m, as_stream(stream));
}

int av_mosaic_tiled_execute(AV_MOSAIC_PARAMS, void *workspace, size_t workspace_bytes,
                            void *stream) {
  clear_error();
  int rc = check_mosaic("av_mosaic_tiled_execute", grid, sum_weight, do_psf, vis, weight, uvw,
                        freq, chan_map, pol_map, cf_baseline_map, cf_chan_map, cf_pol_map, cf,
                        n_cf_baseline, n_cf_chan, n_cf_pol, conv_u, conv_v, support,
                        max_support, n_u, n_v, delta_l, delta_m, os_u, os_v, nt, nb, nchan,
                        npol, n_img_chan, n_img_pol);
  if (rc) return rc;
  AV_CHECK_ARG(os_u == os_v, "av_mosaic_tiled_execute: oversampling must be the same on u, v");
  AV_CHECK_ARG(n_img_pol <= 4, "av_mosaic_tiled_execute: at most 4 image polarisations");
  const size_t smem = mosaic_tiled_smem(max_support, n_img_pol);
  AV_CHECK_ARG(smem <= 220 * 1024,
               "av_mosaic_tiled_execute: sub-grid of %zu bytes exceeds shared memory", smem);
  PlanGeom g;
  Plan p;
  rc = mosaic_geom(g, p, n_u, n_v, max_support, os_u, nt, nb, nchan, n_img_chan, workspace,
                   workspace_bytes, "av_mosaic_tiled_execute");
  if (rc) return rc;
  const int64_t rows = nt * nb * nchan;
  if (rows == 0 || npol == 0) return AV_OK;
  MosaicTiledArgs t;
  fill_mosaic(t.m, grid, sum_weight, do_psf, vis, weight, uvw, freq, chan_map, pol_map,
              cf_baseline_map, cf_chan_map, cf_pol_map, cf, n_cf_baseline, n_cf_chan, n_cf_pol,
              conv_u, conv_v, support, max_support, n_u, n_v, delta_l, delta_m, os_u, os_v, nt,
              nb, nchan, npol, n_img_chan, n_img_pol);
  t.recs = p.recs;
  t.tile_start = p.tile_start;
  t.n_rec = p.n_rec;
  t.sched = p.counters;
  t.n_tiles = g.n_tiles();
  t.ntu = g.ntu;
  t.ntv = g.ntv;
  t.S = max_support;
  t.W = TILE + max_support - 1;
  t.div_nchan = fast_div((uint32_t)nchan);
  t.div_nb = fast_div((uint32_t)nb);
  const int sms = sm_count();
  int64_t chunk = (rows + (int64_t)sms * 16 - 1) / ((int64_t)sms * 16);
  if (chunk < 1024) chunk = 1024;
  t.chunk = chunk;
  int64_t nblocks = (rows + chunk - 1) / chunk;
  if (nblocks > sms) nblocks = sms;
  if (nblocks < 1) nblocks = 1;
  if (smem > 48 * 1024)
    AV_CUDA(cudaFuncSetAttribute(k_mosaic_tiled, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  k_mosaic_tiled<<<(unsigned)nblocks, MT_THREADS, smem, as_stream(stream)>>>(t);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

size_t av_mosaic_taps_size(int64_t n_cf, int max_support, int oversampling) {
  if (n_cf < 1 || max_support < 1 || oversampling < 1) return 0;
  const size_t rows = (size_t)mosaic_tap_rows(n_cf, oversampling);
  return Workspace::need(rows * max_support * max_support * sizeof(double2)) +
         Workspace::need(rows * sizeof(double2));
}

int av_mosaic_runs_execute(AV_MOSAIC_PARAMS, void *workspace, size_t workspace_bytes, void *taps,
                           size_t taps_bytes, void *stream) {
  clear_error();
  const char *who = "av_mosaic_runs_execute";
  int rc = check_mosaic(who, grid, sum_weight, do_psf, vis, weight, uvw, freq, chan_map, pol_map,
                        cf_baseline_map, cf_chan_map, cf_pol_map, cf, n_cf_baseline, n_cf_chan,
                        n_cf_pol, conv_u, conv_v, support, max_support, n_u, n_v, delta_l,
                        delta_m, os_u, os_v, nt, nb, nchan, npol, n_img_chan, n_img_pol);
  if (rc) return rc;
  AV_CHECK_ARG(os_u == os_v, "%s: oversampling must be the same on u, v", who);
  AV_CHECK_ARG(n_img_pol <= 4 && npol <= 4, "%s: at most 4 polarisations", who);
  AV_CHECK_ARG(max_support <= MR_MAX_S, "%s: max_support above %d", who, MR_MAX_S);
  const int64_t n_cf = n_cf_baseline * n_cf_chan * n_cf_pol;
  const int64_t rows_t = mosaic_tap_rows(n_cf, os_u);
  AV_CHECK_ARG(rows_t <= 0x7fffffff, "%s: too many functions and offsets", who);
  if (!taps || (((uintptr_t)taps) & 255) != 0 ||
      taps_bytes < av_mosaic_taps_size(n_cf, max_support, os_u)) {
    set_error("%s: tap workspace missing, misaligned or too small", who);
    return AV_ERR_WORKSPACE;
  }
  PlanGeom g;
  Plan p;
  rc = mosaic_geom(g, p, n_u, n_v, max_support, os_u, nt, nb, nchan, n_img_chan, workspace,
                   workspace_bytes, who);
  if (rc) return rc;
  const int64_t rows = nt * nb * nchan;
  if (rows == 0 || npol == 0) return AV_OK;
  MosaicRunsArgs q;
  MosaicTiledArgs &t = q.t;
  fill_mosaic(t.m, grid, sum_weight, do_psf, vis, weight, uvw, freq, chan_map, pol_map,
              cf_baseline_map, cf_chan_map, cf_pol_map, cf, n_cf_baseline, n_cf_chan, n_cf_pol,
              conv_u, conv_v, support, max_support, n_u, n_v, delta_l, delta_m, os_u, os_v, nt,
              nb, nchan, npol, n_img_chan, n_img_pol);
  t.recs = p.recs;
  t.tile_start = p.tile_start;
  t.n_rec = p.n_rec;
  t.sched = p.counters;
  t.n_tiles = g.n_tiles();
  t.ntu = g.ntu;
  t.ntv = g.ntv;
  t.S = max_support;
  t.W = TILE + max_support - 1;
  t.div_nchan = fast_div((uint32_t)nchan);
  t.div_nb = fast_div((uint32_t)nb);
  // a chunk per CTA slot and a few more to even out their times; at least
  // 1024 records, so a chunk's sub-grid flush stays small against its samples
  const int64_t parts = (int64_t)sm_count() * 16;
  t.chunk = std::max<int64_t>(1024, (rows + parts - 1) / parts);
  Workspace tw(taps, taps_bytes);
  double2 *tab = tw.take<double2>((size_t)rows_t * max_support * max_support);
  double2 *norm = tw.take<double2>((size_t)rows_t);
  q.taps = tab;
  q.norm = norm;
  // floor((u - u_pos) os + 0.5) with |u - u_pos| <= 0.5
  q.first = -(os_u / 2);
  q.n_off = os_u + 1;
  q.zero_row = (int)(rows_t - 1);
  cudaStream_t st = as_stream(stream);
  k_mosaic_taps<<<(unsigned)rows_t, 128, 0, st>>>(t.m, max_support, q.first, q.n_off, tab, norm);
  AV_LAUNCH_CHECK();
  const int64_t n_chunks = (rows + t.chunk - 1) / t.chunk;
  const int cpl = (max_support * max_support + 31) / 32;
  if (cpl == 1) return launch_mosaic_runs<1>(q, n_chunks, st);
  if (cpl == 2) return launch_mosaic_runs<2>(q, n_chunks, st);
  if (cpl == 3) return launch_mosaic_runs<3>(q, n_chunks, st);
  return launch_mosaic_runs<4>(q, n_chunks, st);
}

size_t av_aperture_grid_workspace_size(int64_t n_cf_baseline, int64_t nchan, int64_t npol) {
  return Workspace::need(sizeof(double) * (size_t)(n_cf_baseline < 1 ? 1 : n_cf_baseline) *
                         (nchan < 1 ? 1 : nchan) * (npol < 1 ? 1 : npol));
}

int av_aperture_grid(AV_MOSAIC_PARAMS, void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  int rc = check_mosaic("av_aperture_grid", grid, sum_weight, 1, vis, weight, uvw, freq,
                        chan_map, pol_map, cf_baseline_map, cf_chan_map, cf_pol_map, cf,
                        n_cf_baseline, n_cf_chan, n_cf_pol, conv_u, conv_v, support,
                        max_support, n_u, n_v, delta_l, delta_m, os_u, os_v, nt, nb, nchan,
                        npol, n_img_chan, n_img_pol);
  if (rc) return rc;
  const int64_t rows = nt * nb * nchan;
  if (rows == 0 || npol == 0) return AV_OK;
  const int64_t n_cls = n_cf_baseline * nchan * npol;
  AV_CHECK_ARG(n_cls <= 0x7fffffff, "av_aperture_grid: too many weight classes");
  Workspace ws(workspace, workspace_bytes);
  double *cls = ws.take<double>((size_t)n_cls);
  AV_CHECK_ARG(cls, "av_aperture_grid: workspace too small");
  MosaicArgs a;
  fill_mosaic(a, grid, sum_weight, 1, nullptr, weight, uvw, freq, chan_map, pol_map,
              cf_baseline_map, cf_chan_map, cf_pol_map, cf, n_cf_baseline, n_cf_chan, n_cf_pol,
              conv_u, conv_v, support, max_support, n_u, n_v, delta_l, delta_m, os_u, os_v, nt,
              nb, nchan, npol, n_img_chan, n_img_pol);
  cudaStream_t st = as_stream(stream);
  AV_CUDA(cudaMemsetAsync(cls, 0, sizeof(double) * (size_t)n_cls, st));
  k_aperture_classes<<<mg_blocks(rows, MG_THREADS), MG_THREADS, 0, st>>>(a, cls);
  AV_LAUNCH_CHECK();
  k_aperture_add<<<(unsigned)n_cls, MG_THREADS, 0, st>>>(a, cls);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

}  // extern "C"
