// Natural / Briggs imaging weights (grid_imaging_weights.py:93-206, :285-443;
// briggs_weighting.py:1-31; the input preparation of
// calculate_imaging_weights.py:183-198, 228-261).
#include <math_constants.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace av {

// Polarisation-averaged weight of a sample, NaN where flagged
// (calculate_imaging_weights.py:185-198).
template <int NPOL, typename WT>
__device__ __forceinline__ double pol_avg_weight(const WT *wt, const uint8_t *flag,
                                                 int64_t row) {
  auto w = [&](int p) {
    const int64_t i = row * NPOL + p;
    double v = (double)wt[i];
    if (flag && flag[i]) v = CUDART_NAN;
    return v;
  };
  if (NPOL == 1) return w(0);
  return __dmul_rn(__dadd_rn(w(0), w(NPOL - 1)), 0.5);  // the reference's / 2, exactly
}

// uv scale of a channel along one axis (standard_grid.py:297-299).
__device__ __forceinline__ double uv_scale(double f, double dl, int64_t n) {
  return __ddiv_rn(-__dmul_rn(__dmul_rn(f, dl), (double)n), C_LIGHT);
}

// Nearest cell of a sample in the gridder's convention (int(x + 0.5)), its
// channel's scales given, and the cell of its conjugate.
__device__ __forceinline__ bool scaled_cell(double um, double vm, double us0, double us1,
                                            int64_t n_u, int64_t n_v, long long &ui,
                                            long long &vi, long long &uic, long long &vic) {
  double u = __dmul_rn(um, us0), v = __dmul_rn(vm, us1);
  if (isnan(u) || isnan(v)) return false;
  double u_pos = __dadd_rn(u, (double)(n_u / 2)), v_pos = __dadd_rn(v, (double)(n_v / 2));
  double u_pc = __dadd_rn(-u, (double)(n_u / 2)), v_pc = __dadd_rn(-v, (double)(n_v / 2));
  ui = trunc_ll(__dadd_rn(u_pos, 0.5));
  vi = trunc_ll(__dadd_rn(v_pos, 0.5));
  uic = trunc_ll(__dadd_rn(u_pc, 0.5));
  vic = trunc_ll(__dadd_rn(v_pc, 0.5));
  return (ui < n_u) && (vi < n_v) && (ui >= 0) && (vi >= 0);
}

__device__ __forceinline__ bool nearest_cell(double um, double vm, double f, double dl0,
                                             double dl1, int64_t n_u, int64_t n_v,
                                             long long &ui, long long &vi, long long &uic,
                                             long long &vic) {
  return scaled_cell(um, vm, uv_scale(f, dl0, n_u), uv_scale(f, dl1, n_v), n_u, n_v, ui, vi, uic,
                     vic);
}

// How k_weight_density and k_briggs_apply walk the samples: a thread takes
// `steps` consecutive times of one (baseline, channel) series.  Threads run
// over a group of channels, the baselines, the time blocks and the groups, in
// one line, so that few series leave no lane idle (1M samples of one series:
// weights 218 -> 34 us, density 660 -> 147, against blocks of 256 series).
// At each time the threads of a warp read neighbouring rows of 16 channels;
// the channel's uv scale, with its divides, is formed once; and since a
// baseline stays in one cell for several times, its weights are summed in a
// register and its density looked up once per cell.  A group of 16 channels
// keeps a warp's cells in 16 planes and several baselines of a channel in a
// block, for its sum: the density of one time of 2016 baselines x 512 channels
// takes 30 us, 37 in groups of 8, 56 of 32 (and 57 with all channels in one);
// of 64 times of 2016 x 32 channels 32, 32 and 36.  WT_UNROLL times are loaded
// together (2 with 4 blocks per SM; 4 at once spill there and take a fifth
// longer).
constexpr int WT_THREADS = 256, WT_UNROLL = 2;
constexpr int64_t WT_GROUP = 16;  // channels of a group, at most

// f(npol as a constant), npol 1, 2 or 4.
template <typename F>
static void with_pols(int64_t npol, F f) {
  if (npol == 1) f(std::integral_constant<int, 1>());
  else if (npol == 2) f(std::integral_constant<int, 2>());
  else f(std::integral_constant<int, 4>());
}

struct WeightWalk {
  int64_t steps, time_blocks;
  int64_t width, groups;  // channels of a group (the last one may have fewer)
  unsigned blocks;
};

// Two waves of 1024 threads per SM, at least WT_UNROLL times each.
static WeightWalk weight_walk(int64_t nt, int64_t nb, int64_t nchan) {
  WeightWalk w;
  w.groups = (nchan + WT_GROUP - 1) / WT_GROUP;
  w.width = (nchan + w.groups - 1) / w.groups;
  const int64_t series = nb * w.width * w.groups, want = (int64_t)sm_count() * 2048;
  const int64_t most = (nt + WT_UNROLL - 1) / WT_UNROLL;
  const int64_t parts = std::max<int64_t>(1, std::min(most, (want + series - 1) / series));
  w.steps = (nt + parts - 1) / parts;
  w.steps = (w.steps + WT_UNROLL - 1) / WT_UNROLL * WT_UNROLL;
  w.time_blocks = (nt + w.steps - 1) / w.steps;
  w.blocks = (unsigned)((series * w.time_blocks + WT_THREADS - 1) / WT_THREADS);
  return w;
}

// This thread's place in the walk.
struct WeightPlace {
  int64_t c, group_first, at;  // channel, its group's first one, first row of uvw
  int n;                       // times, none past the end
  __device__ __forceinline__ WeightPlace(const WeightWalk &w, int64_t nt, int64_t nb,
                                         int64_t nchan) {
    const int64_t k = blockIdx.x * (int64_t)WT_THREADS + threadIdx.x;
    const int64_t k1 = k / w.width, k2 = k1 / nb, group = k2 / w.time_blocks;
    group_first = group * w.width;
    c = group_first + (k - k1 * w.width);
    const int64_t t0 = (k2 - group * w.time_blocks) * w.steps;
    at = t0 * nb + (k1 - k2 * nb);
    n = c < nchan ? (int)std::min(nt - t0, w.steps) : 0;
  }
};

// Density grid and sums of weights.  One thread per sample in channel-major
// order, two global FP64 atomics each and the weights read with a stride of a
// whole row, had taken 270 us for 4.1M samples x 4 polarisations (float32,
// 32 planes of 1024^2); this walk takes DDD us.
template <int NPOL, typename WT>
__global__ void __launch_bounds__(WT_THREADS, 4) k_weight_density(
    double *G, double *sumw, const double *__restrict__ uvw, const double *__restrict__ freq,
    const WT *__restrict__ wt, const uint8_t *__restrict__ flag, int64_t n_u, int64_t n_v,
    double dl0, double dl1, int64_t nt, int64_t nb, int64_t nchan, WeightWalk walk) {
  // channels of the groups that the block's threads are of: a group between
  // two others has at least its channels in threads
  constexpr int WT_SUMS = WT_THREADS + 2 * (int)WT_GROUP;
  __shared__ double s_sum[WT_SUMS];
  __shared__ int64_t s_first;
  const WeightPlace place(walk, nt, nb, nchan);
  const int64_t c = place.c;
  if (threadIdx.x == 0) s_first = place.group_first;
  for (int i = threadIdx.x; i < WT_SUMS; i += WT_THREADS) s_sum[i] = 0.0;
  __syncthreads();
  double total = 0.0;
  if (place.n > 0) {
    const double us0 = uv_scale(freq[c], dl0, n_u), us1 = uv_scale(freq[c], dl1, n_v);
    double *plane = G + c * n_u * n_v;
    int64_t cell = -1, conj = -1;
    double acc = 0.0;
    auto flush = [&]() {
      if (cell >= 0 && acc != 0.0) {
        atomicAdd(plane + cell, acc);
        // the conjugate cell is not range-checked by the reference; it is out
        // of range only for index 0 of an even axis, skipped here
        if (conj >= 0) atomicAdd(plane + conj, acc);
      }
      acc = 0.0;
    };
    int64_t at_t = place.at;  // row of uvw
    for (int left = place.n; left > 0; left -= WT_UNROLL, at_t += WT_UNROLL * nb) {
      double um[WT_UNROLL], vm[WT_UNROLL], w[WT_UNROLL];
#pragma unroll
      for (int k = 0; k < WT_UNROLL; ++k)
        if (k < left) {
          const int64_t tb = at_t + k * nb;
          um[k] = uvw[3 * tb];
          vm[k] = uvw[3 * tb + 1];
          w[k] = pol_avg_weight<NPOL>(wt, flag, tb * nchan + c);
        }
#pragma unroll
      for (int k = 0; k < WT_UNROLL; ++k) {
        if (k >= left) continue;
        long long ui, vi, uic, vic;
        if (!scaled_cell(um[k], vm[k], us0, us1, n_u, n_v, ui, vi, uic, vic) || isnan(w[k]))
          continue;
        const int64_t at = ui * n_v + vi;
        const int64_t ac =
            uic >= 0 && uic < n_u && vic >= 0 && vic < n_v ? uic * n_v + vic : -1;
        if (at != cell || ac != conj) {
          flush();
          cell = at;
          conj = ac;
        }
        acc += w[k];
        total += __dmul_rn(2.0, w[k]);
      }
    }
    flush();
  }
  // sums of weights: one atomic per channel and block
  if (total != 0.0) atomicAdd(&s_sum[c - s_first], total);
  __syncthreads();
  for (int i = threadIdx.x; i < WT_SUMS; i += WT_THREADS)
    if (s_sum[i] != 0.0) atomicAdd(&sumw[s_first + i], s_sum[i]);
}

// sum(G^2) per plane: one CTA per (plane, slice), FP64 partials.
__global__ void __launch_bounds__(256) k_sum_sq(const double *G, int64_t plane_n,
                                                int slices, double *partial) {
  int64_t p = blockIdx.x / slices;
  int s = blockIdx.x - (int)p * slices;
  int64_t lo = plane_n * s / slices, hi = plane_n * (s + 1) / slices;
  const double *g = G + p * plane_n;
  double acc = 0.0;
  for (int64_t i0 = lo; i0 < hi; i0 += blockDim.x) {  // one trip count per block
    const int64_t i = i0 + threadIdx.x;
    if (i < hi) {
      double v = g[i];
      acc += v * v;
    }
  }
  __shared__ double sh[8];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
    partial[blockIdx.x] = t;
  }
}

// A warp per plane adds its partial sums (lane by lane, then in a tree: a
// fixed order).
__global__ void __launch_bounds__(128) k_briggs_finish(const double *partial, int slices,
                                                       const double *sumw, int64_t nplanes,
                                                       double robust, double *factors) {
  const int lane = threadIdx.x & 31;
  const int64_t p = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (p >= nplanes) return;
  double sq = 0.0;
  for (int s = lane; s < slices; s += 32) sq += partial[p * slices + s];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if (lane != 0) return;
  double r = 5.0 * pow(10.0, -robust);
  // (5 * 10^-R)^2 / (sum G^2 / sum w): NaN / inf pass through like numpy
  factors[p] = (r * r) / (sq / sumw[p]);
  factors[nplanes + p] = 1.0;
}

template <typename T>
struct PairOf {
  using type = double2;
};
template <>
struct PairOf<float> {
  using type = float2;
};

// Imaging weight of each sample, tiled to every polarisation
// (grid_imaging_weights.py:358-443 + calculate_imaging_weights.py:258-261),
// in the walk above (99 us for the case above with one thread per sample;
// 58 us now).
template <int NPOL, typename OT, typename WT>
__global__ void __launch_bounds__(WT_THREADS, 4) k_briggs_apply(
    OT *out, const double *__restrict__ G, const double *__restrict__ factors, int64_t nplanes,
    const double *__restrict__ uvw, const double *__restrict__ freq, const WT *__restrict__ wt,
    const uint8_t *__restrict__ flag, int64_t n_u, int64_t n_v, double dl0, double dl1,
    int64_t nt, int64_t nb, int64_t nchan, WeightWalk walk, int vec, int *err) {
  const WeightPlace place(walk, nt, nb, nchan);
  if (place.n <= 0) return;
  const int64_t c = place.c;
  const double us0 = uv_scale(freq[c], dl0, n_u), us1 = uv_scale(freq[c], dl1, n_v);
  const double f0 = factors[c], f1 = factors[nplanes + c];
  const bool bad = isnan(f0) || isnan(f1);
  const double *plane = G + c * n_u * n_v;
  int64_t cell = -1;
  double gij = 0.0;
  int64_t at_t = place.at;  // row of uvw
  for (int left = place.n; left > 0; left -= WT_UNROLL, at_t += WT_UNROLL * nb) {
    double um[WT_UNROLL], vm[WT_UNROLL], dw[WT_UNROLL];
#pragma unroll
    for (int k = 0; k < WT_UNROLL; ++k)
      if (k < left) {
        const int64_t tb = at_t + k * nb;
        um[k] = uvw[3 * tb];
        vm[k] = uvw[3 * tb + 1];
        dw[k] = pol_avg_weight<NPOL>(wt, flag, tb * nchan + c);
      }
#pragma unroll
    for (int k = 0; k < WT_UNROLL; ++k) {
      if (k >= left) continue;
      double iw = 0.0;  // off-grid samples keep the zero the reference allocates
      long long ui, vi, uic, vic;
      if (scaled_cell(um[k], vm[k], us0, us1, n_u, n_v, ui, vi, uic, vic)) {
        iw = dw[k];
        if (!isnan(iw) && iw != 0.0) {
          const int64_t at = ui * n_v + vi;
          if (at != cell) {
            cell = at;
            gij = __ldg(plane + at);
          }
          if (!isnan(gij) && gij != 0.0) {
            if (bad) atomicExch(err, 1);
            else iw = __ddiv_rn(iw, __dadd_rn(__dmul_rn(f0, gij), f1));
          }
        }
      }
      OT *o = out + ((at_t + k * nb) * nchan + c) * NPOL;
      const OT v = (OT)iw;
      if (NPOL > 1 && vec) {  // out is 16-byte aligned
        using V = typename PairOf<OT>::type;
        V pair;
        pair.x = pair.y = v;
#pragma unroll
        for (int p = 0; p < NPOL; p += 2) *(V *)(o + p) = pair;
      } else {
#pragma unroll
        for (int p = 0; p < NPOL; ++p) o[p] = v;
      }
    }
  }
}

// standard_imaging_weight_degrid_jit (standard_grid.py:487-604), one thread
// per (time, baseline, channel): for a sample whose nearest cell (gridder
// convention) is on the grid, every polarisation's weight becomes its
// natural weight (the mean of polarisations 0 and 1 when there are two),
// divided by f0 * G + f1 where both the polarisation's own natural weight
// and G, the imaging-weight grid of (chan_map[c], pol_map[p]) at that cell,
// are neither NaN nor zero.  Samples off the grid (or with NaN uv) are left
// as the caller's array holds them.
__global__ void __launch_bounds__(256) k_imaging_weight_degrid(
    double *out, const void *G, int g_dt, int64_t g_chan, int64_t g_pol, const double *factors,
    const double *uvw, const double *freq, const int32_t *chan_map, const int32_t *pol_map,
    const void *wt, int dt, int64_t n_u, int64_t n_v, double dl0, double dl1, int64_t nrows,
    int64_t nchan, int64_t npol) {
  const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (row >= nrows) return;
  const int64_t tb = row / nchan, c = row - tb * nchan;
  long long ui, vi, uic, vic;
  if (!nearest_cell(uvw[3 * tb], uvw[3 * tb + 1], freq[c], dl0, dl1, n_u, n_v, ui, vi, uic,
                    vic))
    return;
  auto w = [&](int64_t p) {
    const int64_t i = row * npol + p;
    return dt == AV_F32 ? (double)((const float *)wt)[i] : ((const double *)wt)[i];
  };
  const int64_t ac = chan_map[c];
  for (int64_t p = 0; p < npol; ++p) {
    const int64_t ap = pol_map[p];
    double iw = npol == 2 ? __ddiv_rn(__dadd_rn(w(0), w(1)), 2.0) : w(p);
    const double nat = w(p);
    if (!isnan(nat) && nat != 0.0) {
      const int64_t gi = ((ac * g_pol + ap) * n_u + ui) * n_v + vi;
      const double g =
          g_dt == AV_F32 ? (double)((const float *)G)[gi] : ((const double *)G)[gi];
      if (!isnan(g) && g != 0.0) {
        const int64_t fi = ac * g_pol + ap;
        const double den = __dadd_rn(__dmul_rn(factors[fi], g), factors[g_chan * g_pol + fi]);
        iw = __ddiv_rn(iw, den);
      }
    }
    out[row * npol + p] = iw;
  }
}

}  // namespace av

using namespace av;

extern "C" {

int av_weight_density(double *density, double *sum_weight, const double *uvw,
                      const double *freq, const void *wt, int wt_dtype, const uint8_t *flag,
                      int64_t n_u, int64_t n_v, double delta_l, double delta_m, int64_t nt,
                      int64_t nb, int64_t nchan, int64_t npol, void *stream) {
  clear_error();
  AV_CHECK_ARG(density && sum_weight && uvw && freq && wt, "av_weight_density: null pointer");
  AV_CHECK_ARG(wt_dtype == AV_F32 || wt_dtype == AV_F64, "av_weight_density: weight dtype");
  AV_CHECK_ARG(npol == 1 || npol == 2 || npol == 4, "av_weight_density: npol must be 1, 2 or 4");
  AV_CHECK_ARG(n_u > 0 && n_v > 0 && nt >= 0 && nb >= 0 && nchan >= 0,
               "av_weight_density: bad shape");
  if (nt * nb * nchan == 0) return AV_OK;
  const WeightWalk walk = weight_walk(nt, nb, nchan);
  auto run = [&](auto pol, const auto *w) {
    k_weight_density<decltype(pol)::value><<<walk.blocks, WT_THREADS, 0, as_stream(stream)>>>(
        density, sum_weight, uvw, freq, w, flag, n_u, n_v, delta_l, delta_m, nt, nb, nchan,
        walk);
  };
  with_pols(npol, [&](auto pol) {
    if (wt_dtype == AV_F32) run(pol, (const float *)wt);
    else run(pol, (const double *)wt);
  });
  AV_LAUNCH_CHECK();
  return AV_OK;
}

size_t av_briggs_factors_workspace_size(int64_t nplanes) {
  return Workspace::need(sizeof(double) * (size_t)nplanes * 64);
}

int av_briggs_factors(const double *density, const double *sum_weight, double *factors,
                         int64_t nplanes, int64_t n_u, int64_t n_v, double robust,
                         void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  AV_CHECK_ARG(density && sum_weight && factors, "av_briggs_factors: null pointer");
  AV_CHECK_ARG(nplanes >= 0 && n_u > 0 && n_v > 0, "av_briggs_factors: bad shape");
  if (nplanes == 0) return AV_OK;
  const int slices = 64;
  if (!workspace || workspace_bytes < av_briggs_factors_workspace_size(nplanes)) {
    set_error("av_briggs_factors: workspace too small");
    return AV_ERR_WORKSPACE;
  }
  cudaStream_t st = as_stream(stream);
  double *partial = (double *)workspace;
  k_sum_sq<<<(unsigned)(nplanes * slices), 256, 0, st>>>(density, n_u * n_v, slices, partial);
  AV_LAUNCH_CHECK();
  k_briggs_finish<<<(unsigned)((nplanes + 3) / 4), 128, 0, st>>>(partial, slices,
                                                                      sum_weight, nplanes,
                                                                      robust, factors);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

int av_briggs_apply(void *out, int out_dtype, const double *density, const double *factors,
                    const double *uvw, const double *freq, const void *wt, int wt_dtype,
                    const uint8_t *flag, int64_t n_u, int64_t n_v, double delta_l,
                    double delta_m, int64_t nt, int64_t nb, int64_t nchan, int64_t npol,
                    int32_t *err_flag, void *stream) {
  clear_error();
  AV_CHECK_ARG(out && density && factors && uvw && freq && wt && err_flag,
               "av_briggs_apply: null pointer");
  AV_CHECK_ARG(out_dtype == AV_F32 || out_dtype == AV_F64, "av_briggs_apply: out dtype");
  AV_CHECK_ARG(wt_dtype == AV_F32 || wt_dtype == AV_F64, "av_briggs_apply: weight dtype");
  AV_CHECK_ARG(npol == 1 || npol == 2 || npol == 4, "av_briggs_apply: npol must be 1, 2 or 4");
  if (nt * nb * nchan == 0) return AV_OK;
  const WeightWalk walk = weight_walk(nt, nb, nchan);
  const int vec = (((uintptr_t)out) & 15) == 0;
  auto run = [&](auto pol, auto *o, const auto *w) {
    k_briggs_apply<decltype(pol)::value><<<walk.blocks, WT_THREADS, 0, as_stream(stream)>>>(
        o, density, factors, nchan, uvw, freq, w, flag, n_u, n_v, delta_l, delta_m, nt, nb, nchan,
        walk, vec, err_flag);
  };
  with_pols(npol, [&](auto pol) {
    if (out_dtype == AV_F64 && wt_dtype == AV_F64) run(pol, (double *)out, (const double *)wt);
    else if (out_dtype == AV_F64) run(pol, (double *)out, (const float *)wt);
    else if (wt_dtype == AV_F64) run(pol, (float *)out, (const double *)wt);
    else run(pol, (float *)out, (const float *)wt);
  });
  AV_LAUNCH_CHECK();
  return AV_OK;
}

int av_imaging_weight_degrid(double *imaging_weight, const void *grid_imaging_weight,
                             int grid_dtype, int64_t g_chan, int64_t g_pol,
                             const double *briggs_factors, const double *uvw, const double *freq,
                             const int32_t *chan_map, const int32_t *pol_map,
                             const void *natural_weight, int wt_dtype, int64_t n_u, int64_t n_v,
                             double delta_l, double delta_m, int64_t nt, int64_t nb,
                             int64_t nchan, int64_t npol, void *stream) {
  clear_error();
  AV_CHECK_ARG(imaging_weight && grid_imaging_weight && briggs_factors && uvw && freq &&
                   chan_map && pol_map && natural_weight,
               "av_imaging_weight_degrid: null pointer");
  AV_CHECK_ARG(grid_dtype == AV_F32 || grid_dtype == AV_F64,
               "av_imaging_weight_degrid: grid dtype");
  AV_CHECK_ARG(wt_dtype == AV_F32 || wt_dtype == AV_F64,
               "av_imaging_weight_degrid: weight dtype");
  AV_CHECK_ARG(n_u > 0 && n_v > 0 && g_chan > 0 && g_pol > 0 && nt >= 0 && nb >= 0 &&
                   nchan >= 0 && npol >= 1,
               "av_imaging_weight_degrid: bad shape");
  const int64_t rows = nt * nb * nchan;
  if (rows == 0) return AV_OK;
  k_imaging_weight_degrid<<<(unsigned)((rows + 255) / 256), 256, 0, as_stream(stream)>>>(
      imaging_weight, grid_imaging_weight, grid_dtype, g_chan, g_pol, briggs_factors, uvw, freq,
      chan_map, pol_map, natural_weight, wt_dtype, n_u, n_v, delta_l, delta_m, rows, nchan,
      npol);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

}  // extern "C"

// ------------------------------------------------- allocation-free variant --
// Some callers may not allocate device memory: a host program whose device
// buffers all come from a pool it sized at start-up and that allows no
// cudaMalloc/cudaFree while it processes (an allocation there synchronises
// the device and can fail mid-run), or a plugin called by another framework
// that owns all device memory and hands it only inputs and outputs.  For them
// av_briggs_factors_noalloc keeps the reduction's partial sums in the static
// array below instead of a caller workspace.

namespace av {

constexpr int kBriggsSlices = 64;  // partial sums per plane, as av_briggs_factors
constexpr int kMaxDevices = 64;

// The partial sums of up to AV_BRIGGS_NOALLOC_MAX_PLANES planes (512 KiB).
// The module holds one copy on every device that loads it, until the process
// exits.  In host code this name is a host-side stand-in: the device address
// comes from cudaGetSymbolAddress, per device.
static __device__ __align__(256) double
    g_briggs_scratch[(size_t)AV_BRIGGS_NOALLOC_MAX_PLANES * kBriggsSlices];

static std::mutex g_briggs_scratch_mu;
static void *g_briggs_scratch_ptr[kMaxDevices];

// Device address of the current device's copy of g_briggs_scratch, looked up
// on the first call made with that device current and cached afterwards (the
// cache does not survive cudaDeviceReset, which may move the array).  The
// stream must belong to the current device: the kernels would otherwise run
// on another device with this device's address.
static int briggs_scratch(cudaStream_t st, void **out) {
  int dev = 0;
  AV_CUDA(cudaGetDevice(&dev));
  if (st != nullptr) {
    int sdev = dev;
    AV_CUDA(cudaStreamGetDevice(st, &sdev));
    if (sdev != dev) {
      set_error("av_briggs_factors_noalloc: the stream belongs to device %d, the current "
                "device is %d",
                sdev, dev);
      return AV_ERR_ARG;
    }
  }
  if (dev < 0 || dev >= kMaxDevices) {
    set_error("av_briggs_factors_noalloc: device %d beyond the %d this library tracks", dev,
              kMaxDevices);
    return AV_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_briggs_scratch_mu);
  if (!g_briggs_scratch_ptr[dev]) {
    void *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_briggs_scratch);
    if (e != cudaSuccess || !ptr) {
      set_error("av_briggs_factors_noalloc: cudaGetSymbolAddress on device %d: %s", dev,
                cudaGetErrorString(e));
      return AV_ERR_CUDA;
    }
    g_briggs_scratch_ptr[dev] = ptr;
  }
  *out = g_briggs_scratch_ptr[dev];
  return AV_OK;
}

}  // namespace av

extern "C" {

int av_briggs_factors_noalloc(const double *density, const double *sum_weight, double *factors,
                              int64_t nplanes, int64_t n_u, int64_t n_v, double robust,
                              void *stream) {
  clear_error();
  AV_CHECK_ARG(density && sum_weight && factors, "av_briggs_factors_noalloc: null pointer");
  AV_CHECK_ARG(nplanes >= 0 && n_u > 0 && n_v > 0, "av_briggs_factors_noalloc: bad shape");
  AV_CHECK_ARG(nplanes <= AV_BRIGGS_NOALLOC_MAX_PLANES,
               "av_briggs_factors_noalloc: %lld planes exceed the static scratch's maximum of "
               "%d planes; use av_briggs_factors with a workspace",
               (long long)nplanes, AV_BRIGGS_NOALLOC_MAX_PLANES);
  static_assert(sizeof(g_briggs_scratch) ==
                    (size_t)AV_BRIGGS_NOALLOC_MAX_PLANES * kBriggsSlices * sizeof(double),
                "scratch size");
  void *scratch = nullptr;
  int rc = briggs_scratch(as_stream(stream), &scratch);
  if (rc != AV_OK) return rc;
  // every partial k_briggs_finish reads, k_sum_sq of the same call writes
  // first: nothing needs clearing between calls
  return av_briggs_factors(density, sum_weight, factors, nplanes, n_u, n_v, robust, scratch,
                           sizeof(g_briggs_scratch), stream);
}

}  // extern "C"
