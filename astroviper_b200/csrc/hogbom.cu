// Hogbom CLEAN minor cycle (hclean::clean, hclean.cpp:106-210) and maximg
// (hclean.cpp:51-81) on one GPU.
//
// One cooperative persistent launch runs many iterations.  Every CTA owns a
// contiguous band of residual rows; when the band fits, it stays in shared
// memory for the whole launch.  Each iteration a CTA subtracts the scaled PSF
// from its band (where the PSF window covers it) and, in the same pass, finds
// the band's largest |r| inside the clean box (first maximum in row-major
// order wins, as the reference's strict '>').  CTAs publish one candidate
// each, meet at a grid barrier with a bounded wait, and every CTA reduces the
// candidates identically, so all of them agree on the next peak and on when
// to stop.  Arithmetic matches the reference bit for bit: products and
// differences are rounded separately (no FMA), the model is accumulated in
// iteration order by one thread.
#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "common.cuh"

namespace av {

struct __align__(16) HogState {
  int iter;      // next iteration
  int px, py;    // current peak
  int stopped;   // 1: threshold reached
  int err;       // device error (1 = barrier timeout)
  unsigned gen;  // barrier generation
  unsigned count;
  int pad;
  double peak;   // r[py, px] for iteration `iter`
  double absval; // |peak| found (0 when no pixel exceeded 0)
  // FP32: the iteration's winner as one 64-bit maximum over the CTAs, bits of
  // |r| above the complement of 2 * index + sign (0: no pixel above 0), two
  // of them used in turn; kpar: the one the next launch starts with
  double pad1[10];  // the keys on the second cache line, away from gen / count
  unsigned long long key[2];
  int kpar;
  int pad3;
  double pad2[13];
};
static_assert(sizeof(HogState) == 256, "state size");
static_assert(offsetof(HogState, key) == 128, "keys on their own cache line");

template <typename T>
struct __align__(16) HogCand {
  T absval;
  T val;
  T at_prev;      // r at the previous peak (owner CTA only)
  int idx;        // linear index of the band maximum (-1 none)
  int has_prev;
};

template <typename T>
struct HogArgs {
  T *model, *resid;
  const T *psf, *mask;
  int nx, ny, pnx, pny;
  int xbeg, xend, ybeg, yend;
  int niter, siter, iter_begin, iter_end;
  T gain, thres, speedup;
  HogState *state;
  HogCand<T> *cand;  // 2 x gridDim.x
  int init;
  int resident;
  unsigned long long timeout_ns;  // bounded wait at the grid barrier
};

__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rn_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double rn_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double rn_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float t_pow(float a, float b) { return powf(a, b); }
__device__ __forceinline__ double t_pow(double a, double b) { return pow(a, b); }

// (a_abs, a_idx) beats (b_abs, b_idx): larger |r|, then lower index.
template <typename T>
__device__ __forceinline__ bool beats(T aa, int ai, T ba, int bi) {
  if (ai < 0) return false;
  if (bi < 0) return true;
  return aa > ba || (aa == ba && ai < bi);
}

// Grid barrier with a bounded wait (timeout_ns of wall time, 2 s unless the
// AV_TUNE_HOGBOM_BARRIER_TIMEOUT_US knob says otherwise); returns false on
// timeout and records it in the state.  Every CTA adds itself to the count
// exactly once per barrier, timed out or not, so the last one to arrive still
// releases the barrier and no CTA waits beyond its own bound.
// The last CTA to arrive clears *reset (if given) before releasing the others.
__device__ bool grid_barrier(HogState *st, int *s_flag, unsigned long long timeout_ns,
                             unsigned long long *reset = nullptr) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned *vgen = &st->gen;
    unsigned g0 = *vgen;
    __threadfence();
    unsigned arrived = atomicAdd(&st->count, 1u);
    int ok = 1;
    if (arrived == gridDim.x - 1) {
      if (reset) atomicExch(reset, 0ull);
      atomicExch(&st->count, 0u);
      __threadfence();
      atomicAdd(&st->gen, 1u);
    } else {
      unsigned long long t0;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
      while (*vgen == g0) {
        __nanosleep(32);
        unsigned long long t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > timeout_ns) {
          ok = 0;
          atomicExch(&st->err, 1);
          break;
        }
      }
    }
    __threadfence();
    *s_flag = ok && (((volatile int *)&st->err)[0] == 0);
  }
  __syncthreads();
  return *s_flag != 0;
}

constexpr int HOG_THREADS = 1024;
// band pass for images up to HOG_NPR * HOG_THREADS columns: a thread's
// columns are fixed, so whether the PSF window and the clean box cover them
// is decided once per iteration and per row, not per pixel
constexpr int HOG_NPR = 2;
constexpr int HOG_RB = 7;  // rows whose PSF values are loaded together
// candidates a lane loads at once in the reduction after the grid barrier
constexpr int HOG_CPL = 4;

template <typename T>
__global__ void __launch_bounds__(HOG_THREADS, 1) k_hogbom(HogArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ T s_abs[32], s_val[32];
  __shared__ int s_idx[32];
  __shared__ int s_flag;
  __shared__ T s_prev;
  __shared__ int s_use_key;
  constexpr bool KEYED = std::is_same<T, float>::value;
  const int G = gridDim.x, b = blockIdx.x;
  const int y_lo = (int)((long long)a.ny * b / G), y_hi = (int)((long long)a.ny * (b + 1) / G);
  const int nx = a.nx;
  T *band = a.resident ? (T *)smem : a.resid + (size_t)y_lo * nx;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  if (a.resident) {
    // one trip count per block: every warp reaches the next barrier converged
    for (int i0 = 0; i0 < (y_hi - y_lo) * nx; i0 += HOG_THREADS) {
      const int i = i0 + threadIdx.x;
      if (i < (y_hi - y_lo) * nx) band[i] = a.resid[(size_t)y_lo * nx + i];
    }
  }
  // current peak
  int px, py, it = a.iter_begin;
  T peak = (T)0, absval = (T)0;
  if (a.init) {
    px = 0;
    py = 0;
  } else {
    px = a.state->px;
    py = a.state->py;
    peak = (T)a.state->peak;
    absval = (T)a.state->absval;
  }
  __syncthreads();

  int par = a.init ? 0 : a.state->kpar;
  bool first = a.init != 0;
  bool stopped = false;
  for (;;) {
    T pv = (T)0;
    bool do_sub = false;
    if (!first) {
      if (it >= a.iter_end) break;
      T cthres = a.thres;
      if (a.speedup > (T)0) cthres = a.thres * t_pow((T)2, (T)(it - a.siter) / a.speedup);
      if (absval < cthres) {
        stopped = true;
        break;
      }
      pv = rn_mul(a.gain, peak);
      do_sub = true;
      if (b == 0 && threadIdx.x == 0) {
        size_t mi = (size_t)py * nx + px;
        a.model[mi] = rn_add(a.model[mi], pv);
      }
    }
    // PSF window (hclean.cpp:172-175 with the PSF's own half sizes)
    const int x1 = max(0, px - a.pnx / 2), y1 = max(0, py - a.pny / 2);
    const int x2 = min(nx - 1, px + a.pnx / 2 - 1), y2 = min(a.ny - 1, py + a.pny / 2 - 1);
    // subtract + band argmax
    T best_abs = (T)0;
    int best_idx = -1;
    T best_val = (T)0;
    const int npr = (nx + HOG_THREADS - 1) / HOG_THREADS;
    const int tpr4 = nx >> 2;  // FP32, 4 pixels per thread: threads per row
    if (std::is_same<T, float>::value && (nx & 3) == 0 && tpr4 > 0 && tpr4 <= HOG_THREADS &&
        HOG_THREADS % tpr4 == 0) {
      // thread t: columns c0 .. c0 + 3 of rows y_lo + t / tpr4, + rpp, ...
      const int rpp = HOG_THREADS / tpr4;
      const int c0 = (threadIdx.x % tpr4) * 4, rofs = threadIdx.x / tpr4;
      // which of the 4 columns the PSF window (with an existing PSF column)
      // and the clean box cover, once per iteration
      const int wlo = max(x1, px - a.pnx / 2), whi = min(x2, px + a.pnx / 2 - 1);
      unsigned wm = 0u, bm = 0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = c0 + j;
        if (do_sub && c >= wlo && c <= whi) wm |= 1u << j;
        if (c >= a.xbeg && c < a.xend) bm |= 1u << j;
      }
      const int pxo0 = a.pnx / 2 + c0 - px;  // PSF column of c0
      for (int iy = y_lo + rofs; iy < y_hi; iy += rpp) {
        const int psf_y = a.pny / 2 + iy - py;
        const bool rsub = wm != 0u && iy >= y1 && iy <= y2 && psf_y >= 0 && psf_y < a.pny;
        float *rp = (float *)band + (size_t)(iy - y_lo) * nx + c0;
        const float4 r4 = *(const float4 *)rp;
        float rr[4] = {r4.x, r4.y, r4.z, r4.w};
        if (rsub) {
          const float *pp = (const float *)a.psf + (size_t)psf_y * a.pnx + pxo0;
          float p4[4];
          if (wm == 0xfu && (((uintptr_t)pp) & 15) == 0) {
            const float4 q = __ldg((const float4 *)pp);
            p4[0] = q.x; p4[1] = q.y; p4[2] = q.z; p4[3] = q.w;
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) p4[j] = ((wm >> j) & 1u) ? __ldg(pp + j) : 0.f;
          }
          const float fpv = (float)pv;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if ((wm >> j) & 1u) rr[j] = __fsub_rn(rr[j], __fmul_rn(fpv, p4[j]));
          *(float4 *)rp = make_float4(rr[0], rr[1], rr[2], rr[3]);
        }
        if (bm != 0u && iy >= a.ybeg && iy < a.yend) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (!((bm >> j) & 1u)) continue;
            if (a.mask != nullptr && !(a.mask[(size_t)iy * nx + c0 + j] > (T)0.5)) continue;
            const float v = rr[j] < 0.f ? -rr[j] : rr[j];
            if ((T)v > best_abs) {
              best_abs = (T)v;
              best_idx = iy * nx + c0 + j;
              best_val = (T)rr[j];
            }
          }
        }
      }
    } else if (npr <= HOG_NPR) {
      // this thread's columns ix = threadIdx.x + k * HOG_THREADS: whether the
      // PSF window (with an existing PSF column) and the clean box cover them
      const int wlo = max(x1, px - a.pnx / 2), whi = min(x2, px + a.pnx / 2 - 1);
      bool colw[HOG_NPR], colb[HOG_NPR];
      int pxo[HOG_NPR];
#pragma unroll
      for (int k = 0; k < HOG_NPR; ++k) {
        const int ix = threadIdx.x + k * HOG_THREADS;
        const bool valid = k < npr && ix < nx;
        colw[k] = valid && do_sub && ix >= wlo && ix <= whi;
        colb[k] = valid && ix >= a.xbeg && ix < a.xend;
        pxo[k] = a.pnx / 2 + ix - px;
      }
      for (int iy0 = y_lo; iy0 < y_hi; iy0 += HOG_RB) {
        // the PSF values of HOG_RB rows through the read-only path, all
        // issued before the band is touched: one L2 round trip per batch
        T pk[HOG_RB][HOG_NPR];
#pragma unroll
        for (int q = 0; q < HOG_RB; ++q) {
          const int iy = iy0 + q;
          const int psf_y = a.pny / 2 + iy - py;
          const bool rsub = iy < y_hi && iy >= y1 && iy <= y2 && psf_y >= 0 && psf_y < a.pny;
          const T *prow = a.psf + (size_t)(rsub ? psf_y : 0) * a.pnx;
#pragma unroll
          for (int k = 0; k < HOG_NPR; ++k)
            pk[q][k] = (rsub && colw[k]) ? __ldg(prow + pxo[k]) : (T)0;
        }
#pragma unroll
        for (int q = 0; q < HOG_RB; ++q) {
          const int iy = iy0 + q;
          if (iy >= y_hi) break;  // the same for every thread of the block
          const int psf_y = a.pny / 2 + iy - py;
          const bool rsub = iy >= y1 && iy <= y2 && psf_y >= 0 && psf_y < a.pny;
          const bool rbox = iy >= a.ybeg && iy < a.yend;
          T *rrow = band + (size_t)(iy - y_lo) * nx;
#pragma unroll
          for (int k = 0; k < HOG_NPR; ++k) {
            const int ix = threadIdx.x + k * HOG_THREADS;
            if (k >= npr || ix >= nx) continue;
            T r = rrow[ix];
            if (rsub && colw[k]) {
              r = rn_sub(r, rn_mul(pv, pk[q][k]));
              rrow[ix] = r;
            }
            if (rbox && colb[k] &&
                (a.mask == nullptr || a.mask[(size_t)iy * nx + ix] > (T)0.5)) {
              const T v = r < (T)0 ? -r : r;
              if (v > best_abs) {
                best_abs = v;
                best_idx = iy * nx + ix;
                best_val = r;
              }
            }
          }
        }
      }
    } else
    for (int iy = y_lo; iy < y_hi; ++iy) {
      const bool row_sub = do_sub && iy >= y1 && iy <= y2;
      const bool row_box = iy >= a.ybeg && iy < a.yend;
      const int psf_y = a.pny / 2 + iy - py;
      const bool psf_row_ok = psf_y >= 0 && psf_y < a.pny;
      T *rrow = band + (size_t)(iy - y_lo) * nx;
      const T *prow = a.psf + (size_t)(psf_row_ok ? psf_y : 0) * a.pnx;
      for (int ix = threadIdx.x; ix < nx; ix += HOG_THREADS) {
        T r = rrow[ix];
        if (row_sub && psf_row_ok && ix >= x1 && ix <= x2) {
          int psf_x = a.pnx / 2 + ix - px;
          if (psf_x >= 0 && psf_x < a.pnx) {
            r = rn_sub(r, rn_mul(pv, prow[psf_x]));
            rrow[ix] = r;
          }
        }
        if (row_box && ix >= a.xbeg && ix < a.xend &&
            (a.mask == nullptr || a.mask[(size_t)iy * nx + ix] > (T)0.5)) {
          T v = r < (T)0 ? -r : r;
          if (v > best_abs) {
            best_abs = v;
            best_idx = iy * nx + ix;
            best_val = r;
          }
        }
      }
    }
    // block reduction (only strictly positive maxima count)
    if (best_idx >= 0 && !(best_abs > (T)0)) best_idx = -1;
    for (int o = 16; o > 0; o >>= 1) {
      T oa = __shfl_xor_sync(0xffffffffu, best_abs, o);
      int oi = __shfl_xor_sync(0xffffffffu, best_idx, o);
      T ov = __shfl_xor_sync(0xffffffffu, best_val, o);
      if (beats(oa, oi, best_abs, best_idx)) {
        best_abs = oa;
        best_idx = oi;
        best_val = ov;
      }
    }
    if (lane == 0) {
      s_abs[warp] = best_abs;
      s_idx[warp] = best_idx;
      s_val[warp] = best_val;
    }
    __syncthreads();
    if (warp == 0) {
      best_abs = s_abs[lane];
      best_idx = s_idx[lane];
      best_val = s_val[lane];
      for (int o = 16; o > 0; o >>= 1) {
        T oa = __shfl_xor_sync(0xffffffffu, best_abs, o);
        int oi = __shfl_xor_sync(0xffffffffu, best_idx, o);
        T ov = __shfl_xor_sync(0xffffffffu, best_val, o);
        if (beats(oa, oi, best_abs, best_idx)) {
          best_abs = oa;
          best_idx = oi;
          best_val = ov;
        }
      }
      if (lane == 0) {
        HogCand<T> c;
        c.absval = best_abs;
        c.val = best_val;
        c.idx = best_idx;
        // value at the current peak, published by its owner (used when no
        // pixel beats 0, where the reference keeps the previous position);
        // the block barrier above has ordered the band pass's writes
        const bool hp = py >= y_lo && py < y_hi;
        c.has_prev = hp ? 1 : 0;
        c.at_prev = hp ? band[(size_t)(py - y_lo) * nx + px] : (T)0;
        a.cand[par * G + b] = c;
        if (KEYED && best_idx >= 0) {
          const uint32_t code = 2u * (uint32_t)best_idx + (best_val < (T)0 ? 1u : 0u);
          const unsigned long long key =
              ((unsigned long long)__float_as_uint((float)best_abs) << 32) |
              (unsigned long long)(0xffffffffu - code);
          atomicMax(&a.state->key[par], key);
        }
      }
    }
    if (!grid_barrier(a.state, &s_flag, a.timeout_ns, KEYED ? &a.state->key[par ^ 1] : nullptr))
      break;
    // FP32: the winner from the 64-bit maximum (one load); otherwise, and
    // when no pixel was above 0, every CTA reduces all candidates the same way
    if (KEYED) {
      if (threadIdx.x == 0) {
        const unsigned long long kv = *(volatile unsigned long long *)&a.state->key[par];
        s_use_key = kv != 0ull;
        if (kv != 0ull) {
          const uint32_t code = 0xffffffffu - (uint32_t)kv;
          const float av = __uint_as_float((uint32_t)(kv >> 32));
          s_abs[0] = (T)av;
          s_idx[0] = (int)(code >> 1);
          s_val[0] = (code & 1u) ? (T)-av : (T)av;
        }
      }
      __syncthreads();
    }
    if (!(KEYED && s_use_key) && warp == 0) {
      T ga = (T)0, gv = (T)0, gprev = (T)0;
      int gi = -1, ghp = 0;
      for (int k0 = 0; k0 < G; k0 += 32 * HOG_CPL) {
        // L2 loads (other CTAs wrote these before the barrier), HOG_CPL
        // candidates per lane issued together, then reduced in index order
        HogCand<T> c[HOG_CPL];
#pragma unroll
        for (int q = 0; q < HOG_CPL; ++q) {
          const int k = k0 + lane + 32 * q;
          c[q].idx = -1;
          c[q].has_prev = 0;
          if (k < G) {
            const HogCand<T> *cp = a.cand + par * G + k;
            c[q].absval = __ldcg(&cp->absval);
            c[q].val = __ldcg(&cp->val);
            c[q].at_prev = __ldcg(&cp->at_prev);
            c[q].idx = __ldcg(&cp->idx);
            c[q].has_prev = __ldcg(&cp->has_prev);
          }
        }
#pragma unroll
        for (int q = 0; q < HOG_CPL; ++q) {
          if (beats(c[q].absval, c[q].idx, ga, gi)) {
            ga = c[q].absval;
            gi = c[q].idx;
            gv = c[q].val;
          }
          if (c[q].has_prev) {
            gprev = c[q].at_prev;
            ghp = 1;
          }
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        T oa = __shfl_xor_sync(0xffffffffu, ga, o);
        int oi = __shfl_xor_sync(0xffffffffu, gi, o);
        T ov = __shfl_xor_sync(0xffffffffu, gv, o);
        T op = __shfl_xor_sync(0xffffffffu, gprev, o);
        int oh = __shfl_xor_sync(0xffffffffu, ghp, o);
        if (beats(oa, oi, ga, gi)) {
          ga = oa;
          gi = oi;
          gv = ov;
        }
        if (oh) {
          gprev = op;
          ghp = 1;
        }
      }
      if (lane == 0) {
        s_abs[0] = ga;
        s_idx[0] = gi;
        s_val[0] = gv;
        s_prev = gprev;
      }
    }
    __syncthreads();
    if (s_idx[0] >= 0) {
      px = s_idx[0] % nx;
      py = s_idx[0] / nx;
      peak = s_val[0];
      absval = s_abs[0];
    } else {
      peak = s_prev;
      absval = (T)0;
    }
    __syncthreads();
    par ^= 1;
    if (first) first = false;
    else ++it;
  }
  // write the band back and publish the state
  __syncthreads();
  if (a.resident) {
    for (int i0 = 0; i0 < (y_hi - y_lo) * nx; i0 += HOG_THREADS) {
      const int i = i0 + threadIdx.x;
      if (i < (y_hi - y_lo) * nx) a.resid[(size_t)y_lo * nx + i] = band[i];
    }
  }
  if (b == 0 && threadIdx.x == 0) {
    a.state->kpar = par;
    a.state->iter = it;
    a.state->px = px;
    a.state->py = py;
    a.state->peak = (double)peak;
    a.state->absval = (double)absval;
    a.state->stopped = stopped ? 1 : 0;
  }
}

// ------------------------------------------------- residual in registers ----
// The FP32 loop for images up to 2048 columns whose bands fit the register
// file (k_hogbom above keeps FP64 and larger ones): the same arithmetic, the
// same winners.
//   - A thread owns RJ rows x NC columns of its CTA's band in registers, and a
//     pixel costs a load, a multiply, a subtraction and a maximum.  The
//     maximum's place is looked for afterwards, by the warps that hold it only.
//     Up to 14 pixels a thread nothing spills; at 28 up to 56 bytes do, and at
//     56, which 2048^2 takes, 388 bytes of spill loads (bulk copies; 604
//     without) of the mask and addresses come from L1 in an iteration.
//   - The PSF rows an iteration needs come to shared memory by bulk copies
//     (one per row, an mbarrier per four steps), 115 KB in flight per SM;
//     4-byte loads through L1 brought 11 bytes a clock (loads cannot be
//     wider: the PSF's columns are shifted by the peak's).  A PSF whose rows
//     are not 16-byte aligned is read by such loads all the same.
//   - Each CTA stores its winner, tagged with the iteration, in every CTA's
//     inbox, and polls its own: one store and one load through L2 in place of
//     an atomic maximum, an arrival count, its release and a read of the
//     winner, and no line that all SMs poll.  Two sets of inboxes are used in
//     turn: a CTA can be at most one exchange ahead of the slowest.
//   - An exchange gives up timeout_ns after its 257th failed poll, looked at in
//     every 256th (at the first with a bound of 0), sets the error flag and
//     leaves; the others then run into their own bound.  A bulk copy has
//     HOG_COPY_NS, whatever timeout_ns is.
// An iteration on 2048^2 takes 6.3 us (k_hogbom 10.2), of which the band pass
// 2.4-3.2 (the PSF from L2 alone: 1.3), the exchange 1.8 and the skew between
// the CTAs' windows the rest; on 512^2 3.4 us, 256^2 3.1 us, mostly exchange.
struct __align__(16) HogSlot {
  unsigned long long best;  // |r| bits << 32 | tag
  unsigned long long code;  // (2 * index + sign) << 32 | tag
};
constexpr int HOG_SLOTS_PER_LANE = 5;  // up to 160 CTAs
constexpr int HOG_MAX_CTAS = 32 * HOG_SLOTS_PER_LANE;

// Two sets, each with an inbox of G slots per CTA and one word per CTA for the
// residual at the current peak (value bits << 32 | tag, sent on demand).
struct HogExchange {
  HogSlot slot[2][HOG_MAX_CTAS][HOG_MAX_CTAS];  // [set][reader][writer]
  unsigned long long prev[2][HOG_MAX_CTAS];
};

__device__ __forceinline__ void slot_store(HogSlot *s, unsigned long long a,
                                           unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(s), "l"(a), "l"(b)
               : "memory");
}
__device__ __forceinline__ void slot_load(const HogSlot *s, unsigned long long &a,
                                          unsigned long long &b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(s)
               : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// a bulk copy that has not arrived after this long never will
constexpr unsigned long long HOG_COPY_NS = 2000000000ull;
constexpr int HOG_RT = 512;  // threads: 56 pixels each at 2048^2, of 128 registers
constexpr unsigned HOG_POLLS = 256;

__device__ __forceinline__ unsigned smem_addr(const void *p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(unsigned long long *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool bar_test(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0u;
}
// dst and src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes,
                                          unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// Floats a staged PSF row takes (its first column is rounded down to 4).
__host__ __device__ constexpr int hog_row(int nx) { return (nx + 11) & ~3; }

// Waits for a barrier's phase; false when it has not completed after
// HOG_COPY_NS (the timer is read once in HOG_POLLS tries: a read takes as long
// as many of them).
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, unsigned parity) {
  unsigned long long t0 = 0ull;
  for (unsigned n = 1; !bar_test(bar, parity); ++n) {
    if (n % HOG_POLLS) continue;
    const unsigned long long t1 = global_ns();
    if (t0 == 0ull) t0 = t1;
    if (t1 - t0 >= HOG_COPY_NS) return false;
  }
  return true;
}

// BULK: the PSF's rows are 16-byte aligned.
template <int NC, int RJ, bool BULK>
__global__ void __launch_bounds__(HOG_RT, 1) k_hogbom_reg(HogArgs<float> a, int tpr) {
  extern __shared__ __align__(128) float s_psf[];  // BULK: [row][hog_row(nx)]
  constexpr int GR = 4, NG = (RJ + GR - 1) / GR;  // steps that share an mbarrier
  constexpr int RB = RJ < 7 ? RJ : 7;             // rows whose PSF values are loaded together
  __shared__ unsigned long long s_bar[NG];
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ unsigned s_max[32];
  __shared__ unsigned s_code, s_abs;
  __shared__ int s_px, s_py, s_ok;
  __shared__ float s_peak, s_prev;
  HogExchange *ex = (HogExchange *)a.cand;  // zero at the launch
  const int G = gridDim.x, b = blockIdx.x, nx = a.nx;
  const int y_lo = (int)((long long)a.ny * b / G), y_hi = (int)((long long)a.ny * (b + 1) / G);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // tpr threads (a multiple of 32) to a row, rg rows at a time
  const int rg = HOG_RT / tpr, tx = threadIdx.x % tpr, gy = threadIdx.x / tpr;
  const int rows = gy < rg ? y_hi - y_lo : 0;  // this thread's rows: gy + rg * j < rows
  float r[RJ][NC];
  // pixels that the clean box and the mask admit; places past the band hold 0,
  // which never wins
  unsigned long long use = 0ull;
  constexpr unsigned long long EVERY = (1ull << (RJ * NC)) - 1ull;
#pragma unroll
  for (int j = 0; j < RJ; ++j)
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      const int y = gy + rg * j, c = tx + m * tpr;
      r[j][m] = 0.f;
      if (y >= rows || c >= nx) {
        use |= 1ull << (j * NC + m);
      } else {
        const size_t i = (size_t)(y_lo + y) * nx + c;
        r[j][m] = a.resid[i];
        if (y_lo + y >= a.ybeg && y_lo + y < a.yend && c >= a.xbeg && c < a.xend &&
            (a.mask == nullptr || a.mask[i] > 0.5f))
          use |= 1ull << (j * NC + m);
      }
    }
  const bool all = __all_sync(FULL, use == EVERY);
  int px = 0, py = 0, it = a.iter_begin;
  float peak = 0.f, absval = 0.f;
  if (!a.init) {
    px = a.state->px;
    py = a.state->py;
    peak = (float)a.state->peak;
    absval = (float)a.state->absval;
  }
  if (threadIdx.x == 0) {
    s_code = FULL;
    s_ok = 1;
  }
  if (threadIdx.x < 32) s_max[threadIdx.x] = 0u;  // HOG_RT / 32 of them are used
  if (BULK && threadIdx.x == 0) {
    for (int g = 0; g < NG; ++g) bar_init(&s_bar[g]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  unsigned round = 0u;  // parity of the barriers
  const int ld = hog_row(nx);
  const int lane_group = lane / (rg * GR);  // the barrier of row `lane`
  float mv = 0.f;
  __syncthreads();
  bool first = a.init != 0, stopped = false;
  const int hx = a.pnx / 2, hy = a.pny / 2;
  for (unsigned tag = 1;; ++tag) {
    float pv = 0.f;
    bool do_sub = false;
    if (!first) {
      if (it >= a.iter_end) break;
      float cthres = a.thres;
      if (a.speedup > 0.f) cthres = a.thres * t_pow(2.f, (float)(it - a.siter) / a.speedup);
      if (absval < cthres) {
        stopped = true;
        break;
      }
      pv = rn_mul(a.gain, peak);
      do_sub = true;
      // read here, written after the exchange: its latency is not waited for
      if (b == 0 && threadIdx.x == HOG_RT - 1) mv = a.model[(size_t)py * nx + px];
    }
    // PSF window (hclean.cpp:172-175 with the PSF's own half sizes), as
    // ranges of columns and rows that a PSF value exists for
    const int x1 = max(max(0, px - hx), px - hx), y1 = max(0, py - hy);
    const int x2 = min(min(nx - 1, px + hx - 1), px - hx + a.pnx - 1);
    const int y2 = min(min(a.ny - 1, py + hy - 1), py - hy + a.pny - 1);
    bool colw[NC];
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      const int c = tx + m * tpr;
      colw[m] = do_sub && c < nx && c >= x1 && c <= x2;
    }
    if constexpr (BULK) {
      if (do_sub) {
        // rows [f0, f1) of the band and columns s0 .. of the PSF are staged
        const bool any = x1 <= x2;
        const int f0 = max(0, y1 - y_lo), f1 = any ? min(y_hi, y2 + 1) - y_lo : 0;
        const int s0 = (hx - px + x1) & ~3, s1 = min(a.pnx, (hx - px + x2 + 4) & ~3);
        if (warp == 0) {
          const unsigned bytes = (unsigned)(s1 - s0) * 4u;
          if (lane < NG) {
            const int n = min(f1, rg * GR * (lane + 1)) - max(f0, rg * GR * lane);
            bar_expect(&s_bar[lane], n > 0 ? bytes * (unsigned)n : 0u);
          }
          __syncwarp();
          for (int y = lane; y < f1; y += 32)
            if (y >= f0)
              bulk_copy(s_psf + y * ld, a.psf + (int64_t)(hy + y_lo + y - py) * a.pnx + s0, bytes,
                        &s_bar[y == lane ? lane_group : y / (rg * GR)]);
        }
        // staged column of each pixel (any staged one where there is none: the
        // value is not used, and the loads need no branches)
        const float *row = s_psf + gy * ld;
        int col[NC];
#pragma unroll
        for (int m = 0; m < NC; ++m) col[m] = colw[m] ? hx + tx + m * tpr - px - s0 : 0;
        const int f1r = min(f1, rows);
        int y = gy;  // this thread's row at each step
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          if (!bar_wait(&s_bar[g], round)) s_ok = 0;
#pragma unroll
          for (int q = 0; q < GR; ++q) {
            const int j = g * GR + q;
            if (j >= RJ) continue;
            if (y >= f0 && y < f1r) {  // the same for the warp
#pragma unroll
              for (int m = 0; m < NC; ++m) {
                const float d = __fsub_rn(r[j][m], __fmul_rn(pv, row[col[m]]));
                r[j][m] = colw[m] ? d : r[j][m];
              }
            }
            row += rg * ld;
            y += rg;
          }
        }
        round ^= 1u;
      }
    } else {
      const float *pp = a.psf + ((int64_t)(hy + y_lo + gy - py) * a.pnx + (hx + tx - px));
      const int64_t step = (int64_t)rg * a.pnx;
#pragma unroll
      for (int j0 = 0; j0 < RJ; j0 += RB) {
        float pk[RB][NC];
        bool roww[RB];
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          const int j = j0 + q, y = gy + rg * j;
          roww[q] = j < RJ && y < rows && y_lo + y >= y1 && y_lo + y <= y2;
#pragma unroll
          for (int m = 0; m < NC; ++m)
            if (roww[q] && colw[m]) pk[q][m] = __ldg(pp + j * step + m * tpr);
        }
#pragma unroll
        for (int q = 0; q < RB; ++q) {
          if (j0 + q >= RJ) continue;
          const int j = j0 + q < RJ ? j0 + q : 0;
#pragma unroll
          for (int m = 0; m < NC; ++m)
            if (roww[q] && colw[m]) r[j][m] = __fsub_rn(r[j][m], __fmul_rn(pv, pk[q][m]));
        }
      }
    }
    // NaN never wins, as with the reference's '>'
    float lmax = 0.f;
    if (all) {
#pragma unroll
      for (int j = 0; j < RJ; ++j)
#pragma unroll
        for (int m = 0; m < NC; ++m) lmax = fmaxf(lmax, fabsf(r[j][m]));
    } else {
#pragma unroll
      for (int j = 0; j < RJ; ++j)
#pragma unroll
        for (int m = 0; m < NC; ++m)
          if ((use >> (j * NC + m)) & 1ull) lmax = fmaxf(lmax, fabsf(r[j][m]));
    }
    const unsigned lb = __float_as_uint(lmax), wb = __reduce_max_sync(FULL, lb);
    if (lane == 0) s_max[warp] = wb;
    __syncthreads();
    const unsigned bm = __reduce_max_sync(FULL, s_max[lane]);
    if (bm != 0u && wb == bm) {
      // the first pixel in row-major order, and its sign
      unsigned code = FULL;
      if (lb == bm) {
        int k = 0;
        bool neg = false;
#pragma unroll
        for (int j = RJ - 1; j >= 0; --j)
#pragma unroll
          for (int m = NC - 1; m >= 0; --m)
            if (((use >> (j * NC + m)) & 1ull) && __float_as_uint(fabsf(r[j][m])) == bm) {
              k = j * NC + m;
              neg = r[j][m] < 0.f;
            }
        code = 2u * (unsigned)((y_lo + gy + rg * (k / NC)) * nx + tx + (k % NC) * tpr) +
               (neg ? 1u : 0u);
      }
      code = __reduce_min_sync(FULL, code);
      if (lane == 0) atomicMin(&s_code, code);
    }
    __syncthreads();
    const unsigned set = tag & 1u;
    if (warp == 0) {
      const unsigned own = s_code;
      __syncwarp();
      if (lane == 0) s_code = FULL;
      unsigned ga = 0u, gc = FULL, missing = 0u;
#pragma unroll
      for (int q = 0; q < HOG_SLOTS_PER_LANE; ++q)
        if (lane + 32 * q < G) {
          missing |= 1u << q;
          slot_store(&ex->slot[set][lane + 32 * q][b], ((unsigned long long)bm << 32) | tag,
                     ((unsigned long long)own << 32) | tag);
        }
      unsigned long long t0 = 0ull;
      unsigned polls = 0u;
      int ok = s_ok;
      while (ok) {
        // every missing slot's load in flight at once
        unsigned long long x[HOG_SLOTS_PER_LANE], y[HOG_SLOTS_PER_LANE];
#pragma unroll
        for (int q = 0; q < HOG_SLOTS_PER_LANE; ++q) {
          x[q] = y[q] = 0ull;
          if ((missing >> q) & 1u) slot_load(&ex->slot[set][b][lane + 32 * q], x[q], y[q]);
        }
#pragma unroll
        for (int q = 0; q < HOG_SLOTS_PER_LANE; ++q) {
          if ((unsigned)x[q] != tag || (unsigned)y[q] != tag) continue;
          missing &= ~(1u << q);
          const unsigned xa = (unsigned)(x[q] >> 32), xc = (unsigned)(y[q] >> 32);
          if (xa > ga || (xa == ga && xc < gc)) {
            ga = xa;
            gc = xc;
          }
        }
        if (!__any_sync(FULL, missing != 0u)) break;
        // the timer is read once in HOG_POLLS failed polls: a read takes as
        // long as a poll
        if (polls++ % HOG_POLLS == 0u && (polls > 1u || a.timeout_ns == 0ull)) {
          const unsigned long long t1 = __shfl_sync(FULL, global_ns(), 0);
          if (t0 == 0ull) t0 = t1;
          if (t1 - t0 >= a.timeout_ns) {
            ok = 0;
            break;
          }
        }
      }
      const unsigned gm = __reduce_max_sync(FULL, ga);
      const unsigned code = __reduce_min_sync(FULL, ga == gm ? gc : FULL);
      if (lane == 0) {
        if (!ok) atomicExch(&a.state->err, 1);
        s_ok = ok;
        s_abs = gm;
        if (gm != 0u) {
          const int idx = (int)(code >> 1);
          s_px = idx % nx;
          s_py = idx / nx;
          s_peak = (code & 1u) ? -__uint_as_float(gm) : __uint_as_float(gm);
        }
      }
    }
    __syncthreads();
    if (do_sub && b == 0 && threadIdx.x == HOG_RT - 1)
      a.model[(size_t)py * nx + px] = rn_add(mv, pv);
    if (!s_ok) break;
    if (s_abs != 0u) {
      px = s_px;
      py = s_py;
      peak = s_peak;
      absval = __uint_as_float(s_abs);
    } else {
      // no pixel above 0: the position stays, and its owner passes the value on
      const int oy = py - y_lo - gy, ox = px - tx;
      if (gy < rg && oy >= 0 && oy + gy < rows && oy % rg == 0 && ox >= 0 && ox % tpr == 0 &&
          ox / tpr < NC) {
        const int k = oy / rg * NC + ox / tpr;
#pragma unroll
        for (int i = 0; i < RJ * NC; ++i)
          if (i == k) s_prev = r[i / NC][i % NC];
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        volatile unsigned long long *mine = &ex->prev[set][b];
        if (py >= y_lo && py < y_hi)
          *mine = ((unsigned long long)__float_as_uint(s_prev) << 32) | tag;
        int own = (int)(((long long)py * G) / a.ny);  // the band that holds row py
        while ((long long)a.ny * (own + 1) / G <= py) ++own;
        while ((long long)a.ny * own / G > py) --own;
        volatile const unsigned long long *theirs = &ex->prev[set][own];
        unsigned long long x = *theirs, t0 = 0ull;
        while ((unsigned)x != tag) {
          const unsigned long long t1 = global_ns();
          if (t0 == 0ull) t0 = t1;
          if (t1 - t0 >= a.timeout_ns) {
            atomicExch(&a.state->err, 1);
            s_ok = 0;
            break;
          }
          x = *theirs;
        }
        s_peak = __uint_as_float((unsigned)(x >> 32));
      }
      __syncthreads();
      if (!s_ok) break;
      peak = s_peak;
      absval = 0.f;
      __syncthreads();
    }
    if (first) first = false;
    else ++it;
  }
#pragma unroll
  for (int j = 0; j < RJ; ++j)
#pragma unroll
    for (int m = 0; m < NC; ++m) {
      const int y = gy + rg * j, c = tx + m * tpr;
      if (y < rows && c < nx) a.resid[(size_t)(y_lo + y) * nx + c] = r[j][m];
    }
  if (b == 0 && threadIdx.x == 0) {
    a.state->iter = it;
    a.state->px = px;
    a.state->py = py;
    a.state->peak = (double)peak;
    a.state->absval = (double)absval;
    a.state->stopped = stopped ? 1 : 0;
  }
}

template <int NC, int RJ>
static int launch_hogbom_reg(HogArgs<float> a, int tpr, int grid, cudaStream_t st) {
  AV_CUDA(cudaMemsetAsync(a.cand, 0, sizeof(HogExchange), st));
  void *args[] = {&a, &tpr};
  const bool bulk = a.pnx % 4 == 0 && ((uintptr_t)a.psf & 15) == 0;
  const size_t smem =
      bulk ? (size_t)((a.ny + grid - 1) / grid) * hog_row(a.nx) * sizeof(float) : 0;
  const void *kernel = bulk ? (const void *)k_hogbom_reg<NC, RJ, true>
                            : (const void *)k_hogbom_reg<NC, RJ, false>;
  AV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  AV_CUDA(cudaLaunchCooperativeKernel(kernel, grid, HOG_RT, args, smem, st));
  count_launch();
  return AV_OK;
}

// k_hogbom_reg's smallest variant that holds the bands in registers; false
// when none does (more than 2048 columns, 56 pixels a thread or 160 CTAs) or
// k_hogbom is the faster: on tall narrow images whose width lets it take four
// pixels per thread with no thread idle (a power of two).  There a row is too
// short for a bulk copy to pay, and the variants of more than 14 rows per
// thread spill.  200 iterations against k_hogbom: 256 columns, 15-50 rows per
// thread 1.00-1.06 (14: 0.65); 128 columns, 16-56 rows 1.13-1.35 (14: 0.76);
// 64 columns, 15-56 rows 1.38-1.89 (14: 0.92); 512 columns, 15 and 16 rows
// 1.05, 20-56 rows 0.98-0.91; up to 32 columns, bands of 80 rows 0.97-1.02,
// of 90 1.00-1.08, of 300 1.9-2.8.  Other widths take k_hogbom_reg to the end
// (100 columns 0.48-0.23, 300 0.70-0.45, 450 0.89-0.44, 600-1024 0.65-0.41).
static bool hogbom_reg(const HogArgs<float> &a, int grid, cudaStream_t st, int &rc) {
  if (a.nx > 4 * HOG_RT || grid > HOG_MAX_CTAS) return false;
  const int nc = a.nx <= HOG_RT ? 1 : (a.nx <= 2 * HOG_RT ? 2 : 4);
  const int tpr = ((a.nx + nc - 1) / nc + 31) / 32 * 32;
  const int rg = HOG_RT / tpr, band = (a.ny + grid - 1) / grid;
  const int rj = (band + rg - 1) / rg;
  if (rj * nc > 56) return false;
  const bool four_wide = a.nx >= 4 && a.nx <= 512 && (a.nx & (a.nx - 1)) == 0;
  if (four_wide && ((rj > 14 && (a.nx < 512 || rj < 20)) || (a.nx <= 32 && band > 80)))
    return false;
  if (nc == 1) {
    if (rj <= 1) rc = launch_hogbom_reg<1, 1>(a, tpr, grid, st);
    else if (rj <= 2) rc = launch_hogbom_reg<1, 2>(a, tpr, grid, st);
    else if (rj <= 4) rc = launch_hogbom_reg<1, 4>(a, tpr, grid, st);
    else if (rj <= 14) rc = launch_hogbom_reg<1, 14>(a, tpr, grid, st);
    else rc = launch_hogbom_reg<1, 56>(a, tpr, grid, st);
  } else if (nc == 2) {
    if (rj <= 4) rc = launch_hogbom_reg<2, 4>(a, tpr, grid, st);
    else if (rj <= 7) rc = launch_hogbom_reg<2, 7>(a, tpr, grid, st);
    else if (rj <= 14) rc = launch_hogbom_reg<2, 14>(a, tpr, grid, st);
    else rc = launch_hogbom_reg<2, 28>(a, tpr, grid, st);
  } else {
    if (rj <= 7) rc = launch_hogbom_reg<4, 7>(a, tpr, grid, st);
    else rc = launch_hogbom_reg<4, 14>(a, tpr, grid, st);
  }
  return true;
}

// ------------------------------------------------------------------ maximg --
// Minimum and maximum straight into out: a float's order is its bits' signed
// order from 0 up and their reversed unsigned order below (-0 below 0), so the
// blocks' results meet in integer atomics and no scratch is needed.  (One CTA took
// 389 us for 2048^2; 296 take 5.6.)
template <typename T>
struct OrderBits;
template <>
struct OrderBits<float> {
  using S = int;
  using U = unsigned;
};
template <>
struct OrderBits<double> {
  using S = long long;
  using U = unsigned long long;
};

template <typename T>
__device__ __forceinline__ void atomic_extreme(T *p, T v, bool want_max) {
  using S = typename OrderBits<T>::S;
  using U = typename OrderBits<T>::U;
  S s;
  memcpy(&s, &v, sizeof(T));
  if (want_max ? s >= 0 : s < 0) {
    // max of a non-negative value, min of a negative one: larger bits win
    if (want_max) atomicMax((S *)p, s);
    else atomicMax((U *)p, (U)s);
  } else {
    if (want_max) atomicMin((U *)p, (U)s);
    else atomicMin((S *)p, s);
  }
}

template <typename T>
__global__ void k_maximg_init(T *out) {
  if (threadIdx.x == 0) {
    out[0] = (T)1e20;
    out[1] = (T)-1e20;
  }
}

constexpr int MAXIMG_THREADS = 512;

template <typename T>
__global__ void __launch_bounds__(MAXIMG_THREADS) k_maximg(const T *img, const T *mask,
                                                           int64_t n, T *out) {
  T mn = (T)1e20, mx = (T)-1e20;
  const int64_t stride = (int64_t)gridDim.x * MAXIMG_THREADS;
#pragma unroll 4
  for (int64_t i = blockIdx.x * (int64_t)MAXIMG_THREADS + threadIdx.x; i < n; i += stride) {
    if (mask == nullptr || mask[i] > (T)0.5) {
      T w = img[i];
      if (w > mx) mx = w;
      if (w < mn) mn = w;
    }
  }
  __shared__ T smn[MAXIMG_THREADS / 32], smx[MAXIMG_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) {
    T a = __shfl_xor_sync(0xffffffffu, mn, o), c = __shfl_xor_sync(0xffffffffu, mx, o);
    if (a < mn) mn = a;
    if (c > mx) mx = c;
  }
  if ((threadIdx.x & 31) == 0) {
    smn[threadIdx.x >> 5] = mn;
    smx[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < MAXIMG_THREADS / 32; ++w) {
      if (smn[w] < mn) mn = smn[w];
      if (smx[w] > mx) mx = smx[w];
    }
    if (mn < (T)1e20) atomic_extreme(out, mn, false);
    if (mx > (T)-1e20) atomic_extreme(out + 1, mx, true);
  }
}

// --------------------------------------------------- ordered |x| summation --
// Sum of |x| in index order with sequential addition: zeros do not change a
// running sum, so the non-zeros are compacted in order and summed by one
// thread.
constexpr int ABS_THREADS = 1024;
constexpr int64_t ABS_PER_BLOCK = 16384;  // elements a block takes (more above 1024 blocks)

__device__ __forceinline__ void abs_range(int64_t n, int64_t &lo, int64_t &hi) {
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  lo = min(n, blockIdx.x * per);
  hi = min(n, lo + per);
}

// Non-zeros of each block's range.
template <typename T>
__global__ void __launch_bounds__(ABS_THREADS) k_nz_count(const T *x, int64_t n,
                                                          uint32_t *counts) {
  int64_t lo, hi;
  abs_range(n, lo, hi);
  uint32_t c = 0;
#pragma unroll 4
  for (int64_t i = lo + threadIdx.x; i < hi; i += ABS_THREADS) c += x[i] != (T)0;
  __shared__ uint32_t sh[32];
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x < 32) {
    c = __reduce_add_sync(0xffffffffu, sh[threadIdx.x]);
    if (threadIdx.x == 0) counts[blockIdx.x] = c;
  }
}

// Their magnitudes in index order: 1024 consecutive elements at a time,
// placed by ballots.  (A thread per contiguous stretch and a serial scan of
// the threads' counts had taken 75 us for 2048^2; 7.7 now.)
template <typename T>
__global__ void __launch_bounds__(ABS_THREADS) k_nz_write(const T *x, int64_t n,
                                                          const uint32_t *counts, T *out) {
  __shared__ uint32_t sh[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (counts[blockIdx.x] == 0u) return;
  uint32_t c = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += ABS_THREADS) c += counts[k];
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0) sh[warp] = c;
  __syncthreads();
  uint32_t pos = __reduce_add_sync(0xffffffffu, sh[lane]);  // of the block's first
  int64_t lo, hi;
  abs_range(n, lo, hi);
  for (int64_t i0 = lo; i0 < hi; i0 += ABS_THREADS) {
    const int64_t i = i0 + threadIdx.x;
    const T v = i < hi ? x[i] : (T)0;
    const bool nz = v != (T)0;
    const unsigned m = __ballot_sync(0xffffffffu, nz);
    if (!__syncthreads_or(nz)) continue;  // also: sh of the round before is read
    if (lane == 0) sh[warp] = __popc(m);
    __syncthreads();
    const uint32_t w = sh[lane];
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
    const uint32_t total = __reduce_add_sync(0xffffffffu, w);
    if (nz) out[pos + before + __popc(m & ((1u << lane) - 1u))] = v < (T)0 ? -v : v;
    pos += total;
  }
}

template <typename T>
__global__ void k_seq_sum(const T *v, const uint32_t *counts, int nblocks, T *out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  uint32_t n = 0;
  for (int k = 0; k < nblocks; ++k) n += counts[k];
  T s = (T)0;
  for (uint32_t i = 0; i < n; ++i) s = rn_add(s, v[i]);
  out[0] = s;
}

template <typename T>
static int hogbom_launch(HogArgs<T> a, int grid, size_t smem, cudaStream_t st) {
  void *args[] = {&a};
  AV_CUDA(cudaLaunchCooperativeKernel((const void *)k_hogbom<T>, grid, HOG_THREADS, args, smem,
                                      st));
  count_launch();
  return AV_OK;
}

}  // namespace av

using namespace av;

extern "C" {

size_t av_hogbom_state_size(void) { return sizeof(HogState); }

// What k_hogbom needs; k_hogbom_reg is used where there is room for its
// exchange.
static size_t hogbom_least(int dtype) {
  size_t cs = dtype == AV_F64 ? sizeof(HogCand<double>) : sizeof(HogCand<float>);
  return Workspace::need(cs * 2 * 1024);
}

size_t av_hogbom_workspace_size(int64_t nx, int64_t ny, int dtype) {
  (void)nx;
  (void)ny;
  return std::max(hogbom_least(dtype), Workspace::need(sizeof(HogExchange)));
}

int av_hogbom_run(void *model, void *residual, const void *psf, const void *mask, int dtype,
                  int64_t nx, int64_t ny, int64_t pnx, int64_t pny, int xbeg, int xend,
                  int ybeg, int yend, int niter, int siter, int iter_begin, int iter_end,
                  double gain, double threshold, double speedup, void *state, int init_state,
                  void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  AV_CHECK_ARG(model && residual && psf && state && workspace, "av_hogbom_run: null pointer");
  AV_CHECK_ARG(dtype == AV_F32 || dtype == AV_F64, "av_hogbom_run: dtype");
  AV_CHECK_ARG(nx > 0 && ny > 0 && pnx > 0 && pny > 0 && nx * ny < (1LL << 31),
               "av_hogbom_run: bad shape");
  AV_CHECK_ARG(xbeg >= 0 && xend <= nx && xbeg < xend && ybeg >= 0 && yend <= ny && ybeg < yend,
               "av_hogbom_run: bad clean box");
  AV_CHECK_ARG(workspace_bytes >= hogbom_least(dtype),
               "av_hogbom_run: workspace too small");
  cudaStream_t st = as_stream(stream);
  int dev = 0;
  AV_CUDA(cudaGetDevice(&dev));
  const unsigned long long timeout_ns =
      (unsigned long long)tune_value(AV_TUNE_HOGBOM_BARRIER_TIMEOUT_US) * 1000ull;
  int sms = sm_count();
  int grid = (int)std::min<int64_t>(sms, ny);
  if (grid > 1024) grid = 1024;
  size_t esz = dtype == AV_F64 ? 8 : 4;
  int64_t band_rows = (ny + grid - 1) / grid;
  size_t band_bytes = (size_t)band_rows * nx * esz;
  int max_smem = 0;
  AV_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  int resident = band_bytes + 4096 <= (size_t)max_smem;
  size_t smem = resident ? band_bytes : 0;
  if (init_state) AV_CUDA(cudaMemsetAsync(state, 0, sizeof(HogState), st));
  if (dtype == AV_F32) {
    HogArgs<float> a;
    a.model = (float *)model; a.resid = (float *)residual; a.psf = (const float *)psf;
    a.mask = (const float *)mask;
    a.nx = (int)nx; a.ny = (int)ny; a.pnx = (int)pnx; a.pny = (int)pny;
    a.xbeg = xbeg; a.xend = xend; a.ybeg = ybeg; a.yend = yend;
    a.niter = niter; a.siter = siter; a.iter_begin = iter_begin; a.iter_end = iter_end;
    a.gain = (float)gain; a.thres = (float)threshold; a.speedup = (float)speedup;
    a.state = (HogState *)state; a.cand = (HogCand<float> *)workspace;
    a.init = init_state; a.resident = resident; a.timeout_ns = timeout_ns;
    int rc = AV_OK;
    if (workspace_bytes >= sizeof(HogExchange) && hogbom_reg(a, grid, st, rc)) return rc;
    AV_CUDA(cudaFuncSetAttribute(k_hogbom<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    int per_sm = 0;
    AV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_hogbom<float>, HOG_THREADS,
                                                          smem));
    if (per_sm < 1) {
      set_error("av_hogbom_run: kernel cannot be resident (smem %zu)", smem);
      return AV_ERR_UNSUPPORTED;
    }
    return hogbom_launch<float>(a, grid, smem, st);
  }
  AV_CUDA(cudaFuncSetAttribute(k_hogbom<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
  int per_sm = 0;
  AV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_hogbom<double>, HOG_THREADS,
                                                        smem));
  if (per_sm < 1) {
    set_error("av_hogbom_run: kernel cannot be resident (smem %zu)", smem);
    return AV_ERR_UNSUPPORTED;
  }
  HogArgs<double> a;
  a.model = (double *)model; a.resid = (double *)residual; a.psf = (const double *)psf;
  a.mask = (const double *)mask;
  a.nx = (int)nx; a.ny = (int)ny; a.pnx = (int)pnx; a.pny = (int)pny;
  a.xbeg = xbeg; a.xend = xend; a.ybeg = ybeg; a.yend = yend;
  a.niter = niter; a.siter = siter; a.iter_begin = iter_begin; a.iter_end = iter_end;
  a.gain = gain; a.thres = threshold; a.speedup = speedup;
  a.state = (HogState *)state; a.cand = (HogCand<double> *)workspace;
  a.init = init_state; a.resident = resident; a.timeout_ns = timeout_ns;
  return hogbom_launch<double>(a, grid, smem, st);
}

int av_hogbom_state_read(const void *state, int32_t *out_i, double *out_d, void *stream) {
  clear_error();
  AV_CHECK_ARG(state && out_i && out_d, "av_hogbom_state_read: null pointer");
  HogState h;
  cudaStream_t st = as_stream(stream);
  AV_CUDA(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
  AV_CUDA(cudaStreamSynchronize(st));
  out_i[0] = h.iter;
  out_i[1] = h.px;
  out_i[2] = h.py;
  out_i[3] = h.stopped;
  out_i[4] = h.err;
  out_d[0] = h.peak;
  out_d[1] = h.absval;
  if (h.err) {
    set_error("av_hogbom_run: grid barrier timed out");
    return AV_ERR_TIMEOUT;
  }
  return AV_OK;
}

int av_maximg(const void *image, const void *mask, int dtype, int64_t nx, int64_t ny, void *out,
              void *stream) {
  clear_error();
  AV_CHECK_ARG(image && out, "av_maximg: null pointer");
  AV_CHECK_ARG(dtype == AV_F32 || dtype == AV_F64, "av_maximg: dtype");
  AV_CHECK_ARG(nx >= 0 && ny >= 0, "av_maximg: bad shape");
  cudaStream_t st = as_stream(stream);
  int64_t n = nx * ny;
  const unsigned blocks = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>((int64_t)sm_count() * 2, (n + MAXIMG_THREADS - 1) / MAXIMG_THREADS));
  if (dtype == AV_F32) {
    k_maximg_init<float><<<1, 32, 0, st>>>((float *)out);
    AV_LAUNCH_CHECK();
    k_maximg<float><<<blocks, MAXIMG_THREADS, 0, st>>>((const float *)image, (const float *)mask,
                                                       n, (float *)out);
  } else {
    k_maximg_init<double><<<1, 32, 0, st>>>((double *)out);
    AV_LAUNCH_CHECK();
    k_maximg<double><<<blocks, MAXIMG_THREADS, 0, st>>>((const double *)image,
                                                        (const double *)mask, n, (double *)out);
  }
  AV_LAUNCH_CHECK();
  return AV_OK;
}

size_t av_abs_sum_workspace_size(int64_t n, int dtype) {
  size_t esz = dtype == AV_F64 ? 8 : 4;
  return Workspace::need(sizeof(uint32_t) * 1024) + Workspace::need(esz * (size_t)(n > 0 ? n : 1));
}

int av_abs_sum_ordered(const void *model, int dtype, int64_t n, void *out, void *workspace,
                       size_t workspace_bytes, void *stream) {
  clear_error();
  AV_CHECK_ARG(model && out && workspace, "av_abs_sum_ordered: null pointer");
  AV_CHECK_ARG(dtype == AV_F32 || dtype == AV_F64, "av_abs_sum_ordered: dtype");
  AV_CHECK_ARG(workspace_bytes >= av_abs_sum_workspace_size(n, dtype),
               "av_abs_sum_ordered: workspace too small");
  cudaStream_t st = as_stream(stream);
  Workspace ws(workspace, workspace_bytes);
  uint32_t *counts = ws.take<uint32_t>(1024);
  int nb = (int)std::min<int64_t>(std::max<int64_t>(1, (n + ABS_PER_BLOCK - 1) / ABS_PER_BLOCK), 1024);
  if (dtype == AV_F32) {
    float *buf = ws.take<float>(n > 0 ? n : 1);
    k_nz_count<float><<<nb, ABS_THREADS, 0, st>>>((const float *)model, n, counts);
    AV_LAUNCH_CHECK();
    k_nz_write<float><<<nb, ABS_THREADS, 0, st>>>((const float *)model, n, counts, buf);
    AV_LAUNCH_CHECK();
    k_seq_sum<float><<<1, 32, 0, st>>>(buf, counts, nb, (float *)out);
  } else {
    double *buf = ws.take<double>(n > 0 ? n : 1);
    k_nz_count<double><<<nb, ABS_THREADS, 0, st>>>((const double *)model, n, counts);
    AV_LAUNCH_CHECK();
    k_nz_write<double><<<nb, ABS_THREADS, 0, st>>>((const double *)model, n, counts, buf);
    AV_LAUNCH_CHECK();
    k_seq_sum<double><<<1, 32, 0, st>>>(buf, counts, nb, (double *)out);
  }
  AV_LAUNCH_CHECK();
  return AV_OK;
}

}  // extern "C"
