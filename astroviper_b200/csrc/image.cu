// Image formation (grid2image_spheroid_ms4, standard_grid.py:693-708) and the
// centred FFT helpers (fft.py:5, ifft.py:5).
//
// The image is the real part of the inverse transform, which is the inverse
// transform of the grid's Hermitian part: k_herm_in gathers it (with the
// ifftshift) into half-spectrum rows, cuFFT runs Z2D, and k_image_epilogue
// does the fftshift, the grid correction 1 / (grdsf(x) grdsf(y)) and the
// nx*ny / sumwt scaling.  numpy's ifft2 carries 1/(nx*ny), which the
// reference multiplies back: the unnormalised cuFFT inverse is the same
// quantity.  A real image's forward transform is D2Z, and k_herm_out writes
// both halves of its spectrum.  Complex data go through Z2Z / C2C
// (av_fft_shifted).
#include <cufft.h>
#include <math_constants.h>

#include <algorithm>
#include <deque>
#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace av {

// ----------------------------------------------------------- plan cache ---
enum FftKind { FFT_C2C, FFT_Z2Z, FFT_Z2D, FFT_D2Z };

struct FftPlan {
  int dev;
  int64_t nplanes, nx, ny;
  FftKind kind;
  cufftHandle h;
  size_t work;
};
static std::mutex g_fft_mu;
static std::deque<FftPlan> g_fft_plans;  // stable addresses on push_back

#define AV_CUFFT(call)                                                        \
  do {                                                                        \
    cufftResult r_ = (call);                                                  \
    if (r_ != CUFFT_SUCCESS) {                                                \
      ::av::set_error("%s failed: cufftResult %d (%s:%d)", #call, (int)r_,    \
                      __FILE__, __LINE__);                                    \
      return AV_ERR_CUDA;                                                     \
    }                                                                         \
  } while (0)

// Complex columns of a half-spectrum row; a real row in the same buffer is
// 2 * half_cols doubles apart.
__host__ __device__ constexpr int64_t half_cols(int64_t ny) { return ny / 2 + 1; }

// Plan for nplanes batched (nx, ny) transforms in place, without
// auto-allocated work area (the caller's workspace is attached per call).
// The real transforms keep ny / 2 + 1 complex (2 (ny / 2 + 1) real) columns.
static int get_plan(int64_t nplanes, int64_t nx, int64_t ny, FftKind kind, FftPlan **out) {
  int dev = 0;
  AV_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_fft_mu);
  for (auto &p : g_fft_plans)
    if (p.dev == dev && p.nplanes == nplanes && p.nx == nx && p.ny == ny && p.kind == kind) {
      *out = &p;
      return AV_OK;
    }
  FftPlan p;
  p.dev = dev;
  p.nplanes = nplanes;
  p.nx = nx;
  p.ny = ny;
  p.kind = kind;
  AV_CUFFT(cufftCreate(&p.h));
  AV_CUFFT(cufftSetAutoAllocation(p.h, 0));
  long long n[2] = {nx, ny};
  size_t ws = 0;
  if (kind == FFT_Z2D || kind == FFT_D2Z) {
    const long long h = half_cols(ny);
    long long cplx[2] = {nx, h}, real[2] = {nx, 2 * h};
    const bool inv = kind == FFT_Z2D;
    AV_CUFFT(cufftMakePlanMany64(p.h, 2, n, inv ? cplx : real, 1, nx * (inv ? h : 2 * h),
                                 inv ? real : cplx, 1, nx * (inv ? 2 * h : h),
                                 inv ? CUFFT_Z2D : CUFFT_D2Z, nplanes, &ws));
  } else {
    AV_CUFFT(cufftMakePlanMany64(p.h, 2, n, nullptr, 1, nx * ny, nullptr, 1, nx * ny,
                                 kind == FFT_Z2Z ? CUFFT_Z2Z : CUFFT_C2C, nplanes, &ws));
  }
  p.work = ws;
  g_fft_plans.push_back(p);
  *out = &g_fft_plans.back();
  return AV_OK;
}

// Work-area bytes of the (cached) plan for this size.
static size_t fft_work_bytes(int64_t nplanes, int64_t nx, int64_t ny, FftKind kind) {
  FftPlan *p = nullptr;
  if (get_plan(nplanes, nx, ny, kind, &p) != AV_OK) return 0;
  return p->work;
}

// ifftshift gather: buf[i, j] = in[(i + nx/2) % nx, (j + ny/2) % ny]
template <typename CT, typename IT>
__global__ void k_ishift_in(const IT *in, CT *buf, int64_t nplanes, int64_t nx, int64_t ny) {
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t n = nplanes * nx * ny;
  if (k >= n) return;
  int64_t p = k / (nx * ny), r = k - p * nx * ny;
  int64_t i = r / ny, j = r - i * ny;
  int64_t si = i + nx / 2;
  if (si >= nx) si -= nx;
  int64_t sj = j + ny / 2;
  if (sj >= ny) sj -= ny;
  IT v = in[p * nx * ny + si * ny + sj];
  CT o;
  o.x = v.x;
  o.y = v.y;
  buf[k] = o;
}

// The kernels around the real transforms.  A block takes 128 columns of 16
// rows of one plane (grid: column tiles, row groups, planes), so a
// thread evaluates the grid correction's factor of its column once and the
// block the factors of its rows once: an evaluation per pixel, a long chain
// of FP64 operations and divides, had made the epilogue of four 2048^2 images
// 548 us (85 with the factors per row and column, 61 now).  IMG_UNROLL rows in
// flight per thread: 8 take the epilogue there from 68 to 61 us and the gather
// from 65 to 62 against 4, 2 79 us.  16 rows to a block give a 1024^2 image
// enough blocks (prologue and epilogue 20 us; 30 with 32 rows).
// The real transforms themselves halve what the complex ones moved: the
// gather 95 -> 62 us and cuFFT 289 -> 175 us for four 2048^2 planes, whole
// images 932 -> 302 us.  Batches of planes small enough to stay in L2 between
// the passes gained nothing (374 us: cuFFT is bound by its FP64 work there).
// A plane whose blocks would leave SMs idle takes 4 rows to a block (257^2:
// 33 us -> 31, 512^2 25 -> 23), and one of up to 64 columns, whose rows would
// leave most threads idle, eight groups of 4 rows side by side (20,000 x 20:
// 39 -> 32 us, 100,000 x 2 74 -> 50).  Single planes of odd size below 500^2
// stay slower than with complex transforms (257^2: 23 us), for the library's
// real ones: hidden behind the call's host work.
constexpr int IMG_THREADS = 128, IMG_UNROLL = 8;

// LANES groups of ROWS rows side by side, THREADS / LANES columns wide.
template <int LANES_, int ROWS_>
struct ImgBlock {
  static constexpr int LANES = LANES_, ROWS = ROWS_, COLS = IMG_THREADS / LANES;
  static constexpr int UNROLL = ROWS < IMG_UNROLL ? ROWS : IMG_UNROLL;
  static_assert(COLS >= ROWS, "a group's threads set up its rows");
  static dim3 grid(int64_t nplanes, int64_t rows, int64_t cols) {
    return dim3((unsigned)((cols + COLS - 1) / COLS),
                (unsigned)std::min<int64_t>((rows + LANES * ROWS - 1) / (LANES * ROWS), 65535),
                (unsigned)std::min<int64_t>(nplanes, 65535));
  }
  // For the passes with the grid correction: two planes to a block where that
  // leaves 16 blocks per SM, so a factor serves twice the pixels (four 2048^2
  // images 68 -> 61 us).
  static dim3 pixel_grid(int64_t nplanes, int64_t nx, int64_t ny) {
    dim3 g = grid(nplanes, nx, ny);
    const int64_t pairs = (nplanes + 1) / 2;
    if (pairs <= 65535 && (int64_t)g.x * g.y * pairs >= (int64_t)sm_count() * 16)
      g.z = (unsigned)pairs;
    return g;
  }
  static __device__ __forceinline__ int place() {  // in the group
    return LANES == 1 ? threadIdx.x : threadIdx.x % COLS;
  }
  static __device__ __forceinline__ int64_t col() {
    return blockIdx.x * (int64_t)COLS + place();
  }
  static __device__ __forceinline__ int lane() { return LANES == 1 ? 0 : threadIdx.x / COLS; }
};

// f(the block's shape) for planes of rows x cols.
template <typename F>
static void with_img_block(int64_t nplanes, int64_t rows, int64_t cols, F f) {
  using Wide = ImgBlock<1, 16>;
  if (cols <= 64) return f(ImgBlock<8, 4>());
  const dim3 g = Wide::grid(nplanes, rows, cols);
  if ((int64_t)g.x * g.y * g.z < 2 * (int64_t)sm_count()) return f(ImgBlock<1, 4>());
  f(Wide());
}

// i + s for 0 <= i < n, 0 <= s <= n, modulo n.
__device__ __forceinline__ int64_t wrap(int64_t i, int64_t s, int64_t n) {
  i += s;
  return i >= n ? i - n : i;
}

// Grid-correction factor of pixel i of n along one axis.
__device__ __forceinline__ double corr_factor(int64_t i, int64_t n) {
  return pswf_grdsf(fabs(2.0 * ((double)(i - n / 2) / (double)n)));
}

// v / d for 1e-20 < |d| < 1e300 and r near 1 / d (a few ulp), by Markstein's
// correction ("Computation of elementary functions on the IBM RISC System/6000
// processor", 1990): one Newton step makes r the rounded reciprocal, and the
// exact remainder of v r corrects the quotient's last bit.  7 FP64 operations
// per pixel in place of a divide's call; zeros, infinities, NaN and results
// whose remainder could leave the normal range take the divide.
__device__ __forceinline__ double quotient(double v, double d, double r) {
  r = fma(r, fma(-d, r, 1.0), r);
  double q = v * r;
  const double m = fabs(q);
  if (!(m > 1e-250 && m < 1e250)) return v / d;
  return fma(fma(-q, d, v), r, q);
}

// 1 / d rounded where quotient_by corrects its products; NaN, which sends
// every quotient to the divide, for a d so small that a remainder could fall
// below the normal range, or so large that 1 / d does.
__device__ __forceinline__ double reciprocal_for_quotient(double d) {
  const double m = fabs(d);
  return m > 1e-20 && m < 1e300 ? 1.0 / d : CUDART_NAN;
}

// v / d for r = reciprocal_for_quotient(d): as above without the Newton step.
__device__ __forceinline__ double quotient_by(double v, double d, double r) {
  const double q = v * r;
  const double m = fabs(q);
  if (!(m > 1e-250 && m < 1e250)) return v / d;
  return fma(fma(-q, d, v), r, q);
}

// Carries every pixel of this block's share from f.in to f.out, B::UNROLL
// rows at a time, with the grid correction's factors and their reciprocals (1
// without apply_corr).  The rows' wrapped offsets are worked out once for the
// block's planes: 64-bit index arithmetic per pixel had made the pass issue
// bound.
template <typename B, typename F>
__device__ __forceinline__ void for_pixels(int64_t nplanes, int64_t nx, int64_t ny,
                                           int apply_corr, F f) {
  __shared__ double2 sh_gx[B::LANES][B::ROWS];
  __shared__ int64_t sh_in[B::LANES][B::ROWS], sh_out[B::LANES][B::ROWS];
  double2 *s_gx = sh_gx[B::lane()];
  int64_t *s_in = sh_in[B::lane()], *s_out = sh_out[B::lane()];
  const int t = B::place();
  const int64_t j = B::col();
  double2 gy = make_double2(1.0, 1.0);
  if (apply_corr && j < ny) {
    gy.x = corr_factor(j, ny);
    gy.y = 1.0 / gy.x;
  }
  constexpr int64_t STEP = B::LANES * B::ROWS;
  for (int64_t first = blockIdx.y * STEP; first < nx; first += gridDim.y * STEP) {
    const int64_t i0 = first + B::lane() * B::ROWS;
    __syncthreads();
    if (t < B::ROWS && i0 + t < nx) {
      const int64_t i = i0 + t;
      const double g = apply_corr ? corr_factor(i, nx) : 1.0;
      s_gx[t] = make_double2(g, 1.0 / g);
      s_in[t] = f.row_in(i);
      s_out[t] = f.row_out(i);
    }
    __syncthreads();
    if (j >= ny) continue;
    const int rows = (int)std::min<int64_t>(B::ROWS, nx - i0);  // below 1 past the image
    for (int64_t p = blockIdx.z; p < nplanes; p += gridDim.z) {
      const double sw = f.sumw ? f.sumw[p] : 1.0, rsw = reciprocal_for_quotient(sw);
      const auto *in = f.in + p * f.plane_in() + f.col_in(j);
      auto *out = f.out + p * f.plane_out() + f.col_out(j);
      for (int r = 0; r < rows; r += B::UNROLL) {
        double v[B::UNROLL];
#pragma unroll
        for (int k = 0; k < B::UNROLL; ++k)
          if (r + k < rows) v[k] = (double)in[s_in[r + k]];
#pragma unroll
        for (int k = 0; k < B::UNROLL; ++k)
          if (r + k < rows) {
            const double2 gx = s_gx[r + k];
            if (apply_corr) v[k] = quotient(v[k], gx.x * gy.x, gx.y * gy.y);
            if (f.sumw) v[k] = quotient_by(v[k], sw, rsw);
            f.store(out + s_out[r + k], v[k]);
          }
      }
    }
  }
}

// Half spectrum of the Hermitian part of the ifftshifted grid:
// buf[i, j] = (s[i, j] + conj(s[-i, -j])) / 2, j <= ny / 2, with
// s[i, j] = grid[(i + nx/2) % nx, (j + ny/2) % ny].
template <typename B, typename IT>
__global__ void __launch_bounds__(IMG_THREADS) k_herm_in(const IT *grid, double2 *buf,
                                                         int64_t nplanes, int64_t nx, int64_t ny) {
  const int64_t h = half_cols(ny);
  const int64_t j = B::col();
  if (j >= h) return;
  const int64_t ja = wrap(j, ny / 2, ny);
  const int64_t jb = wrap(j == 0 ? 0 : ny - j, ny / 2, ny);
  constexpr int64_t STEP = B::LANES * B::ROWS;
  for (int64_t i0 = blockIdx.y * STEP + B::lane() * B::ROWS; i0 < nx; i0 += gridDim.y * STEP) {
    const int rows = (int)std::min<int64_t>(B::ROWS, nx - i0);
    for (int64_t p = blockIdx.z; p < nplanes; p += gridDim.z) {
      const IT *g = grid + p * nx * ny;
      for (int r = 0; r < rows; r += B::UNROLL) {
        IT a[B::UNROLL], b[B::UNROLL];
#pragma unroll
        for (int k = 0; k < B::UNROLL; ++k)
          if (r + k < rows) {
            const int64_t i = i0 + r + k;
            a[k] = __ldcs(g + wrap(i, nx / 2, nx) * ny + ja);
            b[k] = __ldcs(g + wrap(i == 0 ? 0 : nx - i, nx / 2, nx) * ny + jb);
          }
#pragma unroll
        for (int k = 0; k < B::UNROLL; ++k)
          if (r + k < rows)
            buf[(p * nx + i0 + r + k) * h + j] =
                make_double2(0.5 * ((double)a[k].x + (double)b[k].x),
                             0.5 * ((double)a[k].y - (double)b[k].y));
      }
    }
  }
}

// fftshift of the transform + grid correction + normalisation:
// img[i, j] = t[(i + nx - nx/2) % nx, (j + ny - ny/2) % ny] / (gx gy) / sumw.
template <typename OT>
struct ImageEpilogue {
  const double *in;
  OT *out;
  const double *sumw;
  int64_t nx, ny;
  int apply_corr;
  __device__ int64_t plane_in() const { return nx * 2 * half_cols(ny); }
  __device__ int64_t plane_out() const { return nx * ny; }
  __device__ int64_t row_in(int64_t i) const {
    return wrap(i, nx - nx / 2, nx) * 2 * half_cols(ny);
  }
  __device__ int64_t row_out(int64_t i) const { return i * ny; }
  __device__ int64_t col_in(int64_t j) const { return wrap(j, ny - ny / 2, ny); }
  __device__ int64_t col_out(int64_t j) const { return j; }
  __device__ void store(OT *at, double v) const { __stcs(at, (OT)v); }
};

template <typename B, typename OT>
__global__ void __launch_bounds__(IMG_THREADS) k_image_epilogue(ImageEpilogue<OT> f,
                                                                int64_t nplanes) {
  for_pixels<B>(nplanes, f.nx, f.ny, f.apply_corr, f);
}

// ifftshift of a real image into the transform's real rows, divided by the
// grid correction when asked.
template <typename IT>
struct ImagePrologue {
  const IT *in;
  double *out;
  const double *sumw;  // none
  int64_t nx, ny;
  int apply_corr;
  __device__ int64_t plane_in() const { return nx * ny; }
  __device__ int64_t plane_out() const { return nx * 2 * half_cols(ny); }
  __device__ int64_t row_in(int64_t i) const { return i * ny; }
  __device__ int64_t row_out(int64_t i) const {
    return wrap(i, nx - nx / 2, nx) * 2 * half_cols(ny);
  }
  __device__ int64_t col_in(int64_t j) const { return j; }
  __device__ int64_t col_out(int64_t j) const { return wrap(j, ny - ny / 2, ny); }
  __device__ void store(double *at, double v) const { *at = v; }
};

template <typename B, typename IT>
__global__ void __launch_bounds__(IMG_THREADS) k_image_prologue(ImagePrologue<IT> f,
                                                                int64_t nplanes) {
  for_pixels<B>(nplanes, f.nx, f.ny, f.apply_corr, f);
}

// fftshift of a half spectrum to a full grid: the other half is the
// conjugate of the mirrored one.
template <typename B, typename OT>
__global__ void __launch_bounds__(IMG_THREADS) k_herm_out(const double2 *buf, OT *grid,
                                                          int64_t nplanes, int64_t nx,
                                                          int64_t ny) {
  const int64_t h = half_cols(ny);
  const int64_t j = B::col();
  if (j >= ny) return;
  const int64_t sj = wrap(j, ny - ny / 2, ny);
  const bool mirror = sj >= h;
  const int64_t bj = mirror ? ny - sj : sj;
  constexpr int64_t STEP = B::LANES * B::ROWS;
  for (int64_t i0 = blockIdx.y * STEP + B::lane() * B::ROWS; i0 < nx; i0 += gridDim.y * STEP) {
    const int rows = (int)std::min<int64_t>(B::ROWS, nx - i0);
    for (int64_t p = blockIdx.z; p < nplanes; p += gridDim.z)
      for (int r = 0; r < rows; r += B::UNROLL) {
        double2 v[B::UNROLL];
#pragma unroll
        for (int k = 0; k < B::UNROLL; ++k)
          if (r + k < rows) {
            int64_t si = wrap(i0 + r + k, nx - nx / 2, nx);
            if (mirror && si != 0) si = nx - si;
            v[k] = buf[(p * nx + si) * h + bj];
          }
#pragma unroll
        for (int k = 0; k < B::UNROLL; ++k)
          if (r + k < rows) {
            OT o;
            o.x = v[k].x;
            o.y = mirror ? -v[k].y : v[k].y;
            grid[(p * nx + i0 + r + k) * ny + j] = o;
          }
      }
  }
}

// fftshift gather of a complex result: out[i] = buf[(i + nx - nx/2) % nx].
template <typename CT, typename OT>
__global__ void k_shift_out(const CT *buf, OT *out, int64_t nplanes, int64_t nx, int64_t ny,
                            double scale) {
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t n = nplanes * nx * ny;
  if (k >= n) return;
  int64_t p = k / (nx * ny), r = k - p * nx * ny;
  int64_t i = r / ny, j = r - i * ny;
  int64_t si = i + (nx - nx / 2);
  if (si >= nx) si -= nx;
  int64_t sj = j + (ny - ny / 2);
  if (sj >= ny) sj -= ny;
  CT v = buf[p * nx * ny + si * ny + sj];
  OT o;
  o.x = v.x * scale;
  o.y = v.y * scale;
  out[k] = o;
}

// In place on buf; dir counts for the complex kinds.
static int run_fft(void *buf, FftKind kind, int64_t nplanes, int64_t nx, int64_t ny, int dir,
                   void *work, cudaStream_t st) {
  FftPlan *p = nullptr;
  int rc = get_plan(nplanes, nx, ny, kind, &p);
  if (rc) return rc;
  AV_CUFFT(cufftSetStream(p->h, st));
  AV_CUFFT(cufftSetWorkArea(p->h, work));
  switch (kind) {
    case FFT_C2C:
      AV_CUFFT(cufftExecC2C(p->h, (cufftComplex *)buf, (cufftComplex *)buf, dir));
      break;
    case FFT_Z2Z:
      AV_CUFFT(cufftExecZ2Z(p->h, (cufftDoubleComplex *)buf, (cufftDoubleComplex *)buf, dir));
      break;
    case FFT_Z2D:
      AV_CUFFT(cufftExecZ2D(p->h, (cufftDoubleComplex *)buf, (cufftDoubleReal *)buf));
      break;
    case FFT_D2Z:
      AV_CUFFT(cufftExecD2Z(p->h, (cufftDoubleReal *)buf, (cufftDoubleComplex *)buf));
      break;
  }
  return AV_OK;
}

// Buffer and work area of a real transform of nplanes planes.
static int real_fft_need(int64_t nplanes, int64_t nx, int64_t ny, FftKind kind, size_t *buf,
                         size_t *work) {
  *buf = (size_t)nplanes * nx * half_cols(ny) * 16;
  FftPlan *p = nullptr;
  int rc = get_plan(nplanes, nx, ny, kind, &p);
  if (rc) return rc;
  *work = p->work;
  return AV_OK;
}

}  // namespace av

using namespace av;

extern "C" {

size_t av_fft_workspace_size(int64_t nplanes, int64_t nx, int64_t ny, int precision) {
  int dbl = precision == AV_F64 || precision == AV_C128;
  size_t buf = (size_t)nplanes * nx * ny * (dbl ? 16 : 8);
  return Workspace::need(buf) +
         Workspace::need(fft_work_bytes(nplanes, nx, ny, dbl ? FFT_Z2Z : FFT_C2C));
}

size_t av_real_fft_workspace_size(int64_t nplanes, int64_t nx, int64_t ny, int inverse) {
  size_t buf = 0, work = 0;
  if (nplanes <= 0 || nx <= 0 || ny <= 0) return 0;
  real_fft_need(nplanes, nx, ny, inverse ? FFT_Z2D : FFT_D2Z, &buf, &work);
  return Workspace::need(buf) + Workspace::need(work);
}

size_t av_grid_to_image_workspace_size(int64_t nplanes, int64_t nx, int64_t ny) {
  return std::max(av_real_fft_workspace_size(nplanes, nx, ny, 1),
                  av_real_fft_workspace_size(nplanes, nx, ny, 0));
}

// The transform is always FP64: the grid correction divides by a taper
// that is ~4e-3 at the image edges, which would amplify FP32 transform
// rounding to ~1e-4 relative error in the image.
int av_grid_to_image(const void *grid, int grid_dtype, const double *sum_weight, void *image,
                     int image_dtype, int64_t nplanes, int64_t nx, int64_t ny, int apply_corr,
                     void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  AV_CHECK_ARG(grid && image, "av_grid_to_image: null pointer");
  AV_CHECK_ARG(grid_dtype == AV_C64 || grid_dtype == AV_C128, "av_grid_to_image: grid dtype");
  AV_CHECK_ARG(image_dtype == AV_F32 || image_dtype == AV_F64, "av_grid_to_image: image dtype");
  AV_CHECK_ARG(nplanes >= 0 && nx > 0 && ny > 0, "av_grid_to_image: bad shape");
  if (nplanes == 0) return AV_OK;
  size_t bufb = 0, workb = 0;
  int rc = real_fft_need(nplanes, nx, ny, FFT_Z2D, &bufb, &workb);
  if (rc) return rc;
  if (!workspace || workspace_bytes < Workspace::need(bufb) + Workspace::need(workb)) {
    set_error("av_grid_to_image: workspace too small (%zu < %zu)", workspace_bytes,
              Workspace::need(bufb) + Workspace::need(workb));
    return AV_ERR_WORKSPACE;
  }
  Workspace ws(workspace, workspace_bytes);
  double2 *buf = ws.take<double2>(bufb / sizeof(double2));
  void *work = ws.take<char>(workb > 0 ? workb : 1);
  cudaStream_t st = as_stream(stream);
  with_img_block(nplanes, nx, half_cols(ny), [&](auto block) {
    using B = decltype(block);
    const dim3 g = B::grid(nplanes, nx, half_cols(ny));
    if (grid_dtype == AV_C128)
      k_herm_in<B><<<g, IMG_THREADS, 0, st>>>((const double2 *)grid, buf, nplanes, nx, ny);
    else
      k_herm_in<B><<<g, IMG_THREADS, 0, st>>>((const float2 *)grid, buf, nplanes, nx, ny);
  });
  AV_LAUNCH_CHECK();
  rc = run_fft(buf, FFT_Z2D, nplanes, nx, ny, CUFFT_INVERSE, work, st);
  if (rc) return rc;
  with_img_block(nplanes, nx, ny, [&](auto block) {
    using B = decltype(block);
    const dim3 g = B::pixel_grid(nplanes, nx, ny);
    auto run = [&](auto *out) {
      using T = std::remove_pointer_t<decltype(out)>;
      k_image_epilogue<B, T><<<g, IMG_THREADS, 0, st>>>(
          ImageEpilogue<T>{(const double *)buf, out, sum_weight, nx, ny, apply_corr}, nplanes);
    };
    if (image_dtype == AV_F64) run((double *)image);
    else run((float *)image);
  });
  AV_LAUNCH_CHECK();
  return AV_OK;
}

// fft_lm_to_uv(image / corrTerm) (fft.py:5 with the grid correction of
// gcf_prolate_spheroidal.py:73-79): the forward model's image -> grid step,
// the adjoint of av_grid_to_image without sum_weight.  FP64 transform.
int av_image_to_grid(const void *image, int image_dtype, void *grid, int grid_dtype,
                     int64_t nplanes, int64_t nx, int64_t ny, int apply_corr, void *workspace,
                     size_t workspace_bytes, void *stream) {
  clear_error();
  AV_CHECK_ARG(image && grid, "av_image_to_grid: null pointer");
  AV_CHECK_ARG(image_dtype == AV_F32 || image_dtype == AV_F64, "av_image_to_grid: image dtype");
  AV_CHECK_ARG(grid_dtype == AV_C64 || grid_dtype == AV_C128, "av_image_to_grid: grid dtype");
  AV_CHECK_ARG(nplanes >= 0 && nx > 0 && ny > 0, "av_image_to_grid: bad shape");
  if (nplanes == 0) return AV_OK;
  size_t bufb = 0, workb = 0;
  int rc = real_fft_need(nplanes, nx, ny, FFT_D2Z, &bufb, &workb);
  if (rc) return rc;
  if (!workspace || workspace_bytes < Workspace::need(bufb) + Workspace::need(workb)) {
    set_error("av_image_to_grid: workspace too small");
    return AV_ERR_WORKSPACE;
  }
  Workspace ws(workspace, workspace_bytes);
  double2 *buf = ws.take<double2>(bufb / sizeof(double2));
  void *work = ws.take<char>(workb > 0 ? workb : 1);
  cudaStream_t st = as_stream(stream);
  with_img_block(nplanes, nx, ny, [&](auto block) {
    using B = decltype(block);
    const dim3 g = B::pixel_grid(nplanes, nx, ny);
    auto run = [&](const auto *in) {
      using T = std::remove_const_t<std::remove_pointer_t<decltype(in)>>;
      k_image_prologue<B, T><<<g, IMG_THREADS, 0, st>>>(
          ImagePrologue<T>{in, (double *)buf, nullptr, nx, ny, apply_corr}, nplanes);
    };
    if (image_dtype == AV_F64) run((const double *)image);
    else run((const float *)image);
  });
  AV_LAUNCH_CHECK();
  rc = run_fft(buf, FFT_D2Z, nplanes, nx, ny, CUFFT_FORWARD, work, st);
  if (rc) return rc;
  with_img_block(nplanes, nx, ny, [&](auto block) {
    using B = decltype(block);
    const dim3 g = B::grid(nplanes, nx, ny);
    if (grid_dtype == AV_C128)
      k_herm_out<B><<<g, IMG_THREADS, 0, st>>>(buf, (double2 *)grid, nplanes, nx, ny);
    else
      k_herm_out<B><<<g, IMG_THREADS, 0, st>>>(buf, (float2 *)grid, nplanes, nx, ny);
  });
  AV_LAUNCH_CHECK();
  return AV_OK;
}

int av_fft_shifted(const void *in, void *out, int dtype, int64_t nplanes, int64_t nx, int64_t ny,
                   int inverse, void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  AV_CHECK_ARG(in && out, "av_fft_shifted: null pointer");
  AV_CHECK_ARG(dtype == AV_C64 || dtype == AV_C128, "av_fft_shifted: dtype");
  AV_CHECK_ARG(nplanes >= 0 && nx > 0 && ny > 0, "av_fft_shifted: bad shape");
  if (nplanes == 0) return AV_OK;
  int dbl = dtype == AV_C128;
  const FftKind kind = dbl ? FFT_Z2Z : FFT_C2C;
  FftPlan *p = nullptr;
  int rc = get_plan(nplanes, nx, ny, kind, &p);
  if (rc) return rc;
  size_t bufb = (size_t)nplanes * nx * ny * (dbl ? 16 : 8);
  if (!workspace || workspace_bytes < Workspace::need(bufb) + Workspace::need(p->work)) {
    set_error("av_fft_shifted: workspace too small");
    return AV_ERR_WORKSPACE;
  }
  Workspace ws(workspace, workspace_bytes);
  void *buf = ws.take<char>(bufb);
  void *work = ws.take<char>(p->work > 0 ? p->work : 1);
  cudaStream_t st = as_stream(stream);
  int64_t n = nplanes * nx * ny;
  unsigned blocks = (unsigned)((n + 255) / 256);
  double scale = inverse ? 1.0 / ((double)nx * (double)ny) : 1.0;
  if (dbl)
    k_ishift_in<double2, double2><<<blocks, 256, 0, st>>>((const double2 *)in, (double2 *)buf,
                                                         nplanes, nx, ny);
  else
    k_ishift_in<float2, float2><<<blocks, 256, 0, st>>>((const float2 *)in, (float2 *)buf,
                                                       nplanes, nx, ny);
  AV_LAUNCH_CHECK();
  rc = run_fft(buf, kind, nplanes, nx, ny, inverse ? CUFFT_INVERSE : CUFFT_FORWARD, work, st);
  if (rc) return rc;
  if (dbl)
    k_shift_out<double2, double2><<<blocks, 256, 0, st>>>((const double2 *)buf, (double2 *)out,
                                                         nplanes, nx, ny, scale);
  else
    k_shift_out<float2, float2><<<blocks, 256, 0, st>>>((const float2 *)buf, (float2 *)out,
                                                       nplanes, nx, ny, scale);
  AV_LAUNCH_CHECK();
  return AV_OK;
}

}  // extern "C"
