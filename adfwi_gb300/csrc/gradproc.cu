// Gaussian smoothing of model-sized planes for the gradient processor (sm_103a, FP64).
//
// Reference (paths inside liufeng2317/ADFWI): ADFWI/propagator/gradient_process.py:14-49
// (gauss2, smooth2d) as used by GradProcessor.forward (74-134) for the illumination
// preconditioner and the gradient smoothing. smooth2d(Z, span) convolves Z ('same' size, zero
// outside) with a normalised 2-D Gaussian of standard deviation `span` sampled at the points
// -2 span, -2 span + 2, ..., 2 span of both axes, and divides by the same convolution of a
// plane of ones. The Gaussian is the outer product of its 1-D sampling, so the convolution is
// applied as two 1-D passes (rows, then columns) with weights w_k = f_k / sum(f),
// f_k = exp(-(x_k / span)^2 / 2), and the normaliser is the product of the 1-D weight sums
// over the taps that fall inside the plane. Everything is FP64, as the reference's numpy.
//
// What bounds a pass is FP64 arithmetic, two lanes per clock and SM: 81 multiply-adds a cell at span 40
// are 17 us of a 200 x 600 plane. So the normalisers, sums of the same weights for a whole row or
// column, are formed once per row and column (in every cell they took two thirds of the column
// pass), and the elementwise steps of the processor ride on the passes and two more launches: a 200 x
// 600 gradient with illumination, taper, smoothing and scaling in seven launches, 395 -> 113 us.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/adfwi_gb300.h"
#include "common.cuh"

namespace adfwi {
namespace gp {

constexpr int kThreads = 256;

// A smoothing of rows of nx values: weights w, and the sums wz, wx of the weights that fall inside the
// plane of nz rows for each row and column. span 0: none.
struct Filter {
  int span, nz;
  double *w, *wz, *wx;
};

// One block per filter: w[k] = f_k / sum(f) for k = 0 .. 2 span (fixed-order sum), then its normalisers;
// the maxima's keys start at 0, below every value's.
__global__ void __launch_bounds__(kThreads) weights(Filter f0, Filter f1, int nx, unsigned long long* keys) {
  __shared__ double part[kThreads];
  const Filter f = blockIdx.x == 0 ? f0 : f1;
  if (blockIdx.x == 0 && threadIdx.x < 2 && keys != nullptr) keys[threadIdx.x] = 0ull;
  const int span = f.span, n = 2 * span + 1;
  if (span == 0) return;
  double acc = 0.0;
  for (int k = threadIdx.x; k < n; k += kThreads) {
    const double x = (-2.0 * span + 2.0 * k) / span;
    const double v = exp(-0.5 * x * x);
    f.w[k] = v;
    acc += v;
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) part[threadIdx.x] += part[threadIdx.x + s];
    __syncthreads();
  }
  const double total = part[0];
  for (int k = threadIdx.x; k < n; k += kThreads) f.w[k] = f.w[k] / total;
  __syncthreads();
  for (int e = threadIdx.x; e < f.nz + nx; e += kThreads) {
    const int i = e < f.nz ? e : e - f.nz, m = e < f.nz ? f.nz : nx;
    double sum = 0.0;
    for (int b = max(-span, -i); b <= min(span, m - 1 - i); ++b) sum += f.w[span + b];
    (e < f.nz ? f.wz : f.wx)[i] = sum;
  }
}

// Order-preserving keys of doubles for atomicMax, a NaN above all (as torch.max propagates it).
__device__ __forceinline__ unsigned long long key_of(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return isnan(v) ? ~0ull : (b >> 63 ? ~b : b | 1ull << 63);
}
__device__ __forceinline__ double value_of(unsigned long long k) {
  return __longlong_as_double((long long)(k == ~0ull ? k : (k >> 63 ? k & ~(1ull << 63) : ~k)));
}
// The maximum over the block's threads into *key (every thread calls it; without a value v = -inf).
__device__ __forceinline__ void block_max(double v, unsigned long long* key) {
  __shared__ unsigned long long part[kThreads / 32];
  unsigned long long k = key_of(v);
  for (int s = 16; s > 0; s >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, s));
  if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = k;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < kThreads / 32; ++q) k = max(k, part[q]);
    atomicMax(key, k);
  }
}

// Row pass: t(i, j) = sum_b w[span + b] z(i, j + b), zero outside the plane. STAGED: the block's part of
// the row lies in shared memory in double precision (converting a single at each of the 2 span + 1 taps
// would take as long as the arithmetic); spans whose part exceeds kStagedBytes read it in place.
constexpr int kStagedBytes = 48 * 1024;
template <typename T, bool STAGED>
__global__ void __launch_bounds__(kThreads) pass_rows(int nx, Filter f, const T* __restrict__ z, double* __restrict__ t) {
  extern __shared__ double row_s[];
  const int j0 = blockIdx.x * blockDim.x, j = j0 + threadIdx.x, i = blockIdx.y, span = f.span;
  const T* row = z + (int64_t)i * nx;
  if (STAGED) {
    for (int k = threadIdx.x; k < kThreads + 2 * span; k += kThreads) {
      const int c = j0 - span + k;
      row_s[k] = c >= 0 && c < nx ? (double)row[c] : 0.0;
    }
    __syncthreads();
  }
  if (j >= nx) return;
  const int b0 = max(-span, -j), b1 = min(span, nx - 1 - j);
  double acc = 0.0;
  for (int b = b0; b <= b1; ++b) acc += __ldg(f.w + span + b) * (STAGED ? row_s[threadIdx.x + span + b] : (double)row[j + b]);
  t[(int64_t)i * nx + j] = acc;
}
template <typename T>
void launch_rows(dim3 grid, int nx, const Filter& f, const T* z, double* t, cudaStream_t st) {
  const int64_t bytes = (kThreads + 2 * (int64_t)f.span) * 8;
  if (bytes <= kStagedBytes)
    ADFWI_LAUNCH(kAux, st, (pass_rows<T, true><<<grid, kThreads, (size_t)bytes, st>>>(nx, f, z, t)));
  else
    ADFWI_LAUNCH(kAux, st, (pass_rows<T, false><<<grid, kThreads, 0, st>>>(nx, f, z, t)));
}

// Column pass and normalisation: out(i, j) = sum_a w[span + a] t(i + a, j) / (wz(i) wx(j)); key: the
// maximum of what is written plus `shift` (absolute values with shift < 0).
__global__ void __launch_bounds__(kThreads) pass_cols(int nx, Filter f, const double* __restrict__ t,
                                                      double* __restrict__ out, double shift, unsigned long long* key) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y, span = f.span;
  double v = 0.0;
  if (j < nx) {
    const int a0 = max(-span, -i), a1 = min(span, f.nz - 1 - i);
    double acc = 0.0;
    for (int a = a0; a <= a1; ++a) acc += __ldg(f.w + span + a) * t[(int64_t)(i + a) * nx + j];
    v = acc / (__ldg(f.wz + i) * __ldg(f.wx + j));
    out[(int64_t)i * nx + j] = v;
  }
  if (key != nullptr) block_max(j >= nx ? -INFINITY : (shift < 0.0 ? fabs(v) : v + shift), key);
}

// The gradient with taper and mask (each product rounded to single), divided by the squared
// preconditioner: p / max(p + 1e-5), at least 1e-4. key: the maximum of the absolute values of the rows
// above `rows` (those that no smoothing follows).
__global__ void __launch_bounds__(kThreads) precondition(int64_t n, int64_t rows_n, const float* __restrict__ g,
                                                         const double* __restrict__ taper, const double* __restrict__ mask,
                                                         const double* __restrict__ p, const unsigned long long* pmax,
                                                         double* __restrict__ out, unsigned long long* key) {
  const int64_t e = blockIdx.x * (int64_t)kThreads + threadIdx.x;
  double v = -INFINITY;
  if (e < n) {
    float x = g[e];
    if (taper != nullptr) x = (float)((double)x * taper[e]);
    if (mask != nullptr) x = (float)((double)x * mask[e]);
    double q = p[e] / value_of(*pmax);
    q = q < 1e-4 ? 1e-4 : q;
    v = (double)x / (q * q);
    out[e] = v;
    v = e < rows_n ? fabs(v) : -INFINITY;
  }
  block_max(v, key);
}

__global__ void __launch_bounds__(kThreads) scale(int64_t n, double vmax, const unsigned long long* gmax, double* g) {
  const int64_t e = blockIdx.x * (int64_t)kThreads + threadIdx.x;
  if (e < n) g[e] = vmax * g[e] / value_of(*gmax);
}

int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

// A filter's arrays (weights, normalisers) laid out at `at`; bytes they take.
int64_t filter_bytes(int nz, int nx, int span) { return align256(((int64_t)2 * span + 1 + nz + nx) * 8); }
Filter filter(int nz, int nx, int span, void* at) {
  double* w = static_cast<double*>(at);
  return {span, nz, w, w + 2 * span + 1, w + 2 * span + 1 + nz};
}
dim3 plane_grid(int nz, int nx) { return dim3((unsigned)((nx + kThreads - 1) / kThreads), (unsigned)nz); }

}  // namespace gp
}  // namespace adfwi

using namespace adfwi;

extern "C" {

int adfwi_smooth2d_workspace_bytes(int32_t nz, int32_t nx, int32_t span, int64_t* bytes) {
  ADFWI_CHECK_ARG(bytes != nullptr, "null output pointer");
  ADFWI_CHECK_ARG(nz > 0 && nx > 0 && span > 0, "nz, nx and span must be positive");
  *bytes = gp::align256((int64_t)nz * nx * 8) + gp::filter_bytes(nz, nx, span);
  return kOk;
}

int adfwi_smooth2d(int32_t nz, int32_t nx, int32_t span, const double* in, double* out, void* workspace,
                   int64_t workspace_bytes, void* stream) {
  ADFWI_CHECK_ARG(nz > 0 && nx > 0 && span > 0, "nz, nx and span must be positive");
  ADFWI_CHECK_ARG(in && out && workspace, "null array");
  int64_t need = 0;
  adfwi_smooth2d_workspace_bytes(nz, nx, span, &need);
  if (workspace_bytes < need) {
    set_error("smooth2d workspace too small: %lld bytes given, %lld needed", (long long)workspace_bytes,
              (long long)need);
    return kWorkspaceTooSmall;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double* t = static_cast<double*>(workspace);
  const gp::Filter f = gp::filter(nz, nx, span, static_cast<unsigned char*>(workspace) + gp::align256((int64_t)nz * nx * 8));
  const dim3 grid = gp::plane_grid(nz, nx);
  ADFWI_LAUNCH(kAux, st, (gp::weights<<<1, gp::kThreads, 0, st>>>(f, f, nx, nullptr)));
  gp::launch_rows(grid, nx, f, in, t, st);
  ADFWI_LAUNCH(kAux, st, (gp::pass_cols<<<grid, gp::kThreads, 0, st>>>(nx, f, t, out, 0.0, nullptr)));
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

int adfwi_gradproc_workspace_bytes(int32_t nz, int32_t nx, int32_t span, int32_t smooth, int64_t* bytes) {
  ADFWI_CHECK_ARG(bytes != nullptr, "null output pointer");
  ADFWI_CHECK_ARG(nz > 0 && nx > 0 && span > 0 && smooth >= 0, "nz, nx and span must be positive");
  *bytes = 256 + 2 * gp::align256((int64_t)nz * nx * 8) + gp::filter_bytes(nz, nx, span) + gp::filter_bytes(nz, nx, smooth);
  return kOk;
}

int adfwi_gradproc(int32_t nz, int32_t nx, int32_t span, int32_t smooth, int32_t keep_rows, const float* grad,
                   const double* taper, const double* mask, int32_t illum_dtype, const void* illum, int32_t norm,
                   double vmax, double* out, void* workspace, int64_t workspace_bytes, void* stream) {
  int64_t need = 0;
  const int rc = adfwi_gradproc_workspace_bytes(nz, nx, span, smooth, &need);
  if (rc) return rc;
  ADFWI_CHECK_ARG(grad && illum && out && workspace, "null array");
  ADFWI_CHECK_ARG(illum_dtype == ADFWI_F32 || illum_dtype == ADFWI_F64, "illumination must be ADFWI_F32 or ADFWI_F64");
  ADFWI_CHECK_ARG(keep_rows >= 0 && keep_rows < nz, "keep_rows must leave a row to smooth");
  if (workspace_bytes < need) {
    set_error("gradproc workspace too small: %lld bytes given, %lld needed", (long long)workspace_bytes, (long long)need);
    return kWorkspaceTooSmall;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  const int64_t n = (int64_t)nz * nx, plane = gp::align256(n * 8);
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(ws);
  double* t = reinterpret_cast<double*>(ws + 256);
  double* p = reinterpret_cast<double*>(ws + 256 + plane);
  const gp::Filter fi = gp::filter(nz, nx, span, ws + 256 + 2 * plane);
  const gp::Filter fs = gp::filter(nz - keep_rows, nx, smooth, ws + 256 + 2 * plane + gp::filter_bytes(nz, nx, span));
  const dim3 grid = gp::plane_grid(nz, nx);
  const unsigned blocks = (unsigned)((n + gp::kThreads - 1) / gp::kThreads);
  ADFWI_LAUNCH(kAux, st, (gp::weights<<<2, gp::kThreads, 0, st>>>(fi, fs, nx, keys)));
  if (illum_dtype == ADFWI_F32)
    gp::launch_rows(grid, nx, fi, static_cast<const float*>(illum), t, st);
  else
    gp::launch_rows(grid, nx, fi, static_cast<const double*>(illum), t, st);
  ADFWI_LAUNCH(kAux, st, (gp::pass_cols<<<grid, gp::kThreads, 0, st>>>(nx, fi, t, p, 1e-5, keys)));
  ADFWI_LAUNCH(kAux, st, (gp::precondition<<<blocks, gp::kThreads, 0, st>>>(
                             n, smooth ? (int64_t)keep_rows * nx : n, grad, taper, mask, p, keys, out, keys + 1)));
  if (smooth) {
    const dim3 gs = gp::plane_grid(nz - keep_rows, nx);
    double* o = out + (int64_t)keep_rows * nx;
    gp::launch_rows(gs, nx, fs, (const double*)o, t, st);
    ADFWI_LAUNCH(kAux, st, (gp::pass_cols<<<gs, gp::kThreads, 0, st>>>(nx, fs, t, o, -1.0, keys + 1)));
  }
  if (norm) ADFWI_LAUNCH(kAux, st, (gp::scale<<<blocks, gp::kThreads, 0, st>>>(n, vmax, keys + 1, out)));
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // extern "C"
