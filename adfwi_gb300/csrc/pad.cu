// Edge-replicate padding of model planes and its adjoint, one launch each for all planes of a solve.
//
// Reference: ADFWI/propagator/acoustic_kernels.py:16-37, elastic_kernels.py:175-216 pad every
// coefficient plane by its own operation; the adjoint folds the padded strips into the edge rows and
// columns and the corner blocks into the corner cells. Both are launch-bound at model sizes (a few
// hundred kB): eight planes took 8 launches forward and some 100 in reverse (four strips and four
// corners of each, every one a sum and an addition), 1.7 ms of a gradient; they take one of 3 us and one of 6.
//
// A folded cell is summed in double precision in a fixed order (a warp's strided partial sums, then a
// shuffle tree), so a gradient is the same on every run.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/adfwi_gb300.h"
#include "common.cuh"

namespace adfwi {
namespace pad {

constexpr int kMost = ADFWI_PAD_PLANES, kThreads = 256, kWarps = kThreads / 32;

struct Planes {
  const void* src[kMost];
  void* dst[kMost];
  int h[kMost], w[kMost];  // the unpadded plane
  int top, bottom, left, right;
};

template <typename T>
__global__ void __launch_bounds__(kThreads) replicate(Planes p) {
  const int q = blockIdx.y, h = p.h[q], w = p.w[q], wp = w + p.left + p.right;
  const int64_t n = (int64_t)(h + p.top + p.bottom) * wp;
  const T* src = static_cast<const T*>(p.src[q]);
  T* dst = static_cast<T*>(p.dst[q]);
  for (int64_t e = blockIdx.x * (int64_t)kThreads + threadIdx.x; e < n; e += (int64_t)gridDim.x * kThreads) {
    const int i = (int)(e / wp), j = (int)(e - (int64_t)i * wp);
    dst[e] = src[(int64_t)min(max(i - p.top, 0), h - 1) * w + min(max(j - p.left, 0), w - 1)];
  }
}

// dst = the padded plane src folded to h x w. Cells off the edge are copied by one thread each; an edge
// cell is summed by a warp, a corner by a block (the last four).
template <typename T>
__global__ void __launch_bounds__(kThreads) fold(Planes p, int copy_blocks) {
  __shared__ double part[kWarps];
  const int q = blockIdx.y, h = p.h[q], w = p.w[q], wp = w + p.left + p.right;
  const T* src = static_cast<const T*>(p.src[q]);
  T* dst = static_cast<T*>(p.dst[q]);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if ((int)blockIdx.x < copy_blocks) {
    const int64_t n = (int64_t)h * w;
    for (int64_t e = blockIdx.x * (int64_t)kThreads + threadIdx.x; e < n; e += (int64_t)copy_blocks * kThreads) {
      const int i = (int)(e / w), j = (int)(e - (int64_t)i * w);
      if (i > 0 && i < h - 1 && j > 0 && j < w - 1) dst[e] = src[(int64_t)(i + p.top) * wp + j + p.left];
    }
    return;
  }
  const bool corner = blockIdx.x + 4 >= gridDim.x;
  int i, j;
  if (corner) {
    const int c = (int)(gridDim.x - 1 - blockIdx.x);
    i = c / 2 * (h - 1);
    j = c % 2 * (w - 1);
  } else {  // the rows 0 and h - 1, then the columns 0 and w - 1 between them
    const int e = ((int)blockIdx.x - copy_blocks) * kWarps + warp;
    if (e < 2 * w) {
      i = e / w * (h - 1);
      j = e % w;
    } else {
      i = 1 + (e - 2 * w) / 2;
      j = (e & 1) * (w - 1);
      if (i >= h - 1) return;
    }
    if ((i == 0 || i == h - 1) && (j == 0 || j == w - 1)) return;
  }
  // the rows and columns of src that map to (i, j)
  const int r0 = i == 0 ? 0 : i + p.top, r1 = (i == h - 1 ? h + p.top + p.bottom : i + p.top + 1);
  const int c0 = j == 0 ? 0 : j + p.left, nc = (j == w - 1 ? wp : j + p.left + 1) - c0;
  const int n = (r1 - r0) * nc;
  double acc = 0.0;
  for (int k = corner ? (int)threadIdx.x : lane; k < n; k += corner ? kThreads : 32) {
    const int r = k / nc;
    acc += (double)src[(int64_t)(r0 + r) * wp + c0 + k - r * nc];
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, s);
  if (corner) {
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < kWarps; ++k) acc += part[k];
      dst[(int64_t)i * w + j] = (T)acc;
    }
  } else if (lane == 0) {
    dst[(int64_t)i * w + j] = (T)acc;
  }
}

int planes(Planes* p, int n, const void* const* src, void* const* dst, const int32_t* shapes, int top, int bottom,
           int left, int right) {
  ADFWI_CHECK_ARG(n >= 1 && n <= kMost, "between 1 and ADFWI_PAD_PLANES planes");
  ADFWI_CHECK_ARG(src && dst && shapes, "null array");
  ADFWI_CHECK_ARG(top >= 0 && bottom >= 0 && left >= 0 && right >= 0, "negative padding");
  p->top = top;
  p->bottom = bottom;
  p->left = left;
  p->right = right;
  for (int q = 0; q < n; ++q) {
    ADFWI_CHECK_ARG(src[q] && dst[q], "null plane");
    ADFWI_CHECK_ARG(shapes[2 * q] >= 1 && shapes[2 * q + 1] >= 1, "empty plane");
    p->src[q] = src[q];
    p->dst[q] = dst[q];
    p->h[q] = shapes[2 * q];
    p->w[q] = shapes[2 * q + 1];
  }
  return kOk;
}

}  // namespace pad
}  // namespace adfwi

using namespace adfwi;

extern "C" {

int adfwi_pad_replicate(int32_t n, int32_t dtype, const void* const* src, void* const* dst, const int32_t* shapes,
                        int32_t top, int32_t bottom, int32_t left, int32_t right, void* stream) {
  ADFWI_CHECK_ARG(dtype == ADFWI_F32 || dtype == ADFWI_F64, "dtype must be ADFWI_F32 or ADFWI_F64");
  pad::Planes p;
  const int rc = pad::planes(&p, n, src, dst, shapes, top, bottom, left, right);
  if (rc) return rc;
  int64_t most = 1;
  for (int q = 0; q < n; ++q) most = std::max(most, (int64_t)(p.h[q] + top + bottom) * (p.w[q] + left + right));
  const dim3 g((unsigned)std::min<int64_t>((most + pad::kThreads - 1) / pad::kThreads, 4096), n);
  auto k = dtype == ADFWI_F32 ? pad::replicate<float> : pad::replicate<double>;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ADFWI_LAUNCH(kAux, st, (k<<<g, pad::kThreads, 0, st>>>(p)));
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

int adfwi_fold_replicate(int32_t n, int32_t dtype, const void* const* src, void* const* dst, const int32_t* shapes,
                         int32_t top, int32_t bottom, int32_t left, int32_t right, void* stream) {
  ADFWI_CHECK_ARG(dtype == ADFWI_F32 || dtype == ADFWI_F64, "dtype must be ADFWI_F32 or ADFWI_F64");
  pad::Planes p;
  const int rc = pad::planes(&p, n, src, dst, shapes, top, bottom, left, right);
  if (rc) return rc;
  int64_t cells = 1, edges = 1;
  for (int q = 0; q < n; ++q) {
    cells = std::max(cells, (int64_t)p.h[q] * p.w[q]);
    edges = std::max(edges, 2 * (int64_t)p.w[q] + 2 * (int64_t)p.h[q]);
  }
  const int64_t copy = std::min<int64_t>((cells + pad::kThreads - 1) / pad::kThreads, 4096);
  const dim3 g((unsigned)(copy + (edges + pad::kWarps - 1) / pad::kWarps + 4), n);
  auto k = dtype == ADFWI_F32 ? pad::fold<float> : pad::fold<double>;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ADFWI_LAUNCH(kAux, st, (k<<<g, pad::kThreads, 0, st>>>(p, (int)copy)));
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

}  // extern "C"
