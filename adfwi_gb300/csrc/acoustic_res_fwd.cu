// Variants of the resident forward time loop.
#include "acoustic_res.cuh"

namespace adfwi {
namespace res {
namespace {

template <int RB, int MT>
ResKernel pick(bool sums, bool glb) {
  if (sums) return glb ? time_loop<RB, MT, false, true, true> : time_loop<RB, MT, false, true, false>;
  return glb ? time_loop<RB, MT, false, false, true> : time_loop<RB, MT, false, false, false>;
}

// Self-test of the strips' waits: words of step 1 that nothing writes, in global memory for `limit_ns`, then
// in shared memory, where the raised flag ends the wait at once.
__device__ __align__(32) f2 no_words[4];
__global__ void row_wait_selftest(unsigned long long limit_ns, int* flag, float* row) {
  __shared__ __align__(32) f2 box[4];
  __shared__ __align__(16) float dst[8];
  __shared__ int dead[2];
  if (threadIdx.x != 0) return;
  for (int q = 0; q < 4; ++q) box[q] = 0ull;
  for (int q = 0; q < 8; ++q) dst[q] = 1.0f;
  dead[0] = dead[1] = 0;
  take_row<true>(no_words, 1u, dst, flag, dead, limit_ns);
  take_row<false>(box, 1u, dst + 4, flag, dead + 1, limit_ns);
  for (int q = 0; q < 8; ++q) row[q] = dead[q / 4] ? dst[q] : -1.0f;
}

}  // namespace

int row_wait_selftest(int64_t limit_ns, int* flag, float* row, cudaStream_t st) {
  ADFWI_LAUNCH(kAux, st, (row_wait_selftest<<<1, 32, 0, st>>>((unsigned long long)limit_ns, flag, row)));
  ADFWI_CUDA_TRY(cudaGetLastError());
  return kOk;
}

ResKernel forward_kernel(int rb, int mt, bool sums, bool glb) {
  if (rb == 2) return pick<2, 512>(sums, glb);
  if (rb == 3) return mt == 512 ? pick<3, 512>(sums, glb) : pick<3, 768>(sums, glb);
  if (rb == 4) return mt == 512 ? pick<4, 512>(sums, glb) : pick<4, 640>(sums, glb);
  return pick<6, 512>(sums, glb);
}

}  // namespace res
}  // namespace adfwi
