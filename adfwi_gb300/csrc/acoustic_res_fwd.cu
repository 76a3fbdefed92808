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

}  // namespace

ResKernel forward_kernel(int rb, int mt, bool sums, bool glb) {
  if (rb == 2) return pick<2, 512>(sums, glb);
  if (rb == 3) return mt == 512 ? pick<3, 512>(sums, glb) : pick<3, 768>(sums, glb);
  if (rb == 4) return mt == 512 ? pick<4, 512>(sums, glb) : pick<4, 640>(sums, glb);
  return pick<6, 512>(sums, glb);
}

}  // namespace res
}  // namespace adfwi
