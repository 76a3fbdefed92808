// Variants of the resident adjoint time loop.
#include "acoustic_res.cuh"

namespace adfwi {
namespace res {
namespace {

template <int RB, int MT>
ResKernel pick(bool glb) {
  return glb ? time_loop<RB, MT, true, true, true> : time_loop<RB, MT, true, true, false>;
}

}  // namespace

ResKernel adjoint_kernel(int rb, int mt, bool glb) {
  if (rb == 3) return mt == 512 ? pick<3, 512>(glb) : pick<3, 768>(glb);
  if (rb == 4) return mt == 512 ? pick<4, 512>(glb) : pick<4, 640>(glb);
  return mt == 384 ? pick<6, 384>(glb) : pick<6, 512>(glb);
}

}  // namespace res
}  // namespace adfwi
