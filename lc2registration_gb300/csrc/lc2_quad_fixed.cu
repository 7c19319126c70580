// lc2_quad_fixed.cu -- the 3D moments pass of a resampled ultrasound
// (lc2_quad_fixed.cuh).
#include "lc2_quad_fixed.cuh"

namespace lc2 {

cudaError_t fixed_quad_launch(const FixedLaunch& L, const int* q, const PadLayout& lay,
                              const QuadPlan& plan) {
  switch (L.P.r) {
    case 1: return fixed_quad_launch_r<1>(L, q, lay, plan);
    case 2: return fixed_quad_launch_r<2>(L, q, lay, plan);
    case 3: return fixed_quad_launch_r<3>(L, q, lay, plan);
    case 4: return fixed_quad_launch_r<4>(L, q, lay, plan);
  }
  return cudaErrorInvalidValue;
}

}  // namespace lc2
