// lc2_quad.cu -- the 3D moments pass on presampled images (lc2_quad.cuh).
#include "lc2_quad.cuh"

namespace lc2 {

cudaError_t quad_launch(const FusedLaunch& L, const float* M, const int* uq, const int2* ss,
                        const PadLayout& lay, const QuadPlan& plan) {
  switch (L.P.r) {
    case 1: return quad_launch_r<1>(L, M, uq, ss, lay, plan);
    case 2: return quad_launch_r<2>(L, M, uq, ss, lay, plan);
    case 3: return quad_launch_r<3>(L, M, uq, ss, lay, plan);
    case 4: return quad_launch_r<4>(L, M, uq, ss, lay, plan);
  }
  return cudaErrorInvalidValue;
}

}  // namespace lc2
