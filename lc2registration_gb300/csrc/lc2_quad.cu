// lc2_quad.cu -- the 3D moments pass on presampled images (lc2_quad.cuh).
#include "lc2_quad.cuh"

namespace lc2 {

cudaError_t quad_launch(const FusedLaunch& L, const float* M, const int* uq, const int2* ss,
                        const PadLayout& lay) {
  const bool tall = L.tile_height == 24;
  switch (L.P.r) {
    case 1: return tall ? quad_launch_r<24, 1>(L, M, uq, ss, lay) : quad_launch_r<16, 1>(L, M, uq, ss, lay);
    case 2: return tall ? quad_launch_r<24, 2>(L, M, uq, ss, lay) : quad_launch_r<16, 2>(L, M, uq, ss, lay);
    case 3: return tall ? quad_launch_r<24, 3>(L, M, uq, ss, lay) : quad_launch_r<16, 3>(L, M, uq, ss, lay);
    case 4: return tall ? quad_launch_r<24, 4>(L, M, uq, ss, lay) : quad_launch_r<16, 4>(L, M, uq, ss, lay);
  }
  return cudaErrorInvalidValue;
}

}  // namespace lc2
