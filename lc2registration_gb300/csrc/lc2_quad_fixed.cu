// lc2_quad_fixed.cu -- the 3D moments pass of a resampled ultrasound
// (lc2_quad_fixed.cuh).
#include "lc2_quad_fixed.cuh"

namespace lc2 {

cudaError_t fixed_quad_launch(const FixedLaunch& L, const int* q, const PadLayout& lay) {
  const bool tall = L.tile_height == 24;
  switch (L.P.r) {
    case 1: return tall ? fixed_quad_launch_r<24, 1>(L, q, lay) : fixed_quad_launch_r<16, 1>(L, q, lay);
    case 2: return tall ? fixed_quad_launch_r<24, 2>(L, q, lay) : fixed_quad_launch_r<16, 2>(L, q, lay);
    case 3: return tall ? fixed_quad_launch_r<24, 3>(L, q, lay) : fixed_quad_launch_r<16, 3>(L, q, lay);
    case 4: return tall ? fixed_quad_launch_r<24, 4>(L, q, lay) : fixed_quad_launch_r<16, 4>(L, q, lay);
  }
  return cudaErrorInvalidValue;
}

}  // namespace lc2
