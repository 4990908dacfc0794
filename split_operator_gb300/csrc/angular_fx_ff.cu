// Fixed-point lane-matrix pass (angular_fx.cuh) of float-float states, a translation unit of its
// own so that the two sets of kernels compile side by side.
#include "angular_fx_launch.cuh"

namespace so {

cudaError_t launch_fx_angular_ff(int halves, int kp, int cols, const void* one, const FxTcParams* params,
                                 const uint2* owners, int64_t tiles, unsigned grid, cudaStream_t s) {
  return fx_angular_launch<true, false>(halves, kp, cols, one, params, owners, tiles, grid, s);
}

}  // namespace so
