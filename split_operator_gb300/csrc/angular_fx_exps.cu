// Fixed-point lane-matrix pass (angular_fx.cuh) of FP64 states with an exponent per column in the
// tables: a translation unit of its own.
#include "angular_fx_launch.cuh"

namespace so {

cudaError_t launch_fx_angular_exps(int halves, int kp, int cols, const void* one, const FxTcParams* params,
                                   const uint2* owners, int64_t tiles, unsigned grid, cudaStream_t s) {
  return fx_angular_launch<false, true>(halves, kp, cols, one, params, owners, tiles, grid, s);
}

}  // namespace so
