// Fixed-point lane-matrix pass (angular_fx.cuh) of float-float states with an exponent per column in the
// tables: a translation unit of its own.
#include "angular_fx_launch.cuh"

namespace so {

cudaError_t launch_fx_angular_ff_exps(int halves, int kp, int cols, const void* one, const FxTcParams* params,
                                      const uint2* owners, int64_t tiles, unsigned grid, cudaStream_t s) {
  return fx_angular_launch<true, true>(halves, kp, cols, one, params, owners, tiles, grid, s);
}

}  // namespace so
