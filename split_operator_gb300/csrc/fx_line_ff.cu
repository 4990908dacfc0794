// Fixed-point resident 1-D propagation (fx_line.cuh) of float-float states: a translation unit
// of its own, so that the two sets of kernels compile side by side.
#include "fx_line.cuh"

namespace so {

cudaError_t launch_fx_line_ff(const PassParams& p, cudaStream_t s) {
  return p.fx_chirp ? launch_line_any<true, true>(p, s) : launch_line_any<true, false>(p, s);
}

}  // namespace so
