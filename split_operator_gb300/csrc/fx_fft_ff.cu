// Fixed-point FFT pair (fx_pair.cuh) of float-float states: a translation unit of its own, so
// that the two sets of kernels compile side by side.
#include "fx_pair.cuh"

namespace so {

cudaError_t launch_fx_pair_ff(int lgn, const PassParams* one, const PassParams* params, const int64_t* offsets,
                              int count, int64_t blocks, int threads, size_t smem, cudaStream_t s) {
  return launch_any<true, false>(lgn, one, params, offsets, count, blocks, threads, smem, s);
}

}  // namespace so
