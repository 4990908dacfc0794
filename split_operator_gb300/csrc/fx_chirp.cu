// Fixed-point FFT pair of other lengths (fx_pair.cuh), FP64 states: a translation unit of its own.
#include "fx_pair.cuh"

namespace so {

cudaError_t launch_fx_chirp(int lgn, const PassParams* one, const PassParams* params, const int64_t* offsets,
                            int count, int64_t blocks, int threads, size_t smem, cudaStream_t s) {
  return launch_any<false, true>(lgn, one, params, offsets, count, blocks, threads, smem, s);
}

}  // namespace so
