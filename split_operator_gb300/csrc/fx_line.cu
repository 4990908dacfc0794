// Fixed-point resident 1-D propagation (fx_line.cuh): planning and the FP64 kernels.
#include "fx_line.cuh"

namespace so {

// fx_line_ff.cu
cudaError_t launch_fx_line_ff(const PassParams& p, cudaStream_t s);

bool fx_line_plan(PassParams& p, int real, const double* table_max) {
  const Geometry& g = p.g;
  const bool pow2 = (g.n & (g.n - 1)) == 0;
  if (real == kRealF32 || g.ndim != 1 || !p.resident || g.n < 16 || g.n > (pow2 ? 4096 : 2048)) return false;
  int ffts = 0, scales = 0;
  double prod = 1.0;
  for (int i = 0; i < p.nops; ++i) {
    switch (p.ops[i].kind) {
      case OP_FFT:
        // one transform pair a step
        if (++ffts > 2 || p.ops[i].dir != (ffts == 1 ? -1 : 1)) return false;
        break;
      case OP_DIAG1D: case OP_DIAGND:
        if (!(table_max[i] >= kMinTable && table_max[i] <= kMaxTable)) return false;
        prod *= table_max[i] > 1.0 ? table_max[i] : 1.0;
        break;
      // the headroom of the values holds two factors of up to 1.25: the ones after them stay below 1
      case OP_SCALE: p.ops[i].a = ++scales > 2 ? 1 : 0; break;
      case OP_NORM: case OP_COPY: case OP_LOSS: case OP_SETC: case OP_RECORD: break;
      default: return false;
    }
  }
  if (ffts != 2 || !(prod <= kMaxProduct)) return false;
  int lg = 0;
  while ((int64_t)1 << lg < (pow2 ? g.n : 2 * g.n - 1)) ++lg;
  p.fx = lg;
  p.fx_chirp = pow2 ? 0 : 1;
  return true;
}

cudaError_t launch_fx_line(int real, const PassParams& p, cudaStream_t s) {
  if (real == kRealFF) return launch_fx_line_ff(p, s);
  return p.fx_chirp ? launch_line_any<false, true>(p, s) : launch_line_any<false, false>(p, s);
}

}  // namespace so
