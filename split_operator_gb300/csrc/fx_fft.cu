// Fixed-point FFT pair (fx_pair.cuh): planning, the FP64 kernels and the factor tables.
#include "fx_pair.cuh"

namespace so {

// the other kernels, each set in a translation unit of its own (they compile side by side)
cudaError_t launch_fx_pair_ff(int lgn, const PassParams* one, const PassParams* params, const int64_t* offsets,
                              int count, int64_t blocks, int threads, size_t smem, cudaStream_t s);
cudaError_t launch_fx_chirp(int lgn, const PassParams* one, const PassParams* params, const int64_t* offsets,
                            int count, int64_t blocks, int threads, size_t smem, cudaStream_t s);
cudaError_t launch_fx_chirp_ff(int lgn, const PassParams* one, const PassParams* params, const int64_t* offsets,
                               int count, int64_t blocks, int threads, size_t smem, cudaStream_t s);

namespace {

// a table's values as digits of w 2^62
template <bool FF>
__global__ void fx_table_kernel(int4* dst, const longlong2* src, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const longlong2 v = src[i];
    i64 d[2] = {raw_to_fx<FF>(v.x, -1), raw_to_fx<FF>(v.y, -1)};  // x 2^61, |x| < 2
    int4 o;
    int* w = &o.x;
    for (int k = 0; k < 2; ++k) {
      d[k] *= 2;
      if ((int)d[k] == (int)0x80000000) d[k] += 2;  // digits stay negatable
      const dig g = split(d[k]);
      w[2 * k] = g.l;
      w[2 * k + 1] = g.h;
    }
    dst[i] = o;
  }
}

}  // namespace

bool fx_pair_plan(PassParams& p, int real, const double* table_max) {
  Geometry& g = p.g;
  // powers of two from 16 to 8192 points; other lengths through transforms of M >= 2 n - 1 points
  const bool pow2 = (g.n & (g.n - 1)) == 0;
  if (real == kRealF32 || g.inner != 1 || g.n < 16 || g.n > (pow2 ? 8192 : 4096)) return false;
  if (p.nops < 2 || p.ops[0].kind != OP_FFT || p.ops[0].dir != -1) return false;
  int ffts = 0;
  double prod = 1.0;
  for (int i = 0; i < p.nops; ++i) {
    const DevOp& op = p.ops[i];
    if (op.kind == OP_FFT) {
      if (++ffts == 2 && op.dir != 1) return false;
    } else if (op.kind == OP_DIAGND || (op.kind == OP_DIAG1D && op.axis == g.sweep_axis)) {
      // (a table that is not finite has the maximum infinity)
      if (!(table_max[i] >= kMinTable && table_max[i] <= kMaxTable)) return false;
      prod *= table_max[i] > 1.0 ? table_max[i] : 1.0;
    } else {
      return false;
    }
  }
  if (ffts != 2 || !(prod <= kMaxProduct)) return false;
  int lg = 0;
  while ((int64_t)1 << lg < (pow2 ? g.n : 2 * g.n - 1)) ++lg;
  const int64_t m = (int64_t)1 << lg;
  // 512 threads a CTA, fewer while the tiles do not fill the SMs twice
  const int V = pair_vals(lg);
  int T = kPairThreads;
  const int least = m / V > 32 ? (int)(m / V) : 32;
  while (T > least && (g.outer * m + (int64_t)V * T - 1) / ((int64_t)V * T) < 304) T /= 2;
  const int64_t L = (int64_t)V * T / m;
  g.lanes_per_tile = (int32_t)L;
  g.tiles_per_outer = 1;
  g.tiles = (g.outer + L - 1) / L;
  g.vals = V;
  g.lane_stride = (int32_t)(m + m / (V == 16 ? 16 : 8) + 1);
  p.fx_chirp = pow2 ? 0 : 1;
  p.fused = 1;
  p.radix = V;
  p.fx = lg;
  return true;
}

cudaError_t launch_fx_pair(int real, bool chirp, int lgn, const PassParams* one, const PassParams* params_dev,
                           const int64_t* offsets_dev, int count, int64_t blocks, int threads, size_t smem,
                           cudaStream_t s) {
  if (chirp)
    return real == kRealFF ? launch_fx_chirp_ff(lgn, one, params_dev, offsets_dev, count, blocks, threads, smem, s)
                           : launch_fx_chirp(lgn, one, params_dev, offsets_dev, count, blocks, threads, smem, s);
  return real == kRealFF ? launch_fx_pair_ff(lgn, one, params_dev, offsets_dev, count, blocks, threads, smem, s)
                         : launch_any<false, false>(lgn, one, params_dev, offsets_dev, count, blocks, threads, smem, s);
}

cudaError_t launch_fx_table(void* dst, const void* src, int real, int64_t n, cudaStream_t s) {
  const unsigned blocks = (unsigned)(n + 255 < 256 * 1216 ? (n + 255) / 256 : 1216);
  if (real == kRealFF)
    fx_table_kernel<true><<<blocks, 256, 0, s>>>((int4*)dst, (const longlong2*)src, n);
  else
    fx_table_kernel<false><<<blocks, 256, 0, s>>>((int4*)dst, (const longlong2*)src, n);
  count_launch();
  return cudaGetLastError();
}

}  // namespace so
