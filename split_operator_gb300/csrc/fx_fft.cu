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

// 2 log2 |v| of a table's value, to 2^-9 (zero: far below every other)
template <bool FF>
__device__ __forceinline__ float log_square(longlong2 v) {
  const int e = max(max(raw_exp<FF>(v.x), raw_exp<FF>(v.y)), kMinExp<FF>);
  const bool least = e == kMinExp<FF>;
  const float x = least ? raw_rel_least<FF>(v.x) : raw_rel<FF>(v.x, e);
  const float y = least ? raw_rel_least<FF>(v.y) : raw_rel<FF>(v.y, e);
  const float s = fmaf(x, x, y * y);
  return s > 0.0f ? 2.0f * (float)(e - 1023) + log2f(s) : -1e6f;
}

// Exponents of a table's lanes (`lanes` = outer x inner lanes of n values, `inner` apart): k with the
// largest |value| 2^k in [1/2, 1] where that value is below 1/4, else 0.  A warp per contiguous lane,
// a thread per lane of strided ones.  *any: set when an exponent is not 0.
template <bool FF>
__global__ void fx_exponent_kernel(int16_t* exps, int* any, const longlong2* src, int64_t n, int64_t inner, int64_t lanes) {
  const int per = inner == 1 ? 32 : 1, sub = threadIdx.x % per;
  const int64_t step = (int64_t)gridDim.x * blockDim.x / per;
  // (whole warps stay in the loop together)
  for (int64_t l0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / per; l0 - (threadIdx.x & 31) / per < lanes; l0 += step) {
    float m = -1e6f;
    if (l0 < lanes) {
      const int64_t o = l0 / inner, i = l0 - o * inner;
      const longlong2* at = src + o * n * inner + i;
#pragma unroll 8
      for (int64_t j = sub; j < n; j += per) m = fmaxf(m, log_square<FF>(__ldg(at + j * inner)));
    }
    if (per == 32)
      for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    if (l0 < lanes && sub == 0) {
      // (a lane of zeros has no exponent)
      const int k = m < -4.0f && m > -1e5f ? min((int)floorf(-0.5f * m), 1024 - kMinExp<FF> - 1) : 0;
      if (k) *any = 1;
      exps[l0] = (int16_t)k;
    }
  }
}

// a table's values as digits of w 2^62, of w 2^(62 + k) with the exponents of its lanes
template <bool FF>
__global__ void fx_table_kernel(int4* dst, const longlong2* src, int64_t n, const int16_t* exps, int64_t lane_n,
                                int64_t inner) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const longlong2 v = src[i];
    const int e = -1 - (exps ? exps[i / (lane_n * inner) * inner + i % inner] : 0);
    i64 d[2] = {raw_to_fx<FF>(v.x, e), raw_to_fx<FF>(v.y, e)};  // x 2^(61 + k), |x| 2^k < 2
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
  while (T > least && (g.outer * m + (int64_t)V * T - 1) / ((int64_t)V * T) < 2 * sm_count()) T /= 2;
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

cudaError_t launch_fx_exponents(int16_t* exps, int* any, const void* src, int real, int64_t lanes, int64_t lane_n,
                                int64_t inner, cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(any, 0, sizeof(int), s);
  if (e != cudaSuccess) return e;
  const int64_t threads = lanes * (inner == 1 ? 32 : 1);
  const unsigned blocks = (unsigned)(threads + 255 < 256 * 1216 ? (threads + 255) / 256 : 1216);
  if (real == kRealFF)
    fx_exponent_kernel<true><<<blocks, 256, 0, s>>>(exps, any, (const longlong2*)src, lane_n, inner, lanes);
  else
    fx_exponent_kernel<false><<<blocks, 256, 0, s>>>(exps, any, (const longlong2*)src, lane_n, inner, lanes);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_fx_table(void* dst, const void* src, int real, int64_t n, const int16_t* exps, int64_t lane_n,
                            int64_t inner, cudaStream_t s) {
  const unsigned blocks = (unsigned)(n + 255 < 256 * 1216 ? (n + 255) / 256 : 1216);
  if (real == kRealFF)
    fx_table_kernel<true><<<blocks, 256, 0, s>>>((int4*)dst, (const longlong2*)src, n, exps, lane_n, inner);
  else
    fx_table_kernel<false><<<blocks, 256, 0, s>>>((int4*)dst, (const longlong2*)src, n, exps, lane_n, inner);
  count_launch();
  return cudaGetLastError();
}

}  // namespace so
