// Multilayer perceptron for learned starting states of imaginary-time relaxation
// (no counterpart in the reference crate).  Hand-written CUDA kernels:
//   forward   Z = X W^T + b, tanh on hidden layers (BF16 weights, FP32 accumulate)
//   backward  dW = dZ^T X, db = column sums of dZ, dX = dZ W
//   Adam      on FP32 master weights, then a BF16 copy for the next forward pass
// The three products run on the tensor cores (tcgen05.mma kind::f16, accumulators in
// TMEM) with FP32 activations and gradients split into two BF16 parts.  Every product and
// sum runs in a fixed order, so training is deterministic.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <random>
#include <stdexcept>
#include <vector>

#include <cuda_bf16.h>

#include "../../include/split_operator.h"
#include "common.cuh"
#include "tc_common.cuh"

namespace so {

void set_last_error(const char* msg);

namespace {

// ---- operands
// Every product's operand is a bf16 matrix (or a hi + lo pair of them: x = bf16(x) + bf16(x -
// bf16(x)), 16 significant bits together) in one tiled layout: blocks of 128 rows x 64
// columns (16 KB), row block by row block, each block in core matrices of 8 rows x 8 columns
// (128 bytes), a row group's eight core matrices after one another.  A core matrix serves as
// K-major (rows = M or N, columns = K) and, transposed by the tensor core, as MN-major
// operand (rows = K), so activations, gradients and weights are stored once and read by every
// product they enter, by bulk TMA copies of whole blocks, half blocks or row groups.
// Rows and columns are padded to multiples of 128 with zeros.  The gradients dZ use blocks of 128
// columns (32 KB, sixteen core matrices to a row group): both of their products then read
// contiguous pieces of 16 KB and more (copies of one row group, 1 KB each, held a weight
// gradient of 64 K values x 128 x 64 at 1.4 us a chunk).
constexpr int kPadTo = 128;
constexpr uint32_t kBlockBytes = 16384, kGroupBytes = 1024;  // 128 x 64 block; 8 rows x 64 columns

int padded(int n) { return (n + kPadTo - 1) / kPadTo * kPadTo; }

// byte offset of element (r, c) of a matrix with `cols` (padded) columns
__host__ __device__ __forceinline__ size_t tiled(int64_t r, int c, int cols) {
  return ((size_t)(r >> 7) * (size_t)(cols >> 6) + (size_t)(c >> 6)) * kBlockBytes + (size_t)((r & 127) >> 3) * kGroupBytes +
         (size_t)((c & 63) >> 3) * 128 + (size_t)(r & 7) * 16 + (size_t)(c & 7) * 2;
}

__host__ __device__ __forceinline__ size_t tiled_dz(int64_t r, int c, int cols) {
  return ((size_t)(r >> 7) * (size_t)(cols >> 7) + (size_t)(c >> 7)) * (2 * kBlockBytes) +
         (size_t)((r & 127) >> 3) * (2 * kGroupBytes) + (size_t)((c & 127) >> 3) * 128 + (size_t)(r & 7) * 16 +
         (size_t)(c & 7) * 2;
}

// eight consecutive columns of one row as bf16 hi and lo parts (c a multiple of 8)
__device__ __forceinline__ void store_split8(unsigned char* hi, unsigned char* lo, size_t off, const float* x) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    uint16_t h0, l0, h1, l1;
    tc::split_bf16(x[2 * k], h0, l0);
    tc::split_bf16(x[2 * k + 1], h1, l1);
    h[k] = h0 | (uint32_t)h1 << 16;
    l[k] = l0 | (uint32_t)l1 << 16;
  }
  *reinterpret_cast<uint4*>(hi + off) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(lo + off) = make_uint4(l[0], l[1], l[2], l[3]);
}

struct Operand {
  const unsigned char *hi, *lo;  // lo: nullptr for exact bf16 values (weights)
  int cols;                      // padded columns
};

// ---- tensor-core product C[m][n] = sum_k A(m, k) B(n, k) on tiles of 128 x 64
// FORM 0, forward: A = activations, B = weights, both K-major, K in chunks of 64.
// FORM 1, dX: A = dZ, K-major; B = weights, MN-major (rows = K); K in chunks of 128.
// FORM 2, dW: A = dZ and B = activations (split), both MN-major; K (rows) in chunks of 64.
// Warp 4 streams the chunks
// through shared-memory stages by bulk copies, warp 5 issues hi hi + lo hi (+ hi lo when B
// is split; the lo lo term is 2^-16 of the result) per K step of 16 into one FP32 accumulator
// (K is not split over CTAs: the tensor core truncates as it accumulates, so the order of the
// sums is part of the result, and Adam makes a whole step of a gradient that is all rounding),
// warps 0-3 run the epilogue (thread = one row, 64 columns).  Two CTAs per SM: one's epilogue
// runs beside the other's products.  Staging FP32 operands element by element in one thread per
// row, as this kernel did before, took 4.3 ms for a training step of 1024 x (5, 256, 256, 256,
// 4096).
enum Epilogue {
  EPI_RAW,     // C in FP32 (row-major, padded)
  EPI_HIDDEN,  // bias, tanh: FP32 activation and its bf16 parts
  EPI_LOSS,    // bias, squared error: the gradient in FP32 and bf16 parts, loss partials
  EPI_OUT      // bias: FP32 output (row-major, unpadded)
};
struct GemmArgs {
  Operand a, b;
  int chunks;            // K / 64 (dX: K / 128)
  float* c;              // EPI_RAW: product; EPI_HIDDEN: activation; EPI_LOSS: gradient; EPI_OUT: output
  int rows, cols;        // valid extent of C (EPI_LOSS, EPI_OUT, EPI_HIDDEN)
  int ldc;               // padded columns of C
  const float* bias;
  unsigned char *hi, *lo;  // bf16 parts written (tiled, ldc columns)
  const float* target;     // EPI_LOSS: row-major, `cols` columns
  float scale;             // EPI_LOSS: 2 / (rows cols)
  double* loss;            // EPI_LOSS: one partial per CTA
  int* err;
};
constexpr uint64_t kGWait = 2000000000ull;  // 2 s
constexpr int kGThreads = 192;

// Shared-memory stages: two (and two CTAs per SM) in the forward products, where K is short and
// there are many tiles; dW has few tiles and hides a chunk's latency behind the chunks after it.
__host__ __device__ constexpr int gemm_stages(int form) { return form == 2 ? 4 : 2; }
__host__ __device__ constexpr uint32_t gemm_a_bytes(int form) { return form == 1 ? 2 * kBlockBytes : kBlockBytes; }
__host__ __device__ constexpr uint32_t gemm_b_bytes(int form) { return form == 1 ? kBlockBytes : kBlockBytes / 2; }
__host__ __device__ constexpr uint32_t gemm_stage_bytes(int form) {  // A hi, A lo, B (hi, lo in dW)
  return 2 * gemm_a_bytes(form) + (form == 2 ? 2u : 1u) * gemm_b_bytes(form);
}

template <int FORM, int EPI>
__global__ void __launch_bounds__(kGThreads, FORM == 0 ? 2 : 1) gemm_kernel(const __grid_constant__ GemmArgs g) {
  using namespace tc;
  constexpr uint32_t kA = gemm_a_bytes(FORM), kBb = gemm_b_bytes(FORM), kStage = gemm_stage_bytes(FORM);
  constexpr int kNs = gemm_stages(FORM), kB = FORM == 2 ? 2 : 1, kSteps = FORM == 1 ? 8 : 4;
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ __align__(8) uint64_t full[kNs], empty[kNs], done;
  __shared__ uint32_t tmem_s;
  __shared__ double wloss[4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nt = blockIdx.x, mt = blockIdx.y;
  const int c1 = g.chunks;
  if (tid == 0) {
    for (int i = 0; i < kNs; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&done, 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&tmem_s, 64);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s;
  bool ok = true;
  if (warp == 4) {
    int c = 0;
    for (; c < c1 && ok; ++c) {
      const int s = c % kNs, use = c / kNs;
      if (use > 0) ok = mbar_wait(&empty[s], (use - 1) & 1u, kGWait);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      unsigned char* st = sm + (uint32_t)s * kStage;
      if (lane == 0) mbar_expect_tx(&full[s], kStage);
      __syncwarp();
      if (lane < 2) {
        const unsigned char* src = lane ? g.a.lo : g.a.hi;
        // FORM 0: block (mt, c); 1: 128-wide block (mt, c); 2: half of the 128-wide block (c / 2, mt)
        const size_t at = FORM == 0 ? ((size_t)mt * (g.a.cols >> 6) + c) * kBlockBytes
                          : FORM == 1 ? ((size_t)mt * (g.a.cols >> 7) + c) * (2 * kBlockBytes)
                                      : ((size_t)(c >> 1) * (g.a.cols >> 7) + mt) * (2 * kBlockBytes) +
                                            (size_t)(c & 1) * kBlockBytes;
        bulk_g2s(st + (uint32_t)lane * kA, src + at, kA, &full[s]);
      } else if (lane < 2 + kB) {
        const int q = lane - 2;
        const unsigned char* src = q ? g.b.lo : g.b.hi;
        // FORM 0: half of block (nt / 2, c); 1: block (c, nt); 2: half of block (c / 2, nt)
        const size_t at = FORM == 0 ? ((size_t)(nt >> 1) * (g.b.cols >> 6) + c) * kBlockBytes + (size_t)(nt & 1) * kBb
                          : FORM == 1 ? ((size_t)c * (g.b.cols >> 6) + nt) * kBlockBytes
                                      : ((size_t)(c >> 1) * (g.b.cols >> 6) + nt) * kBlockBytes + (size_t)(c & 1) * kBb;
        bulk_g2s(st + 2 * kA + (uint32_t)q * kBb, src + at, kBb, &full[s]);
      }
    }
    if (!ok && lane == 0)  // let the copies in flight land before the CTA lets go of its shared memory
      for (int k = c < kNs ? 0 : c - kNs; k < c; ++k) mbar_poll(&full[k % kNs], (k / kNs) & 1u, kGWait);
  } else if (warp == 5) {
    const uint32_t base = smem_u32(sm), el = elect_one();
    constexpr uint32_t idesc = idesc_bf16(128, 64) | (FORM == 2 ? 1u << 15 : 0u) | (FORM != 0 ? 1u << 16 : 0u);
    // (K-group stride, M/N-group stride) of each form, and the step of 16 K values
    const uint64_t abits = FORM == 0 ? smem_desc_bits(128, 1024) : (FORM == 1 ? smem_desc_bits(128, 2048)
                                                                                : smem_desc_bits(2048, 128));
    const uint64_t bbits = FORM == 0 ? smem_desc_bits(128, 1024) : smem_desc_bits(1024, 128);
    constexpr uint32_t astep = FORM == 2 ? 4096 : 256, bstep = FORM == 0 ? 256 : 2048;
    for (int c = 0; c < c1 && ok; ++c) {
      const int s = c % kNs, use = c / kNs;
      ok = __all_sync(0xffffffffu, mbar_poll(&full[s], use & 1u, kGWait));
      if (!ok) break;
      tc_fence_after();
      const uint32_t st = base + (uint32_t)s * kStage;
      const uint64_t ah = smem_desc_at(abits, st), bh = smem_desc_at(bbits, st + 2 * kA);
#pragma unroll
      for (int k = 0; k < kSteps; ++k) {
        const uint64_t ak = ah + (uint64_t)((k * astep) >> 4), bk = bh + (uint64_t)((k * bstep) >> 4);
        mma_f16_warp(tmem, ak, bk, idesc, c > 0 || k > 0 ? 1u : 0u, el);
        mma_f16_warp(tmem, ak + (kA >> 4), bk, idesc, 1u, el);
        if constexpr (FORM == 2) mma_f16_warp(tmem, ak, bk + (kBb >> 4), idesc, 1u, el);
      }
      if (el) mma_commit(&empty[s]);
    }
    if (el) mma_commit(&done);  // (after a failed wait: everything issued so far)
    if (!ok) mbar_poll(&done, 0u, kGWait);
  } else {
    ok = mbar_wait(&done, 0u, kGWait);
    tc_fence_after();
  }
  if (!__syncthreads_and(ok)) {
    if (tid == 0) atomicExch(g.err, 1);
  } else if (warp < 4) {
    const int64_t row = (int64_t)mt * 128 + 32 * warp + lane;
    const int n0 = nt * 64;
    float v[64];
    tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16), v);
    tmem_ld32(tmem + ((uint32_t)(32 * warp) << 16) + 32u, v + 32);
    if constexpr (EPI == EPI_RAW) {
      float* dst = g.c + row * g.ldc + n0;
#pragma unroll
      for (int k = 0; k < 64; k += 4) *reinterpret_cast<float4*>(dst + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else if constexpr (EPI == EPI_OUT) {
      if (row < g.rows)
        for (int k = 0; k < 64; ++k)
          if (n0 + k < g.cols) g.c[row * g.cols + n0 + k] = v[k] + __ldg(g.bias + n0 + k);
    } else if constexpr (EPI == EPI_HIDDEN) {
      const bool live = row < g.rows;
#pragma unroll
      for (int k = 0; k < 64; ++k)
        v[k] = live && n0 + k < g.cols ? tanhf(v[k] + __ldg(g.bias + n0 + k)) : 0.0f;
#pragma unroll
      for (int k = 0; k < 64; k += 8) {
        float* dst = g.c + row * g.ldc + n0 + k;
        *reinterpret_cast<float4*>(dst) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(v[k + 4], v[k + 5], v[k + 6], v[k + 7]);
        store_split8(g.hi, g.lo, tiled(row, n0 + k, g.ldc), v + k);
      }
    } else {
      // d = y - t, its square summed in float-float (two-sum, exact products), the gradient 2 d / n
      const bool live = row < g.rows;
      const float* tr = g.target + (live ? row : 0) * g.cols + n0;
      const bool vec = (g.cols & 3) == 0;
      float s = 0.0f, e = 0.0f;
#pragma unroll
      for (int k = 0; k < 64; k += 4) {
        float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (live && vec && n0 + k < g.cols) {
          const float4 q = __ldg(reinterpret_cast<const float4*>(tr + k));
          t[0] = q.x;
          t[1] = q.y;
          t[2] = q.z;
          t[3] = q.w;
        } else if (live) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (n0 + k + u < g.cols) t[u] = __ldg(tr + k + u);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool in = live && n0 + k + u < g.cols;
          const float y = v[k + u] + (in ? __ldg(g.bias + n0 + k + u) : 0.0f);
          const float d = in ? y - t[u] : 0.0f;
          const float p = __fmul_rn(d, d), pe = __fmaf_rn(d, d, -p);
          const float q = __fadd_rn(s, p), bb = __fsub_rn(q, s);
          e = __fadd_rn(e, __fadd_rn(pe, __fadd_rn(__fsub_rn(s, __fsub_rn(q, bb)), __fsub_rn(p, bb))));
          s = q;
          v[k + u] = g.scale * d;
        }
      }
#pragma unroll
      for (int k = 0; k < 64; k += 8) {
        float* dst = g.c + row * g.ldc + n0 + k;
        *reinterpret_cast<float4*>(dst) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(v[k + 4], v[k + 5], v[k + 6], v[k + 7]);
        store_split8(g.hi, g.lo, tiled_dz(row, n0 + k, g.ldc), v + k);
      }
      double l = (double)s + (double)e;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
      if (lane == 0) wloss[warp] = l;
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (EPI == EPI_LOSS) {
    if (tid == 0) g.loss[blockIdx.y * gridDim.x + blockIdx.x] = (wloss[0] + wloss[1]) + (wloss[2] + wloss[3]);
  }
  if (warp == 0) tmem_dealloc(tmem, 64);
}

template <int FORM, int EPI>
void launch_gemm(dim3 grid, const GemmArgs& g, cudaStream_t s) {
  constexpr size_t smem = (size_t)gemm_stages(FORM) * gemm_stage_bytes(FORM);
  static bool done = false;
  auto kern = gemm_kernel<FORM, EPI>;
  if (!done) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    done = true;
  }
  kern<<<grid, kGThreads, smem, s>>>(g);
  count_launch();
}

// dZ = dX (1 - y^2) of a tanh layer, in place, and its bf16 parts; a thread: one row, 8 columns
__global__ void __launch_bounds__(256) tanh_back_kernel(float* dx, const float* act, unsigned char* hi,
                                                        unsigned char* lo, int ld) {
  const int64_t row = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 3);
  const int c = blockIdx.y * 64 + (threadIdx.x & 7) * 8;
  const int64_t at = row * ld + c;
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; k += 4) {
    const float4 q = *reinterpret_cast<const float4*>(dx + at + k);
    const float4 y = *reinterpret_cast<const float4*>(act + at + k);
    v[k] = q.x * (1.0f - y.x * y.x);
    v[k + 1] = q.y * (1.0f - y.y * y.y);
    v[k + 2] = q.z * (1.0f - y.z * y.z);
    v[k + 3] = q.w * (1.0f - y.w * y.w);
    *reinterpret_cast<float4*>(dx + at + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
  }
  store_split8(hi, lo, tiled_dz(row, c, ld), v);
}

// db[c] = sum_r dZ[r][c], rows in order: 256 threads bring 128 rows of 32 columns at a time into
// shared memory (the next ones are on their way meanwhile), one warp adds them up.  (One thread
// per column reading 64 rows ahead from global memory took 34 us for 1024 x 4096.)
__global__ void __launch_bounds__(256) colsum_kernel(const float* dz, float* db, int rows, int ld) {
  __shared__ float sh[2][128][33];
  const int c = threadIdx.x & 31, r = threadIdx.x >> 5, col = blockIdx.x * 32 + c;
  float v[16], s = 0.0f;
  auto fetch = [&](int r0) {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = r0 + r + 8 * k < rows ? dz[(int64_t)(r0 + r + 8 * k) * ld + col] : 0.0f;
  };
  fetch(0);
  for (int r0 = 0, b = 0; r0 < rows; r0 += 128, b ^= 1) {
#pragma unroll
    for (int k = 0; k < 16; ++k) sh[b][r + 8 * k][c] = v[k];
    __syncthreads();
    if (r0 + 128 < rows) fetch(r0 + 128);
    if (r == 0) {
#pragma unroll 16
      for (int k = 0; k < 128; ++k) s += sh[b][k][c];  // (the zeros past the last row change nothing)
    }
  }
  if (r == 0) db[col] = s;
}

// loss of a step: the CTAs' partials in a fixed order, over the number of outputs
__global__ void loss_kernel(const double* part, int count, double inv, double* out) {
  __shared__ double sh[256];
  double a = 0.0;
  for (int i = threadIdx.x; i < count; i += 256) a += part[i];
  sh[threadIdx.x] = a;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0] * inv;
}

// FP32 rows (row-major) into bf16 parts
__global__ void split_kernel(const float* src, int rows, int cols, unsigned char* hi, unsigned char* lo, int ld) {
  const int64_t n = (int64_t)((rows + kPadTo - 1) / kPadTo * kPadTo) * (ld / 8);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / (ld / 8);
    const int c = (int)(i - r * (ld / 8)) * 8;
    float x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = r < rows && c + k < cols ? src[r * cols + c + k] : 0.0f;
    store_split8(hi, lo, tiled(r, c, ld), x);
  }
}

// Parameters of every layer in one launch: Adam on the FP32 masters and the bf16 weights of the
// next products (ADAM), or the gradients alone in the layout of the parameters.
constexpr int kMaxLayers = 8;
struct ParamLayer {
  float *W, *b, *gW, *gb, *mW, *vW, *mb, *vb;
  unsigned char* w16;
  const float *dw, *db;
  int64_t first;  // this layer's first element of the launch
  int in, out, ldi;
};
struct ParamArgs {
  ParamLayer l[kMaxLayers];
  const int* err;  // set: a product of this step or of one before it gave up, and the parameters stay
  int* steps;      // ADAM: the steps applied so far (nullptr: not counted by this launch)
  int n;
  int64_t total;
  float lr, b1, b2, eps, c1, c2;
};
// (the moments' roundings written out: a bias or weight whose gradient is mostly rounding takes a
// full step all the same, so another contraction of the same sums trains another network)
// (stop: nothing is stored; the flag's load runs beside the others)
__device__ __forceinline__ float adam_step(float w, float g, float* m, float* v, const ParamArgs& a, int stop) {
  const float o1 = 1.f - a.b1, o2 = 1.f - a.b2;
  const float mi = __fmaf_rn(o1, g, __fmul_rn(a.b1, *m));
  const float vi = __fmaf_rn(__fmul_rn(o2, g), g, __fmul_rn(a.b2, *v));
  if (stop) return w;
  *m = mi;
  *v = vi;
  return __fsub_rn(w, __fmul_rn(a.lr, mi / a.c1) / (sqrtf(vi / a.c2) + a.eps));
}
template <bool ADAM>
__global__ void param_kernel(const __grid_constant__ ParamArgs a) {
  int stop = 0;
  if constexpr (ADAM) {
    stop = *a.err;
    if (a.steps && blockIdx.x == 0 && threadIdx.x == 0 && !stop) ++*a.steps;
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.total; i += (int64_t)gridDim.x * blockDim.x) {
    int q = 0;
    while (q + 1 < a.n && i >= a.l[q + 1].first) ++q;
    const ParamLayer& L = a.l[q];
    const int64_t k = i - L.first, nw = (int64_t)L.in * L.out;
    if (k < nw) {
      const int o = (int)(k / L.in), c = (int)(k - (int64_t)o * L.in);
      const float g = L.dw[(int64_t)o * L.ldi + c];
      if constexpr (ADAM) {
        const float w = adam_step(L.W[k], g, L.mW + k, L.vW + k, a, stop);
        L.W[k] = w;
        *reinterpret_cast<__nv_bfloat16*>(L.w16 + tiled(o, c, L.ldi)) = __float2bfloat16_rn(w);
      } else {
        L.gW[k] = g;
      }
    } else {
      const int64_t o = k - nw;
      const float g = L.db[o];
      if constexpr (ADAM)
        L.b[o] = adam_step(L.b[o], g, L.mb + o, L.vb + o, a, stop);
      else
        L.gb[o] = g;
    }
  }
}

// bf16 weights of the products from the FP32 masters
__global__ void weights_kernel(const float* W, int out, int in, unsigned char* w16, int ldi) {
  const int64_t n = (int64_t)out * in;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int o = (int)(i / in), c = (int)(i - (int64_t)o * in);
    *reinterpret_cast<__nv_bfloat16*>(w16 + tiled(o, c, ldi)) = __float2bfloat16_rn(W[i]);
  }
}

unsigned grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 4096) b = 4096;
  return (unsigned)(b < 1 ? 1 : b);
}

void check(cudaError_t e, const char* w) {
  if (e == cudaSuccess) return;
  cudaGetLastError();  // an error that the context survives ends with this call
  throw std::runtime_error(std::string(w) + ": " + cudaGetErrorString(e));
}

template <typename T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  void alloc(size_t count) {
    if (p) cudaFree(p);
    p = nullptr;
    n = count;
    check(cudaMalloc(&p, std::max<size_t>(1, count) * sizeof(T)), "cudaMalloc");
    check(cudaMemset(p, 0, std::max<size_t>(1, count) * sizeof(T)), "cudaMemset");
  }
  ~DBuf() {
    if (p) cudaFree(p);
  }
};

}  // namespace

struct Mlp {
  std::vector<int> w;  // widths: input, hidden..., output
  struct Layer {
    int in, out, ldi, ldo;  // widths and their padded sizes
    DBuf<float> W, b, gW, gb, mW, vW, mb, vb;
    DBuf<unsigned char> w16;  // bf16 weights, tiled [out][in]
    // per batch capacity
    DBuf<float> act;                      // hidden layers: FP32 activation [batch][ldo]
    DBuf<unsigned char> ahi, alo;         // ... and its bf16 parts
    DBuf<unsigned char> dhi, dlo;         // bf16 parts of dZ [batch][ldo]
    DBuf<float> dz;                       // dZ in FP32
    DBuf<float> dw, db;
  };
  std::vector<std::unique_ptr<Layer>> layers;
  DBuf<float> x, target, y;
  DBuf<unsigned char> xhi, xlo;
  DBuf<double> loss_part, losses;
  DBuf<int> err;  // [0] set by a tensor-core product whose bounded wait gave up; [1] Adam steps applied
  int cap = 0, loss_cap = 0;
  int64_t t = 0;  // Adam step
  // weight gradients and bias gradients run beside the chain of dX
  cudaStream_t s = nullptr, side = nullptr, side2 = nullptr;
  cudaEvent_t ready = nullptr, joined = nullptr, joined2 = nullptr;
  Mlp() = default;
  Mlp(const Mlp&) = delete;
  void open() {
    check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream");
    check(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking), "stream");
    check(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming), "event");
    check(cudaEventCreateWithFlags(&joined, cudaEventDisableTiming), "event");
    check(cudaStreamCreateWithFlags(&side2, cudaStreamNonBlocking), "stream");
    check(cudaEventCreateWithFlags(&joined2, cudaEventDisableTiming), "event");
  }
  ~Mlp() {
    for (cudaStream_t q : {s, side, side2})
      if (q) {
        cudaStreamSynchronize(q);
        cudaStreamDestroy(q);
      }
    for (cudaEvent_t e : {ready, joined, joined2})
      if (e) cudaEventDestroy(e);
  }

  void ensure(int batch) {
    if (batch <= cap) return;
    cap = 0;  // until every buffer has its new size
    const size_t bp = (size_t)padded(batch);
    x.alloc((size_t)batch * w[0]);
    target.alloc((size_t)batch * w.back());
    y.alloc((size_t)batch * w.back());
    xhi.alloc(2 * bp * padded(w[0]));
    xlo.alloc(2 * bp * padded(w[0]));
    for (size_t l = 0; l < layers.size(); ++l) {
      Layer& L = *layers[l];
      const size_t e = bp * L.ldo;
      if (l + 1 < layers.size()) {
        L.act.alloc(e);
        L.ahi.alloc(2 * e);
        L.alo.alloc(2 * e);
      }
      L.dhi.alloc(2 * e);
      L.dlo.alloc(2 * e);
      L.dz.alloc(e);
      L.dw.alloc((size_t)L.ldo * L.ldi);
      L.db.alloc(L.ldo);
    }
    loss_part.alloc((bp / 128) * (layers.back()->ldo / 64));
    if (!err.p) err.alloc(2);
    check(cudaStreamSynchronize(nullptr), "sync");  // the clears run on the default stream
    cap = batch;
  }

  void need_losses(int n) {
    if (n <= loss_cap) return;
    loss_cap = 0;
    losses.alloc(n);
    check(cudaStreamSynchronize(nullptr), "sync");
    loss_cap = n;
  }

  // a bounded wait inside a tensor-core product gave up: report it (and clear the flag).  No step took
  // part of it (param_kernel), so the optimiser is where the steps applied have brought it.
  void check_err() {
    int e[2] = {0, 0};
    check(cudaGetLastError(), "launch");
    check(cudaMemcpyAsync(e, err.p, sizeof(e), cudaMemcpyDeviceToHost, s), "copy");
    check(cudaStreamSynchronize(s), "sync");
    if (e[0]) {
      t = e[1];
      check(cudaMemsetAsync(err.p, 0, sizeof(int), s), "memset");
      throw std::runtime_error("a tensor-core product's bounded wait gave up");
    }
  }

  void refresh_bf16() {
    for (auto& L : layers) {
      const int64_t n = (int64_t)L->in * L->out;
      weights_kernel<<<grid_for(n), 256, 0, s>>>(L->W.p, L->out, L->in, L->w16.p, L->ldi);
      count_launch();
    }
  }

  // bf16 parts of the inputs (once per call: they serve every step)
  void load_inputs(int batch) {
    split_kernel<<<grid_for((int64_t)padded(batch) * padded(w[0]) / 8), 256, 0, s>>>(x.p, batch, w[0], xhi.p, xlo.p,
                                                                                     padded(w[0]));
    count_launch();
  }

  Operand input_of(size_t l) const {
    if (l == 0) return {xhi.p, xlo.p, padded(w[0])};
    return {layers[l - 1]->ahi.p, layers[l - 1]->alo.p, layers[l - 1]->ldo};
  }

  // train: the output layer's epilogue turns into the loss and its gradient
  void forward(int batch, bool train) {
    const int bp = padded(batch);
    for (size_t l = 0; l < layers.size(); ++l) {
      Layer& L = *layers[l];
      // Z[b][o] = sum_i X[b][i] W[o][i]
      GemmArgs g{};
      g.a = input_of(l);
      g.b = Operand{L.w16.p, nullptr, L.ldi};
      g.chunks = L.ldi / 64;
      g.rows = batch;
      g.cols = L.out;
      g.ldc = L.ldo;
      g.bias = L.b.p;
      g.err = err.p;
      const dim3 grid(L.ldo / 64, bp / 128);
      if (l + 1 < layers.size()) {
        g.c = L.act.p;
        g.hi = L.ahi.p;
        g.lo = L.alo.p;
        launch_gemm<0, EPI_HIDDEN>(grid, g, s);
      } else if (train) {
        g.hi = L.dhi.p;
        g.lo = L.dlo.p;
        g.target = target.p;
        g.scale = 2.0f / (float)((int64_t)batch * L.out);
        g.loss = loss_part.p;
        g.c = L.dz.p;
        launch_gemm<0, EPI_LOSS>(grid, g, s);
      } else {
        g.c = y.p;
        launch_gemm<0, EPI_OUT>(grid, g, s);
      }
    }
  }

  // the step's loss into *out (device), weight and bias gradients into the layers' partials
  void backward(int batch, double* out) {
    const int bp = padded(batch), nl = (int)layers.size();
    const int tiles = (bp / 128) * (layers.back()->ldo / 64);
    for (int l = nl - 1; l >= 0; --l) {
      Layer& L = *layers[l];
      // dW[o][i] = sum_b dZ[b][o] X[b][i]
      GemmArgs g{};
      g.a = Operand{L.dhi.p, L.dlo.p, L.ldo};
      g.b = input_of(l);
      g.chunks = bp / 64;
      g.c = L.dw.p;
      g.ldc = L.ldi;
      g.err = err.p;
      // (beside the chain of the gradient handed down)
      check(cudaEventRecord(ready, s), "event");
      check(cudaStreamWaitEvent(side, ready, 0), "event");
      check(cudaStreamWaitEvent(side2, ready, 0), "event");
      if (l == nl - 1) {
        loss_kernel<<<1, 256, 0, side2>>>(loss_part.p, tiles, 1.0 / ((double)batch * w.back()), out);
        count_launch();
      }
      launch_gemm<2, EPI_RAW>(dim3(L.ldi / 64, L.ldo / 128), g, side);
      colsum_kernel<<<L.ldo / 32, 256, 0, side2>>>(L.dz.p, L.db.p, batch, L.ldo);
      count_launch();
      if (l == 0) continue;
      // dX[b][i] = sum_o dZ[b][o] W[o][i], then the layer below's dZ
      GemmArgs d{};
      d.a = Operand{L.dhi.p, L.dlo.p, L.ldo};
      d.b = Operand{L.w16.p, nullptr, L.ldi};
      d.chunks = L.ldo / 128;
      Layer& D = *layers[l - 1];
      d.c = D.dz.p;
      d.ldc = L.ldi;
      d.err = err.p;
      launch_gemm<1, EPI_RAW>(dim3(L.ldi / 64, bp / 128), d, s);
      tanh_back_kernel<<<dim3(bp / 32, D.ldo / 64), 256, 0, s>>>(D.dz.p, D.act.p, D.dhi.p, D.dlo.p, D.ldo);
      count_launch();
    }
    check(cudaEventRecord(joined, side), "event");
    check(cudaStreamWaitEvent(s, joined, 0), "event");
    check(cudaEventRecord(joined2, side2), "event");
    check(cudaStreamWaitEvent(s, joined2, 0), "event");
  }

  // the parameter kernel over every layer (kMaxLayers to a launch)
  template <bool ADAM>
  void params(int batch, ParamArgs a) {
    const int nl = (int)layers.size();
    for (int first = 0; first < nl; first += kMaxLayers) {
      a.n = std::min(kMaxLayers, nl - first);
      a.total = 0;
      for (int q = 0; q < a.n; ++q) {
        Layer& L = *layers[first + q];
        a.l[q] = ParamLayer{L.W.p, L.b.p, L.gW.p, L.gb.p, L.mW.p, L.vW.p, L.mb.p, L.vb.p, L.w16.p, L.dw.p, L.db.p,
                            a.total, L.in, L.out, L.ldi};
        a.total += (int64_t)L.in * L.out + L.out;
      }
      a.err = err.p;
      a.steps = first == 0 ? err.p + 1 : nullptr;
      param_kernel<ADAM><<<grid_for(a.total), 256, 0, s>>>(a);
      count_launch();
    }
  }

  void gradients(int batch) { params<false>(batch, ParamArgs{}); }

  void adam(int batch, float lr) {
    ++t;
    ParamArgs a{};
    a.lr = lr;
    a.b1 = 0.9f;
    a.b2 = 0.999f;
    a.eps = 1e-8f;
    a.c1 = 1.f - std::pow(a.b1, (float)t);
    a.c2 = 1.f - std::pow(a.b2, (float)t);
    params<true>(batch, a);
  }
};

}  // namespace so

struct so_mlp_t {
  so::Mlp m;
};

namespace {
template <class F>
int mlp_guard(F&& f) {
  try {
    f();
    return SO_OK;
  } catch (const std::exception& e) {
    so::set_last_error(e.what());
    return SO_ERR_CUDA;
  }
}
size_t nparams(const so::Mlp& m) {
  size_t n = 0;
  for (auto& L : m.layers) n += (size_t)L->in * L->out + L->out;
  return n;
}
}  // namespace

extern "C" {

int so_mlp_new(const int* widths, size_t count, uint64_t seed, so_mlp* out) {
  if (!widths || count < 2 || !out) {
    so::set_last_error("so_mlp_new: need at least an input and an output width");
    return SO_ERR_INVALID;
  }
  return mlp_guard([&] {
    auto h = std::make_unique<so_mlp_t>();
    so::Mlp& m = h->m;
    m.open();
    m.w.assign(widths, widths + count);
    std::mt19937_64 rng(seed);
    for (size_t l = 0; l + 1 < count; ++l) {
      auto L = std::make_unique<so::Mlp::Layer>();
      L->in = widths[l];
      L->out = widths[l + 1];
      const size_t nw = (size_t)L->in * L->out;
      for (auto* b : {&L->W, &L->gW, &L->mW, &L->vW}) b->alloc(nw);
      for (auto* b : {&L->b, &L->gb, &L->mb, &L->vb}) b->alloc(L->out);
      L->ldi = so::padded(L->in);
      L->ldo = so::padded(L->out);
      L->w16.alloc(2 * (size_t)L->ldi * L->ldo);  // zeros in the padding
      so::check(cudaStreamSynchronize(nullptr), "sync");  // the clears run on the default stream
      // Glorot-uniform weights, zero biases
      std::uniform_real_distribution<float> u(-1.f, 1.f);
      const float lim = std::sqrt(6.f / (float)(L->in + L->out));
      std::vector<float> w(nw);
      for (float& v : w) v = lim * u(rng);
      so::check(cudaMemcpyAsync(L->W.p, w.data(), nw * sizeof(float), cudaMemcpyHostToDevice, m.s), "copy");
      so::check(cudaStreamSynchronize(m.s), "sync");  // (w goes out of scope)
      m.layers.push_back(std::move(L));
    }
    m.refresh_bf16();
    so::check(cudaDeviceSynchronize(), "sync");
    *out = h.release();
  });
}

int so_mlp_num_params(so_mlp m, size_t* out) {
  if (!m || !out) return SO_ERR_INVALID;
  *out = nparams(m->m);
  return SO_OK;
}

// FP32 master parameters, layer by layer: W (out x in, row-major) then b
int so_mlp_get_params(so_mlp h, float* out) {
  return mlp_guard([&] {
    size_t off = 0;
    for (auto& L : h->m.layers) {
      const size_t nw = (size_t)L->in * L->out;
      so::check(cudaMemcpy(out + off, L->W.p, nw * 4, cudaMemcpyDeviceToHost), "copy");
      off += nw;
      so::check(cudaMemcpy(out + off, L->b.p, L->out * 4, cudaMemcpyDeviceToHost), "copy");
      off += L->out;
    }
  });
}

int so_mlp_set_params(so_mlp h, const float* in) {
  return mlp_guard([&] {
    size_t off = 0;
    for (auto& L : h->m.layers) {
      const size_t nw = (size_t)L->in * L->out;
      so::check(cudaMemcpyAsync(L->W.p, in + off, nw * 4, cudaMemcpyHostToDevice, h->m.s), "copy");
      off += nw;
      so::check(cudaMemcpyAsync(L->b.p, in + off, L->out * 4, cudaMemcpyHostToDevice, h->m.s), "copy");
      off += L->out;
    }
    h->m.refresh_bf16();
    so::check(cudaDeviceSynchronize(), "sync");
  });
}

// y = network(x) for `batch` rows (host arrays, FP32)
int so_mlp_forward(so_mlp h, const float* x, size_t batch, float* y) {
  return mlp_guard([&] {
    so::Mlp& m = h->m;
    m.ensure((int)batch);
    so::check(cudaMemcpyAsync(m.x.p, x, batch * m.w[0] * 4, cudaMemcpyHostToDevice, m.s), "copy");
    m.load_inputs((int)batch);
    m.forward((int)batch, false);
    m.check_err();
    so::check(cudaMemcpy(y, m.y.p, batch * m.w.back() * 4, cudaMemcpyDeviceToHost), "copy");
  });
}

// Loss (mean squared error) and parameter gradients (same order as so_mlp_get_params)
int so_mlp_gradients(so_mlp h, const float* x, const float* target, size_t batch, double* loss, float* grads) {
  return mlp_guard([&] {
    so::Mlp& m = h->m;
    m.ensure((int)batch);
    so::check(cudaMemcpyAsync(m.x.p, x, batch * m.w[0] * 4, cudaMemcpyHostToDevice, m.s), "copy");
    so::check(cudaMemcpyAsync(m.target.p, target, batch * m.w.back() * 4, cudaMemcpyHostToDevice, m.s), "copy");
    m.load_inputs((int)batch);
    m.need_losses(1);
    m.forward((int)batch, true);
    m.backward((int)batch, m.losses.p);
    m.gradients((int)batch);
    so::check(cudaMemcpyAsync(loss, m.losses.p, sizeof(double), cudaMemcpyDeviceToHost, m.s), "copy");
    m.check_err();
    size_t off = 0;
    for (auto& L : m.layers) {
      const size_t nw = (size_t)L->in * L->out;
      so::check(cudaMemcpy(grads + off, L->gW.p, nw * 4, cudaMemcpyDeviceToHost), "copy");
      off += nw;
      so::check(cudaMemcpy(grads + off, L->gb.p, L->out * 4, cudaMemcpyDeviceToHost), "copy");
      off += L->out;
    }
  });
}

// `steps` full-batch Adam steps on (x, target); losses[i] = loss before step i
int so_mlp_train(so_mlp h, const float* x, const float* target, size_t batch, size_t steps, float lr,
                 double* losses) {
  return mlp_guard([&] {
    so::Mlp& m = h->m;
    m.ensure((int)batch);
    so::check(cudaMemcpyAsync(m.x.p, x, batch * m.w[0] * 4, cudaMemcpyHostToDevice, m.s), "copy");
    so::check(cudaMemcpyAsync(m.target.p, target, batch * m.w.back() * 4, cudaMemcpyHostToDevice, m.s), "copy");
    m.load_inputs((int)batch);
    // the losses stay on the device until a run of steps is queued: no step waits for the host
    constexpr size_t kRun = 1024;
    m.need_losses((int)std::min(steps, kRun));
    for (size_t i = 0; i < steps; i += kRun) {
      const size_t n = std::min(steps - i, kRun);
      for (size_t k = 0; k < n; ++k) {
        m.forward((int)batch, true);
        m.backward((int)batch, m.losses.p + k);
        m.adam((int)batch, lr);
      }
      if (losses)
        so::check(cudaMemcpyAsync(losses + i, m.losses.p, n * sizeof(double), cudaMemcpyDeviceToHost, m.s), "copy");
      m.check_err();
    }
  });
}

// Self-test: the next product's error flag is set as if its bounded wait had given up.
int so_selftest_mlp_give_up(so_mlp h) {
  if (!h) return SO_ERR_INVALID;
  return mlp_guard([&] {
    h->m.ensure(1);
    const int one = 1;
    so::check(cudaMemcpyAsync(h->m.err.p, &one, sizeof(int), cudaMemcpyHostToDevice, h->m.s), "copy");
    so::check(cudaStreamSynchronize(h->m.s), "sync");
  });
}

void so_mlp_free(so_mlp h) { delete h; }

}  // extern "C"
