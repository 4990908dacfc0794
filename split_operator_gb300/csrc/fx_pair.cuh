// The radial FFT pair of the 2-D step, [FFT] [point-wise]* [FFT^-1] [point-wise]*, on
// contiguous power-of-two lanes of FP64 or float-float states, in 64-bit fixed point (fx.cuh).
//
// The FP64 form of this pass was bound by the FP64 pipe: about 90 FP64 operations per point
// of a 4096-point lane at ~1.7 per clock and SM.  Here the butterflies are integer additions
// and the products three 32 x 32 + 64 multiply-adds.  A thread holds 8 values: radix-8 stages in
// place in one shared buffer, the first stage from global memory, the point-wise ops between the
// transforms in registers, the second transform in reversed radix order so that its first stage
// needs no shared memory, the last stage to global memory.  The unitary scaling sits in the
// products and in the exponent the lane leaves with.
//
// What bounds it is fetching instructions and latency, not the pipes: the code is one loop over
// the stages, one copy for both transforms (rolled_transform).  Unrolled, with 16 values per
// thread, a lane ran 10,400 instructions in a row on 8 warps and 61 % of the stalls were for
// instructions.  us per pass before / now: 128 lanes of 4096 points in float-float 37.1 / 29.1,
// 64 of 2048 in FP64 28.9 / 18.3, 256 of 256 22.9 / 12.6, 45 of 1000 (through 2048) 53.7 / 28.7.
#pragma once
#include "fx_stage.cuh"
#include "overlap.cuh"

namespace so {

using namespace fx;

namespace {

// values per thread: 8, and 16 where that would take more than 512 threads for a lane
__host__ __device__ constexpr int pair_vals(int lgn) { return lgn >= 13 ? 16 : 8; }
constexpr int kPairThreads = 512;  // most threads of a CTA

// point-wise ops [ob, oe) on the outputs of a last stage of radix RS (span P = n / RS): value
// j RS + q sits at lane b >> lg P, point k + q P
template <int LGN, int KV, int RS>
__device__ __forceinline__ void pointwise(cx (&v)[KV], const PassParams& pp, int ob, int oe, int64_t lane0, int nl) {
  constexpr int kN = 1 << LGN, kP = kN / RS, kLgP = LGN - lg2(RS);
  const int t = threadIdx.x, T = blockDim.x;
#pragma unroll 1
  for (int oi = ob; oi < oe; ++oi) {
    const DevOp& op = pp.ops[oi];
    const bool nd = op.kind == OP_DIAGND;
    const int4* tab = reinterpret_cast<const int4*>(op.ptr) + (nd ? lane0 * kN : 0);
#pragma unroll
    for (int j = 0; j < KV / RS; ++j) {
      const int b = t + j * T, l = b >> kLgP, k = b & (kP - 1);
      if (!nd || l < nl) {
        const int4* tr = tab + (nd ? l * kN : 0) + k;
        int4 w[RS];
#pragma unroll
        for (int q = 0; q < RS; ++q) w[q] = __ldg(tr + q * kP);
#pragma unroll
        for (int q = 0; q < RS; ++q) v[j * RS + q] = cmul<0>(v[j * RS + q], w[q]);
      }
    }
  }
}

// exponent of a lane's factors together (out of line: few passes have them)
__device__ __noinline__ int table_exponent(const PassParams& pp, int64_t lane) {
  int k = 0;
  for (int oi = 0; oi < pp.nops; ++oi)
    if (pp.ops[oi].kind == OP_DIAGND && pp.ops[oi].exps) k += __ldg(pp.ops[oi].exps + lane);
  return k;
}

template <int LGN, bool FF>
__device__ __forceinline__ void fx_pair_tile(const PassParams& pp, int64_t tile) {
  constexpr int kV = pair_vals(LGN);
  using Sh = Shape<LGN, kV>;
  constexpr int kN = Sh::kN, kNb = kN / kV, kLgNb = LGN - Sh::kLgV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ NormPart part[16];
  cx* buf = reinterpret_cast<cx*>(smem_raw);
  const Geometry& g = pp.g;
  const int64_t lane0 = tile * g.lanes_per_tile;
  const int64_t rem = g.outer - lane0;
  const int nl = rem < g.lanes_per_tile ? (int)rem : g.lanes_per_tile;
  longlong2* psi = reinterpret_cast<longlong2*>(pp.psi) + lane0 * kN;
  const int4* tw = reinterpret_cast<const int4*>(pp.twiddle);
  const int t = threadIdx.x;
  cx v[kV];
  // the first stage's inputs straight from the lanes (points i + r n / kV; missing lanes: 0)
  const int l0 = t >> kLgNb, i0 = t & (kNb - 1);
  const bool ok0 = l0 < nl;
  {
    const longlong2* src = psi + l0 * kN + i0;
#pragma unroll
    for (int r = 0; r < kV; ++r) {
      const longlong2 x = ok0 ? src[r * kNb] : longlong2{0, 0};
      v[r] = {x.x, x.y};
    }
  }
  const int e = lane_exponent<LGN, kV, FF>(v, part);
#pragma unroll
  for (int r = 0; r < kV; ++r) {
    v[r].x = e == kNonFinite || e == kZero ? 0 : raw_to_fx<FF>(v[r].x, e);
    v[r].y = e == kNonFinite || e == kZero ? 0 : raw_to_fx<FF>(v[r].y, e);
  }
  int f1 = 1;
  while (f1 < pp.nops && pp.ops[f1].kind != OP_FFT) ++f1;
  // one copy of the code for both transforms: the inverse one is conjugated
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    if (half) conjugate(v);
    rolled_transform<LGN, kV>(v, buf, tw, half != 0);
    if (half) {
      conjugate(v);
    } else if (Sh::kMid > 0) {
#pragma unroll
      for (int r = 0; r < kV; ++r) v[r] = shift_down<Sh::kMid>(v[r]);
    }
    const int ob = half ? f1 + 1 : 1, oe = half ? pp.nops : f1;
    if (Sh::kRl == kV || half)
      pointwise<LGN, kV, kV>(v, pp, ob, oe, lane0, nl);
    else
      pointwise<LGN, kV, Sh::kRl>(v, pp, ob, oe, lane0, nl);
  }
  // the last stage's outputs have the first stage's layout: the same lane, points k + q n / kV
  if (ok0) {
    longlong2* dst = psi + l0 * kN + i0;
    const int x = e - Sh::kOut - (pp.fx_exps ? table_exponent(pp, lane0 + l0) : 0);
    auto store = [&](auto low) {
#pragma unroll
      for (int q = 0; q < kV; ++q) {
        longlong2 o{fx_to_raw<FF, decltype(low)::value>(v[q].x, x), fx_to_raw<FF, decltype(low)::value>(v[q].y, x)};
        if (e == kNonFinite) o = {raw_nan<FF>(), raw_nan<FF>()};
        dst[q * kNb] = o;
      }
    };
    by_exponent<FF>(x, store);
  }
}

// Lanes of other lengths, n <= M / 2 points with M = 2^LGM, by Bluestein's algorithm (L. Bluestein,
// "A linear filtering approach to the computation of the discrete Fourier transform", IEEE
// Trans. Audio Electroacoust. 18, 1970): with w_j = exp(-i pi j^2 / n), the transform of x is
// w_k times the convolution of x_j w_j with conj w, a pair of transforms of M points around a
// product with the filter's spectrum G.  The closing w_k of the forward transform and the
// opening conj w_k of the inverse one cancel in the pair, and the inverse filter is conj G.
// (A direct sum in FP64 took 5.8 ms for 45 lanes of 1000 points.)
// pp.aux: the chirp w (n entries), then G 2^-pp.fx_g (M entries, natural order, magnitudes <= 1).
template <int LGM, bool FF>
__device__ __forceinline__ void fx_chirp_tile(const PassParams& pp, int64_t tile) {
  constexpr int kV = pair_vals(LGM);
  using Sh = Shape<LGM, kV>;
  constexpr int kM = Sh::kN, kNb = kM / kV, kLgNb = LGM - Sh::kLgV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ NormPart part[16];
  cx* buf = reinterpret_cast<cx*>(smem_raw);
  const Geometry& g = pp.g;
  const int n = (int)g.n;
  const int64_t lane0 = tile * g.lanes_per_tile;
  const int64_t rem = g.outer - lane0;
  const int nl = rem < g.lanes_per_tile ? (int)rem : g.lanes_per_tile;
  longlong2* psi = reinterpret_cast<longlong2*>(pp.psi) + lane0 * n;
  const int4* tw = reinterpret_cast<const int4*>(pp.twiddle);
  const int4* chirp = reinterpret_cast<const int4*>(pp.aux);
  const int4* gt = chirp + n;
  const int t = threadIdx.x, T = blockDim.x;
  cx v[kV];
  // value r: point i0 + r M / kV of lane l0 (the layout of the outer stages)
  const int l0 = t >> kLgNb, i0 = t & (kNb - 1);
  const bool ok0 = l0 < nl;
#pragma unroll
  for (int r = 0; r < kV; ++r) {
    const int j = i0 + r * kNb;
    const longlong2 x = ok0 && j < n ? psi[l0 * n + j] : longlong2{0, 0};
    v[r] = {x.x, x.y};
  }
  const int e = lane_exponent<LGM, kV, FF>(v, part);
#pragma unroll
  for (int r = 0; r < kV; ++r) {
    const int j = i0 + r * kNb;
    v[r].x = e == kNonFinite || e == kZero ? 0 : raw_to_fx<FF>(v[r].x, e);
    v[r].y = e == kNonFinite || e == kZero ? 0 : raw_to_fx<FF>(v[r].y, e);
    if (j < n) v[r] = cmul<0>(v[r], __ldg(chirp + j));
  }
  int f1 = 1;
  while (f1 < pp.nops && pp.ops[f1].kind != OP_FFT) ++f1;
  // (one copy of the transforms' code serves all four)
#pragma unroll 1
  for (int quarter = 0; quarter < 4; ++quarter) {
    const int half = quarter >> 1;
    const bool back = quarter & 1;
    if (back) conjugate(v);
    rolled_transform<LGM, kV>(v, buf, tw, back);
    if (!back) {
      // the filter on the outputs of the closing stage (value j RS + q: point k + q P)
      constexpr int RS = Sh::kRl, kP = kM / RS;
#pragma unroll
      for (int j = 0; j < kV / RS; ++j) {
        const int k = (t + j * T) & (kP - 1);
#pragma unroll
        for (int q = 0; q < RS; ++q) {
          int4 w = __ldg(gt + k + q * kP);
          if (half) {
            w.z = -w.z;
            w.w = -w.w;
          }
          v[j * RS + q] = cmul<Sh::kConvMid>(v[j * RS + q], w);
        }
      }
      continue;
    }
    conjugate(v);
    // the n points of the transform, and the ops up to the next one.  A convolution leaves them at
    // 2^(kConvOut - g) of the norm bound; the first one's go back up to 2^60, or the second would round at
    // 2^-56 of it (error of a packet of 1000 points through the pair 1.35e-15 / 4.6e-16 without / with
    // it, 8.0e-16 by the sum in FP64).
    const int ob = half ? f1 + 1 : 1, oe = half ? pp.nops : f1;
    static_assert(Sh::kConvOut <= 62, "g is at least 2: up is not negative");
#pragma unroll
    for (int r = 0; r < kV; ++r) {
      const int j = i0 + r * kNb;
      if (j >= n || !ok0) {
        v[r] = {0, 0};
        continue;
      }
      if (half) {
        int4 w = __ldg(chirp + j);
        w.z = -w.z;
        w.w = -w.w;
        v[r] = cmul<0>(v[r], w);
      } else {
        const int up = 60 - Sh::kConvOut + pp.fx_g;
        v[r] = {v[r].x << up, v[r].y << up};
      }
      for (int oi = ob; oi < oe; ++oi) {
        const DevOp& op = pp.ops[oi];
        const int4* tab = reinterpret_cast<const int4*>(op.ptr) + (op.kind == OP_DIAGND ? (lane0 + l0) * n : 0);
        v[r] = cmul<0>(v[r], __ldg(tab + j));
      }
    }
  }
  if (ok0) {
    const int x = e - (Sh::kConvOut - pp.fx_g) - (pp.fx_exps ? table_exponent(pp, lane0 + l0) : 0);
    auto store = [&](auto low) {
#pragma unroll
      for (int r = 0; r < kV; ++r) {
        const int j = i0 + r * kNb;
        if (j >= n) continue;
        longlong2 o{fx_to_raw<FF, decltype(low)::value>(v[r].x, x), fx_to_raw<FF, decltype(low)::value>(v[r].y, x)};
        if (e == kNonFinite) o = {raw_nan<FF>(), raw_nan<FF>()};
        psi[l0 * n + j] = o;
      }
    };
    by_exponent<FF>(x, store);
  }
}

// one pass (params == nullptr: `one`), or many propagations' passes in one launch: block b
// runs tile (b - offsets[i]) of params[i], offsets[i] <= b < offsets[i + 1]
template <int LGN, bool FF, bool CHIRP>
__global__ void __launch_bounds__(kPairThreads, 1)
    fx_pair_kernel(const __grid_constant__ PassParams one, const PassParams* __restrict__ params,
                   const int64_t* __restrict__ offsets, int count) {
  wait_for_previous();
  if (params == nullptr) {
    if constexpr (CHIRP)
      fx_chirp_tile<LGN, FF>(one, blockIdx.x);
    else
      fx_pair_tile<LGN, FF>(one, blockIdx.x);
    return;
  }
  const int64_t b = blockIdx.x;
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (offsets[mid] <= b)
      lo = mid;
    else
      hi = mid - 1;
  }
  if constexpr (CHIRP)
    fx_chirp_tile<LGN, FF>(params[lo], b - offsets[lo]);
  else
    fx_pair_tile<LGN, FF>(params[lo], b - offsets[lo]);
}

template <int LGN, bool FF, bool CHIRP>
cudaError_t launch_lgn(const PassParams* one, const PassParams* params, const int64_t* offsets, int count,
                       int64_t blocks, int threads, size_t smem, cudaStream_t s) {
  static bool done = false;
  auto kern = fx_pair_kernel<LGN, FF, CHIRP>;
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return e;
    done = true;
  }
  if (smem > 220 * 1024 || threads > kPairThreads) return cudaErrorInvalidValue;
  static const PassParams none{};
  count_launch();
  return launch_overlapped(kern, (unsigned)blocks, threads, one_block_per_sm(blocks, smem), s, one ? *one : none, params, offsets, count);
}

// lgn: log2 of the lane length (CHIRP: of M)
template <bool FF, bool CHIRP>
cudaError_t launch_any(int lgn, const PassParams* one, const PassParams* params, const int64_t* offsets, int count,
                       int64_t blocks, int threads, size_t smem, cudaStream_t s) {
  switch (lgn) {
    case 4:
      if constexpr (!CHIRP) return launch_lgn<4, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
      return cudaErrorInvalidValue;
    case 5:
      if constexpr (!CHIRP) return launch_lgn<5, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
      return cudaErrorInvalidValue;
    case 6: return launch_lgn<6, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    case 7: return launch_lgn<7, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    case 8: return launch_lgn<8, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    case 9: return launch_lgn<9, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    case 10: return launch_lgn<10, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    case 11: return launch_lgn<11, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    case 12: return launch_lgn<12, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    case 13: return launch_lgn<13, FF, CHIRP>(one, params, offsets, count, blocks, threads, smem, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace
}  // namespace so
