// Resident 1-D propagations of FP64 and float-float states in 64-bit fixed point (fx.cuh).
//
// One CTA holds the whole state and runs many identical steps ([norm, scale, point-wise, FFT,
// point-wise, FFT^-1, ...], the reference's Propagation::step over a 1-D grid) in one launch.  In
// FP64 a single SM's FP64 pipe set the pace (about 100 operations per point and step at 1.7 per
// clock: 51 us a step of 1024 points).  Here a thread holds 4 values (radix-4 stages: n / 4
// threads keep every scheduler of the SM busy from 512 points on, where 16 values per thread
// would leave one warp to a scheduler), the norms are integer sums (units of 2^62, sums of 2^56 and
// more; weights of many decades and momentum grids: FP64) and the scalar slots live in shared
// memory during the launch (a dependent access to the slots in global memory costs more than a
// stage).  At the end of every step the state is rounded to its storage precision, as a store and
// load would, so a run of steps gives the same bits however it is split into launches.
// Lengths that are no power of two go through transforms of M >= 2 n - 1 points (fx_pair.cuh).
#pragma once
#include "fx_stage.cuh"

namespace so {

namespace {

constexpr int kLineV = 4;  // values per thread

struct LineShared {
  double slots[kNumSlots];
  NormPart part[32];
  i64 red[2][32];
  int2 f_dig[2];
  int f_x[2];
};

// v times the real factor (digits of f 2^62)
__device__ __forceinline__ i64 rmul(i64 v, int2 f) {
  const dig a = split(v);
  i64 t = mw(a.h, f.x, 1ll << 29);
  t = mw(a.l, f.y, t);
  return (mw(a.h, f.y, 0) << 2) + (t >> 30);
}

// s + w |v|^2 (out of line: the steps' usual norms do not fetch it)
__device__ __noinline__ double norm_term(cx v, double w, double s) {
  const double x = (double)v.x, y = (double)v.y;
  return fma(fma(x, x, y * y), w, s);
}

// digits of d 2^(62 - x), |d| < 2^(x + 1/2)
__device__ __forceinline__ int2 real_digits(double d, int x) {
  i64 v = __double2ll_rn(ldexp(d, 62 - x));
  if ((int)v == (int)0x80000000) ++v;
  const dig g = split(v);
  return {g.l, g.h};
}

template <int LG, bool FF, bool CHIRP>
__global__ void __launch_bounds__((1 << LG) / kLineV, 1) fx_line_kernel(const __grid_constant__ PassParams p) {
  using Sh = Shape<LG, kLineV>;
  constexpr int kM = Sh::kN, kT = kM / kLineV;
  constexpr int kLanes = kT < 32 ? kT : 32, kWarps = (kT + 31) / 32;
  constexpr unsigned kMask = kLanes == 32 ? 0xffffffffu : (1u << (kLanes & 31)) - 1u;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LineShared S;
  cx* buf = reinterpret_cast<cx*>(smem_raw);
  const int n = (int)p.g.n, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  longlong2* psi = reinterpret_cast<longlong2*>(p.psi);
  const int4* tw = reinterpret_cast<const int4*>(p.twiddle);
  const int4* chirp = reinterpret_cast<const int4*>(p.aux);
  const int4* gt = chirp + n;
  for (int k = t; k < kNumSlots; k += kT) S.slots[k] = p.slots[k];
  // value r: point t + r M / 4 (between the transforms of a pair, for an odd log2 n, the middle
  // two values trade places: the closing radix-2 stage leaves them so)
  auto point = [&](int r, bool between) {
    const int q = !CHIRP && between && Sh::kRl == 2 ? ((r & 1) << 1) | (r >> 1) : r;
    return t + q * kT;
  };
  cx v[kLineV];
#pragma unroll
  for (int r = 0; r < kLineV; ++r) {
    const int j = t + r * kT;
    const longlong2 x = j < n ? psi[j] : longlong2{0, 0};
    v[r] = {x.x, x.y};
  }
  // weights of the program's first norm as digits (position grid), scaled by their largest exponent:
  // weights within a factor of 4 leave the sum its bits, others take the general sum below
  const double* w0 = nullptr;
  int2 wd[kLineV];
  int wx = 0;
  for (int oi = 0; oi < p.nops && w0 == nullptr; ++oi)
    if (p.ops[oi].kind == OP_NORM) w0 = p.ops[oi].w[0];
  if (w0) {
    double w[kLineV];
    int m = 1, least = 2047;
#pragma unroll
    for (int r = 0; r < kLineV; ++r) {
      const int j = t + r * kT;
      w[r] = j < n ? __ldg(w0 + j) : 0.0;
      const int e = (int)((__double_as_longlong(w[r]) >> 52) & 0x7ff);
      m = max(m, e);
      if (w[r] != 0.0) least = min(least, e);
    }
    m = __reduce_max_sync(kMask, m);
    least = __reduce_min_sync(kMask, least);
    if (lane == 0) S.part[warp] = {m, (uint32_t)least};
    __syncthreads();
    for (int i = 0; i < kWarps; ++i) {
      m = max(m, S.part[i].ref);
      least = min(least, (int)S.part[i].sum);
    }
    wx = m - 1022;  // |w| < 2^wx
#pragma unroll
    for (int r = 0; r < kLineV; ++r) wd[r] = real_digits(w[r], wx);
    if (m == 2047 || least < m - 2) w0 = nullptr;
  }
  __syncthreads();
  bool bad = false;  // a value was not finite: the state is NaN from here on
  int par = 0;       // parity of the double-buffered exchange slots
  for (int rep = 0; rep < p.repeat; ++rep) {
    const int e = lane_exponent<LG, kLineV, FF>(v, S.part);
    bad = bad || e == kNonFinite;
    const bool zero = bad || e == kZero;
    int ex = zero ? 0 : e - 60;  // value = v 2^ex
#pragma unroll
    for (int r = 0; r < kLineV; ++r)
      v[r] = {zero ? 0 : raw_to_fx<FF>(v[r].x, e), zero ? 0 : raw_to_fx<FF>(v[r].y, e)};
    bool between = false, shift = false;
    for (int oi = 0; oi < p.nops; ++oi) {
      const DevOp& op = p.ops[oi];
      switch (op.kind) {
        case OP_DIAG1D:
        case OP_DIAGND: {
          const int4* tab = reinterpret_cast<const int4*>(op.ptr);
          if (!CHIRP && shift) {
            // the scaling between the transforms rides on the first factor
#pragma unroll
            for (int r = 0; r < kLineV; ++r) v[r] = cmul<Sh::kMid>(v[r], __ldg(tab + point(r, between)));
            shift = false;
          } else {
#pragma unroll
            for (int r = 0; r < kLineV; ++r) {
              const int j = point(r, between);
              if (!CHIRP || j < n) v[r] = cmul<0>(v[r], __ldg(tab + j));
            }
          }
          break;
        }
        case OP_FFT: {
          const bool fwd = op.dir < 0;
          if constexpr (CHIRP) {
            if (fwd) {
#pragma unroll
              for (int r = 0; r < kLineV; ++r) {
                const int j = t + r * kT;
                if (j < n) v[r] = cmul<0>(v[r], __ldg(chirp + j));
              }
            }
            transform<LG, kLineV, false, 0, -1>(v, buf, tw);
            constexpr int RS = Sh::kRl, kP = kM / RS;
#pragma unroll
            for (int j = 0; j < kLineV / RS; ++j) {
              const int k = (t + j * kT) & (kP - 1);
#pragma unroll
              for (int q = 0; q < RS; ++q) {
                int4 w = __ldg(gt + k + q * kP);
                if (!fwd) {
                  w.z = -w.z;
                  w.w = -w.w;
                }
                v[j * RS + q] = cmul<Sh::kMid>(v[j * RS + q], w);
              }
            }
            transform<LG, kLineV, true, 0, 1>(v, buf, tw);
            // a convolution leaves the points 2^up below the scale that ex stands for: moved back up, or
            // the second one and the norms would round at that
            const int up = p.fx_g - Sh::kSc;
#pragma unroll
            for (int r = 0; r < kLineV; ++r) {
              const int j = t + r * kT;
              v[r] = {v[r].x << up, v[r].y << up};
              if (j >= n) {
                v[r] = {0, 0};
              } else if (!fwd) {
                int4 w = __ldg(chirp + j);
                w.z = -w.z;
                w.w = -w.w;
                v[r] = cmul<0>(v[r], w);
              }
            }
          } else {
            if (fwd) {
              transform<LG, kLineV, false, 0, -1>(v, buf, tw);
              shift = true;
            } else {
              if (shift) {
#pragma unroll
                for (int r = 0; r < kLineV; ++r) v[r] = shift_down<Sh::kMid>(v[r]);
                shift = false;
              }
              transform<LG, kLineV, true, 0, 1>(v, buf, tw);
              ex -= Sh::kSc;
            }
          }
          between = fwd;
          break;
        }
        case OP_SCALE: {
          if (t == 0) {
            const double f = sqrt(S.slots[op.b] / S.slots[op.c]);
            int x = 0;
            double m = frexp(f, &x);
            // factors about 1, and below 1.25, or (op.a, from the third of a step on) below 1
            if (m < 0.625 && op.a == 0) {
              m *= 2.0;
              x -= 1;
            }
            S.f_dig[par] = real_digits(isfinite(f) ? m : 0.0, 0);
            S.f_x[par] = isfinite(f) ? x : kNonFinite;
          }
          __syncthreads();
          const int2 f = S.f_dig[par];
          const int x = S.f_x[par];
          par ^= 1;
          bad = bad || x == kNonFinite;
          ex += x == kNonFinite ? 0 : x;
#pragma unroll
          for (int r = 0; r < kLineV; ++r) v[r] = {rmul(v[r].x, f), rmul(v[r].y, f)};
          break;
        }
        case OP_NORM: {
          // sum w |v|^2: squares in units of 2^62 (their sum stays below 2^62) and weighted digits, or
          // (weights of many decades, the momentum grid's) in FP64
          i64 s = 0;
          double sd = 0.0;
          const bool quick = w0 != nullptr && op.w[0] == w0 && !between;
#pragma unroll
          for (int r = 0; r < kLineV; ++r) {
            if (quick) {
              const dig a = split(v[r].x), b = split(v[r].y);
              // (with the low digits' squares, from their upper halves: the thirds of a unit that they come
              // to were 4e-14 of the norm of 500 points)
              const int al = a.l >> 16, bl = b.l >> 16;
              const uint32_t low = ((uint32_t)(al * al) + (uint32_t)(bl * bl) + (1u << 29)) >> 1;
              const i64 q = (mw(b.h, b.h, mw(a.h, a.h, 0)) << 2) + (mw(b.h, b.l, mw(a.h, a.l, (i64)low)) >> 29);
              s += rmul(q, wd[r]);
            } else {
              const int j = point(r, between);
              if (j < n) sd = norm_term(v[r], __ldg(op.w[0] + j), sd);
            }
          }
          if (quick) {
#pragma unroll
            for (int o = kLanes / 2; o > 0; o >>= 1) s += __shfl_down_sync(kMask, s, o);
          } else {
#pragma unroll
            for (int o = kLanes / 2; o > 0; o >>= 1) sd += __shfl_down_sync(kMask, sd, o);
            s = __double_as_longlong(sd);
          }
          if (lane == 0) S.red[par][warp] = s;
          __syncthreads();
          if (t == 0) {
            double tot = 0.0;
            if (quick) {
              i64 a = 0;
              for (int i = 0; i < kWarps; ++i) a += S.red[par][i];
              tot = ldexp((double)a, 62 + wx + 2 * ex);
            } else {
              for (int i = 0; i < kWarps; ++i) tot += __longlong_as_double(S.red[par][i]);
              // between the transforms of a power of two, ex still stands for the values ahead of the
              // forward one: the unitary transform is v 2^(ex + kSumF + kMid - LG / 2), without kMid
              // while that shift has not been made (CHIRP transforms are unitary, ex is theirs)
              const int mid = !CHIRP && between ? 2 * Sh::kSumF - LG + (shift ? 0 : 2 * Sh::kMid) : 0;
              tot = ldexp(tot, 2 * ex + mid);
            }
            if (bad) tot = __longlong_as_double(0x7ff8000000000000ll);
            S.slots[op.a] = tot;
            if (!isfinite(tot) && p.nonfinite_slot >= 0) S.slots[p.nonfinite_slot] = 1.0;
          }
          par ^= 1;
          break;
        }
        case OP_COPY:
          if (t == 0) S.slots[op.a] = S.slots[op.b];
          break;
        case OP_LOSS:
          if (t == 0) S.slots[op.a] += S.slots[op.b] - S.slots[op.c];
          break;
        case OP_SETC:
          if (t == 0) S.slots[op.a] = op.value;
          break;
        case OP_RECORD:
          if (t == 0 && p.record) p.record[op.count] = S.slots[op.a];
          break;
        default:
          break;
      }
    }
    // the step's result in the state's precision
    by_exponent<FF>(ex, [&](auto low) {
      constexpr bool L = decltype(low)::value;
#pragma unroll
      for (int r = 0; r < kLineV; ++r)
        v[r] = {bad ? raw_nan<FF>() : fx_to_raw<FF, L>(v[r].x, ex), bad ? raw_nan<FF>() : fx_to_raw<FF, L>(v[r].y, ex)};
    });
    if (CHIRP) {
#pragma unroll
      for (int r = 0; r < kLineV; ++r)
        if (t + r * kT >= n) v[r] = {0, 0};
    }
  }
#pragma unroll
  for (int r = 0; r < kLineV; ++r) {
    const int j = t + r * kT;
    if (j < n) psi[j] = longlong2{v[r].x, v[r].y};
  }
  __syncthreads();
  for (int k = t; k < kNumSlots; k += kT) p.slots[k] = S.slots[k];
}

template <int LG, bool FF, bool CHIRP>
cudaError_t launch_line_lg(const PassParams& p, cudaStream_t s) {
  static bool done = false;
  auto kern = fx_line_kernel<LG, FF, CHIRP>;
  const size_t smem = (size_t)Shape<LG, kLineV>::kLs * sizeof(cx);
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    done = true;
  }
  kern<<<1, (1 << LG) / kLineV, smem, s>>>(p);
  count_launch();
  return cudaGetLastError();
}

template <bool FF, bool CHIRP>
cudaError_t launch_line_any(const PassParams& p, cudaStream_t s) {
  switch (p.fx) {
    case 4: if constexpr (!CHIRP) return launch_line_lg<4, FF, CHIRP>(p, s); return cudaErrorInvalidValue;
    case 5: if constexpr (!CHIRP) return launch_line_lg<5, FF, CHIRP>(p, s); return cudaErrorInvalidValue;
    case 6: return launch_line_lg<6, FF, CHIRP>(p, s);
    case 7: return launch_line_lg<7, FF, CHIRP>(p, s);
    case 8: return launch_line_lg<8, FF, CHIRP>(p, s);
    case 9: return launch_line_lg<9, FF, CHIRP>(p, s);
    case 10: return launch_line_lg<10, FF, CHIRP>(p, s);
    case 11: return launch_line_lg<11, FF, CHIRP>(p, s);
    case 12: return launch_line_lg<12, FF, CHIRP>(p, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace
}  // namespace so
