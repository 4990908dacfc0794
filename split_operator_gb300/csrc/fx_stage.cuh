// Fixed-point transforms (fx.cuh) of power-of-two lanes held in registers, KV values per thread,
// exchanged in place in one shared buffer; and the norm bound a lane is scaled by.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "fx.cuh"

namespace so {

using namespace fx;

namespace {

__host__ __device__ constexpr int lg2(int x) { return x <= 1 ? 0 : 1 + lg2(x / 2); }

// A power-of-two transform of 2^LGN points with KV values per thread (16, 8 or 4) and radix-KV stages.
// Values come in at 2^60 of the lane's norm bound or below; the first stage is unscaled, a stage
// with twiddles scales by the square root of its radix or a little more in its products.  The norm
// grows by the square root of a stage's radix and stays below 2^62.
template <int LGN, int KV>
struct Shape {
  static constexpr int kN = 1 << LGN, kLgV = lg2(KV);
  static constexpr int kS = (LGN + kLgV - 1) / kLgV;         // radix-KV stages, the last one kRl
  static constexpr int kLgRl = LGN - kLgV * (kS - 1);        // closing radix (2 .. KV)
  static constexpr int kRl = 1 << kLgRl;
  static constexpr int kSc = (kLgV + 1) / 2;                 // scaling of a full stage: 2^-kSc
  static constexpr int kSh = (kLgRl + 1) / 2;                // of the closing stage of the forward order
  static constexpr int kSumF = kS > 1 ? (kS - 2) * kSc + kSh : 0, kSumR = (kS - 1) * kSc;
  // of the factors between a pair's transforms: brings the norm back to 2^60, or (radix 8, whose
  // stages scale by more than they need) just keeps it below 2^62 after the next unscaled stage
  static constexpr int kTop = 120 + LGN - 2 * kSumF + kLgRl;  // half bits of the norm there
  static constexpr int kMid = KV != 8 ? kLgRl / 2 : (kTop > 124 ? (kTop - 123) / 2 : 0);
  // ... of the filter between the transforms of a convolution (a unitary one times 2^-g, g >= 2,
  // magnitudes <= 1): the norm below 2^62 after the next stage, and 2^60.5 or less behind it
  static constexpr int conv_mid() {
    if (KV != 8) return kMid;
    int m = kMid;
    while (kTop - 2 * (m - 1) <= 124 && 120 + 2 * LGN - 2 * kSumF - 2 * (m - 1) - 2 * kSumR <= 121 + 4) --m;
    return m;
  }
  static constexpr int kConvMid = conv_mid();
  static constexpr int kPad = KV == 16 ? 4 : 3;              // one padding element every 2^kPad
  static constexpr int kLs = kN + (kN >> kPad) + 1;          // padded lane stride
  static constexpr int kOut = 60 + LGN - kSumF - kMid - kSumR;  // exponent after a pair: x 2^(kOut - e)
  static constexpr int kConvOut = kOut + kMid - kConvMid;       // ... after a convolution
  __host__ __device__ static constexpr int rs(bool rev, int s) {
    return rev ? (s == 0 ? kRl : KV) : (s + 1 < kS ? KV : kRl);
  }
  __host__ __device__ static constexpr int span(bool rev, int s) {
    return s == 0 ? 1 : span(rev, s - 1) * rs(rev, s - 1);
  }
  // first entry of stage s in the stage-major twiddle table (reversed order: from entry n)
  __host__ __device__ static constexpr int twoff(bool rev, int s) {
    return s == 0 ? (rev ? kN : 0)
                  : twoff(rev, s - 1) + (span(rev, s - 1) > 1 ? (rs(rev, s - 1) - 1) * span(rev, s - 1) : 0);
  }
};

// One stage of radix RS, span P, twiddles from entry OFF; IN: 0 registers, 1 shared memory;
// OUT: 0 registers, 1 shared memory.  SC: the stage scales by 2^-SC (in its products).
template <int LGN, int KV, int RS, int P, int OFF, bool IN, bool OUT, int DIR, int SC>
__device__ __forceinline__ void stage(cx (&v)[KV], cx* buf, const int4* __restrict__ tw) {
  constexpr int kN = 1 << LGN, kNb = kN / RS, kLgNb = LGN - lg2(RS), kLs = Shape<LGN, KV>::kLs, kPad = Shape<LGN, KV>::kPad;
  const int t = threadIdx.x, T = blockDim.x;
  if constexpr (IN) {
#pragma unroll
    for (int j = 0; j < KV / RS; ++j) {
      const int b = t + j * T, l = b >> kLgNb, i = b & (kNb - 1);
      const cx* src = buf + l * kLs + i + (i >> kPad);
#pragma unroll
      for (int r = 0; r < RS; ++r) {
        // element i + r nb: its padding splits into those of i and r nb when nb is a multiple of 2^kPad
        v[j * RS + r] = kNb % (1 << kPad) == 0 ? src[r * kNb + ((r * kNb) >> kPad)]
                                               : buf[l * kLs + i + r * kNb + ((i + r * kNb) >> kPad)];
      }
    }
    __syncthreads();  // every read of the stage before any write (in place)
  }
#pragma unroll
  for (int j = 0; j < KV / RS; ++j) {
    if constexpr (P > 1) {
      // k = i & (P - 1) = b & (P - 1) (P divides nb)
      const int4* w = tw + OFF + ((t + j * T) & (P - 1));
      v[j * RS] = shift_down<SC>(v[j * RS]);
#pragma unroll
      for (int r = 1; r < RS; ++r) {
        int4 wv = __ldg(w + (r - 1) * P);
        if (DIR > 0) {
          wv.z = -wv.z;
          wv.w = -wv.w;
        }
        v[j * RS + r] = cmul<SC>(v[j * RS + r], wv);
      }
    }
    dft_r<RS, DIR>(&v[j * RS]);
  }
  if constexpr (OUT) {
#pragma unroll
    for (int j = 0; j < KV / RS; ++j) {
      const int b = t + j * T, l = b >> kLgNb, i = b & (kNb - 1), k = i & (P - 1);
      const int base = (i - k) * RS + k;
#pragma unroll
      for (int q = 0; q < RS; ++q) {
        const int x = base + q * P;
        buf[l * kLs + x + (x >> kPad)] = v[j * RS + q];
      }
    }
    __syncthreads();
  }
}

template <int LGN, int KV, bool REV, int S, int DIR>
__device__ __forceinline__ void transform(cx (&v)[KV], cx* buf, const int4* tw) {
  using Sh = Shape<LGN, KV>;
  constexpr int rs = Sh::rs(REV, S), p = Sh::span(REV, S);
  constexpr int sc = (!REV && S + 1 == Sh::kS) ? Sh::kSh : Sh::kSc;
  stage<LGN, KV, rs, p, Sh::twoff(REV, S), (S > 0), (S + 1 < Sh::kS), DIR, sc>(v, buf, tw);
  if constexpr (S + 1 < Sh::kS) transform<LGN, KV, REV, S + 1, DIR>(v, buf, tw);
}

// A transform whose full stages are one loop: forward order (REV false), or the reversed radix order
// with its own twiddles.  The direction is forward in both (conjugate around it for the inverse).
// Unrolled, a pair of 4096-point transforms was 10,400 instructions in a row, each executed once
// by a warp, and most of its time went into fetching them (61 % of the stalls).
// Values come and leave in registers: point i + r nb of the first stage, k + q P of the last.
template <int LGN, int KV>
__device__ __forceinline__ void rolled_transform(cx (&v)[KV], cx* buf, const int4* __restrict__ tw, bool rev) {
  using Sh = Shape<LGN, KV>;
  constexpr int kN = Sh::kN, kNb = kN / KV, kLgNb = LGN - Sh::kLgV, kLs = Sh::kLs, kPad = Sh::kPad;
  constexpr bool kEven = Sh::kRl == KV;  // every stage is a full one: both orders are the same
  const int t = threadIdx.x, l = t >> kLgNb, i = t & (kNb - 1);
  cx* const mine = buf + l * kLs;
  if constexpr (!kEven) {
    if (rev) stage<LGN, KV, Sh::kRl, 1, 0, false, true, -1, 0>(v, buf, tw);
  }
  int lgp = !kEven && rev ? Sh::kLgRl : 0;
  const int4* w = tw + (!kEven && rev ? kN : 0);
  constexpr int kFull = kEven ? Sh::kS : Sh::kS - 1;
#pragma unroll 1
  for (int s = 0; s < kFull; ++s) {
    const int k = i & ((1 << lgp) - 1);
    if (lgp > 0) {
      const int4* wk = w + k;
      int4 wv[KV];
#pragma unroll
      for (int r = 1; r < KV; ++r) wv[r] = __ldg(wk + ((r - 1) << lgp));
#pragma unroll
      for (int r = 0; r < KV; ++r)
        v[r] = kNb % (1 << kPad) == 0 ? mine[i + (i >> kPad) + r * kNb + ((r * kNb) >> kPad)]
                                      : mine[i + r * kNb + ((i + r * kNb) >> kPad)];
      __syncthreads();  // every read of the stage before any write (in place)
      v[0] = shift_down<Sh::kSc>(v[0]);
#pragma unroll
      for (int r = 1; r < KV; ++r) v[r] = cmul<Sh::kSc>(v[r], wv[r]);
      w += (KV - 1) << lgp;
    }
    dft_r<KV, -1>(v);
    if (s + 1 < kFull || (!kEven && !rev)) {
      const int base = ((i - k) << Sh::kLgV) + k;
#pragma unroll
      for (int q = 0; q < KV; ++q) {
        const int x = base + (q << lgp);
        mine[x + (x >> kPad)] = v[q];
      }
      __syncthreads();
    }
    lgp += Sh::kLgV;
  }
  if constexpr (!kEven) {
    if (!rev)
      stage<LGN, KV, Sh::kRl, Sh::span(false, Sh::kS - 1), Sh::twoff(false, Sh::kS - 1), true, false, -1, Sh::kSh>(v, buf, tw);
  }
}

template <int KV>
__device__ __forceinline__ void conjugate(cx (&v)[KV]) {
#pragma unroll
  for (int r = 0; r < KV; ++r) v[r].y = -v[r].y;
}

// store(true) for a lane whose results may be subnormal, else store(false): the check once, out of the
// conversions (in each of them it took 2 % of a resident step)
template <bool FF, class F>
__device__ __forceinline__ void by_exponent(int x, F&& store) {
  if (!FF && __builtin_expect(x < kLowExp, 0))
    store(std::integral_constant<bool, true>{});
  else
    store(std::integral_constant<bool, false>{});
}

// Lane norm bounds.  A thread's KV values lie in one lane (lane = t >> lg(n / KV)).  Returns e
// with |lane|_2 <= 2^e, kNonFinite for a lane with a value that is not finite, kZero for one of
// zeros.  part: one entry per warp.
struct NormPart {
  int ref;
  uint32_t sum;  // sum |x|^2 2^(2 (1023 - ref)) in units of 2^-12, rounded up
};
constexpr int kNonFinite = 1 << 20, kZero = -(1 << 20), kNone = -4096;
template <int LGN, int KV, bool FF>
__device__ __forceinline__ int lane_exponent(const cx (&raw)[KV], NormPart* part) {
  constexpr int kTpl = (1 << LGN) / KV;  // threads per lane
  const int t = threadIdx.x, lane = t & 31;
  int m = 0;
#pragma unroll
  for (int e = 0; e < KV; ++e) m = max(m, max(raw_exp<FF>(raw[e].x), raw_exp<FF>(raw[e].y)));
  if (__builtin_expect(m == 0, 0)) {
    // zeros and subnormal values: the exponent these stand for
    unsigned long long any = 0;
#pragma unroll
    for (int e = 0; e < KV; ++e) any |= raw_bits<FF>(raw[e].x) | raw_bits<FF>(raw[e].y);
    m = any ? 64 - __clzll((i64)any) - kSubnormal<FF> + 1022 : kNone;
  }
  constexpr int kG = kTpl < 32 ? kTpl : 32;
  const unsigned mask = kG == 32 ? 0xffffffffu : ((1u << (kG & 31)) - 1u) << (lane & ~(kG - 1));
  m = __reduce_max_sync(mask, m);
  int ref = max(m, 1);
  float s = 0.0f;
#pragma unroll
  for (int e = 0; e < KV; ++e) {
    const float x = raw_rel<FF>(raw[e].x, ref), y = raw_rel<FF>(raw[e].y, ref);
    s = fmaf(x, x, fmaf(y, y, s));
  }
  // (a lane with a value that is not finite: s may be infinite, the conversion saturates)
  uint32_t q = __reduce_add_sync(mask, (uint32_t)min((int)__float2int_ru(s * 4096.0f), 1 << 20));
  float tot = (float)q;
  if constexpr (kTpl > 32) {
    constexpr int kW = kTpl / 32;  // warps per lane
    const int w = t >> 5, w0 = w & ~(kW - 1);
    if (lane == 0) part[w] = {m, q};
    __syncthreads();
    m = kNone;
#pragma unroll
    for (int i = 0; i < kW; ++i) m = max(m, part[w0 + i].ref);
    ref = max(m, 1);
    tot = 0.0f;
#pragma unroll
    for (int i = 0; i < kW; ++i) {
      const int d = ref - max(part[w0 + i].ref, 1);
      tot = fmaf((float)part[w0 + i].sum, d < 60 ? __int_as_float((127 - 2 * d) << 23) : 0.0f, tot);
    }
    tot += 1.0f;  // the terms cut off above, in units of 2^-12 of the largest value's square
  }
  if (m == 2047) return kNonFinite;
  // subnormal values alone: by their number; beside larger ones they are covered by a least exponent
  // (four times what they come to)
  constexpr int kCount = (LGN + 2) / 2, kLeast = kMinExp<FF> - 1023;
  if (__builtin_expect(m < kMinExp<FF>, 0)) return m == kNone ? kZero : max(m - 1022 + kCount, kLeast);
  // |lane|^2 <= tot (1 + 2^-15) 2^-12 2^(2 (ref - 1023)): e = the least integer with 4^e above
  const int ex = (__float_as_int(fmaf(tot, 0x1p-15f, tot)) >> 23) - 127 - 12;  // tot < 2^(ex + 1)
  return max((ref - 1023) + ((ex + 2) >> 1), kLeast + kCount + 2);
}

}  // namespace
}  // namespace so
