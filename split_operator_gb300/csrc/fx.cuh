// 64-bit fixed-point arithmetic for the FP64 and float-float passes.
//
// GB300 issues about 2 FP64 operations per clock and SM (measured 1.7 FMAs), but 64 integer
// additions of 64 bits and 32 multiply-adds 32 x 32 + 64.  A lane transform is linear and
// the factors of the step (twiddles, phases, masks) have magnitudes up to 1, those of a pass
// together up to kMaxProduct, so a lane whose Euclidean norm is at most 2^e can run as 64-bit
// integers v = x 2^(60 - e): no sum of a unitary transform exceeds the norm, and one rounding
// is 2^-60 of it, where FP64 rounds every intermediate value to 2^-53 of itself.  Each lane is
// scaled by its own norm bound when it is loaded and goes back to FP64 (or hi + lo FP32) when it
// is stored.  Error of a transform pair around factors of one, relative L2 of random lanes,
// against the same pair in FP64: 4096 points 2.0e-16 / 3.5e-16, 512 points 3.6e-17 / 3.8e-16,
// 1000 points (convolutions) 4.4e-16 / 1.5e-15.
//
// What a lane shares is its exponent: a value below 2^-9 of the lane's norm has fewer than FP64's
// 53 bits, as it has behind any transform of the lane in FP64.  Factors that are small for a whole
// lane have an exponent of their own (Engine::fx_table).
//
// A factor w (|re|, |im| <= kMaxTable) is held as two signed 32-bit digits, w 2^62 = wh 2^32 + wl;
// a product with a value x = xh 2^32 + xl (balanced digits as well) is
//   xh wh + ((xh wl + xl wh + 2^31) >> 32)  =  x w / 2^64,
// three 32 x 32 + 64 multiply-adds; the dropped xl wl is below one unit.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace so {
namespace fx {

using i64 = long long;

struct cx {
  i64 x, y;
};

// bounds of the largest magnitude a table may have for the fixed-point passes, and of the product
// of a pass's tables (|v| <= 2^62 then stays below 2^62.5)
constexpr double kMaxTable = 1.25, kMaxProduct = 1.35, kMinTable = 0.5;

#ifdef __CUDACC__

__device__ __forceinline__ i64 mw(int a, int b, i64 c) { return (i64)a * (i64)b + c; }

struct dig {
  int h, l;
};
// balanced digits of x (|x| < 2^63 - 2^31): x = h 2^32 + l
__device__ __forceinline__ dig split(i64 x) {
  const int l = (int)x;
  return {(int)(x >> 32) - (l >> 31), l};
}

// v w 2^-SH for a factor given as digits {re.l, re.h, im.l, im.h} of w 2^62
template <int SH>
__device__ __forceinline__ cx cmul(cx v, int4 w) {
  const dig a = split(v.x), b = split(v.y);
  const int nl = -w.z, nh = -w.w;  // digits are above -2^31
  constexpr i64 rnd = 1ll << (29 + SH);
  i64 t = mw(a.h, w.x, rnd);
  t = mw(a.l, w.y, t);
  t = mw(b.h, nl, t);
  t = mw(b.l, nh, t);
  i64 s = mw(a.h, w.z, rnd);
  s = mw(a.l, w.w, s);
  s = mw(b.h, w.x, s);
  s = mw(b.l, w.y, s);
  if constexpr (SH == 2) {
    return {mw(b.h, nh, mw(a.h, w.y, t >> 32)), mw(b.h, w.y, mw(a.h, w.w, s >> 32))};
  } else {
    const i64 u = mw(b.h, nh, mw(a.h, w.y, 0)), q = mw(b.h, w.y, mw(a.h, w.w, 0));
    return {(u << (2 - SH)) + (t >> (30 + SH)), (q << (2 - SH)) + (s >> (30 + SH))};
  }
}

// x a + y b for constants given as balanced digits of a 2^64, b 2^64 (|a|, |b| < 1/2)
__device__ __forceinline__ i64 lin2(dig x, int ah, int al, dig y, int bh, int bl) {
  i64 t = mw(x.h, al, 1ll << 31);
  t = mw(x.l, ah, t);
  t = mw(y.h, bl, t);
  t = mw(y.l, bh, t);
  return mw(y.h, bh, mw(x.h, ah, t >> 32));
}
__device__ __forceinline__ i64 lin1(dig x, int ah, int al) {
  i64 t = mw(x.h, al, 1ll << 31);
  t = mw(x.l, ah, t);
  return mw(x.h, ah, t >> 32);
}

// the butterflies' constants as digits of c 2^64 (below 1/2): 1 - cos(pi/4), 1 - cos(pi/8),
// sin(pi/8)
constexpr int kKhH = 0x4AFB0CCC, kKhL = 0x06219B7C;
constexpr int kK1H = 0x137CA186, kK1L = 0x6B95CEBB;
constexpr int kC3H = 0x61F78A9B, kC3L = -0x455A74B9;

__device__ __forceinline__ cx add(cx a, cx b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cx sub(cx a, cx b) { return {a.x - b.x, a.y - b.y}; }

// forward (S = -1) and inverse (S = +1) butterflies, unscaled
template <int S>
__device__ __forceinline__ void dft2(cx& a, cx& b) {
  const cx t = a;
  a = add(t, b);
  b = sub(t, b);
}
template <int S>
__device__ __forceinline__ void dft4(cx& a0, cx& a1, cx& a2, cx& a3) {
  const cx e0 = add(a0, a2), e1 = sub(a0, a2), o0 = add(a1, a3), d = sub(a1, a3);
  a0 = add(e0, o0);
  a2 = sub(e0, o0);
  const cx p = {e1.x - d.y, e1.y + d.x}, m = {e1.x + d.y, e1.y - d.x};  // e1 +- i d
  a1 = S > 0 ? p : m;
  a3 = S > 0 ? m : p;
}
template <int S>
__device__ __forceinline__ void dft8(cx* a) {
  dft4<S>(a[0], a[2], a[4], a[6]);
  dft4<S>(a[1], a[3], a[5], a[7]);
  // odd outputs times w8^q: q = 1 (1 + S i)/sqrt 2, q = 2 S i, q = 3 (-1 + S i)/sqrt 2
  const cx o1 = a[3], o2 = a[5], o3 = a[7], o0 = a[1];
  const cx e0 = a[0], e1 = a[2], e2 = a[4], e3 = a[6];
  const i64 p1 = S > 0 ? o1.x - o1.y : o1.x + o1.y, q1 = S > 0 ? o1.x + o1.y : o1.y - o1.x;
  const i64 p3 = S > 0 ? o3.x + o3.y : o3.x - o3.y, q3 = S > 0 ? o3.x - o3.y : o3.x + o3.y;  // negated re / im
  const cx r1 = {p1 - lin1(split(p1), kKhH, kKhL), q1 - lin1(split(q1), kKhH, kKhL)};
  const cx r3 = {p3 - lin1(split(p3), kKhH, kKhL), q3 - lin1(split(q3), kKhH, kKhL)};
  a[0] = add(e0, o0);
  a[4] = sub(e0, o0);
  a[1] = add(e1, r1);
  a[5] = sub(e1, r1);
  const cx p2 = {e2.x - o2.y, e2.y + o2.x}, m2 = {e2.x + o2.y, e2.y - o2.x};
  a[2] = S > 0 ? p2 : m2;
  a[6] = S > 0 ? m2 : p2;
  // q = 3: re = -(x + S y) / sqrt 2, im = (S x - y) / sqrt 2
  const cx w3 = S > 0 ? cx{-r3.x, r3.y} : cx{-r3.x, -r3.y};
  a[3] = add(e3, w3);
  a[7] = sub(e3, w3);
}
template <int S>
__device__ __forceinline__ void dft16(cx* a) {
  cx e[8], o[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    e[q] = a[2 * q];
    o[q] = a[2 * q + 1];
  }
  dft8<S>(e);
  dft8<S>(o);
  // o_q *= w16^q = (cos(q pi/8), S sin(q pi/8)), cos(pi/8) = 1 - k1, sin(pi/8) = c3
  constexpr int kh = kK1H, kl = kK1L, sh = S * kC3H, sl = S * kC3L;
  {
    const dig x = split(o[1].x), y = split(o[1].y);  // (1 - k1, S c3)
    o[1] = {o[1].x - lin2(x, kh, kl, y, sh, sl), o[1].y - lin2(y, kh, kl, x, -sh, -sl)};
  }
  {
    const cx v = o[2];
    const i64 p = S > 0 ? v.x - v.y : v.x + v.y, q = S > 0 ? v.x + v.y : v.y - v.x;
    o[2] = {p - lin1(split(p), kKhH, kKhL), q - lin1(split(q), kKhH, kKhL)};
  }
  {
    const cx v = o[3];  // (c3, S (1 - k1))
    const dig x = split(v.x), y = split(v.y);
    const i64 re = lin2(x, kC3H, kC3L, y, S * kh, S * kl), im = lin2(y, kC3H, kC3L, x, -S * kh, -S * kl);
    o[3] = S > 0 ? cx{re - v.y, im + v.x} : cx{re + v.y, im - v.x};
  }
  {
    const cx v = o[5];  // (-c3, S (1 - k1))
    const dig x = split(v.x), y = split(v.y);
    const i64 re = lin2(x, -kC3H, -kC3L, y, S * kh, S * kl), im = lin2(y, -kC3H, -kC3L, x, -S * kh, -S * kl);
    o[5] = S > 0 ? cx{re - v.y, im + v.x} : cx{re + v.y, im - v.x};
  }
  {
    const cx v = o[6];  // (-1, S) / sqrt 2
    const i64 p = S > 0 ? v.x + v.y : v.x - v.y, q = S > 0 ? v.x - v.y : v.x + v.y;
    const i64 r = p - lin1(split(p), kKhH, kKhL), m = q - lin1(split(q), kKhH, kKhL);
    o[6] = S > 0 ? cx{-r, m} : cx{-r, -m};
  }
  {
    const cx v = o[7];  // (-(1 - k1), S c3)
    const dig x = split(v.x), y = split(v.y);
    o[7] = {lin2(x, kh, kl, y, -sh, -sl) - v.x, lin2(y, kh, kl, x, sh, sl) - v.y};
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (q == 4) continue;
    a[q] = add(e[q], o[q]);
    a[q + 8] = sub(e[q], o[q]);
  }
  const cx p4 = {e[4].x - o[4].y, e[4].y + o[4].x}, m4 = {e[4].x + o[4].y, e[4].y - o[4].x};
  a[4] = S > 0 ? p4 : m4;
  a[12] = S > 0 ? m4 : p4;
}
template <int RS, int S>
__device__ __forceinline__ void dft_r(cx* a) {
  if constexpr (RS == 2)
    dft2<S>(a[0], a[1]);
  else if constexpr (RS == 4)
    dft4<S>(a[0], a[1], a[2], a[3]);
  else if constexpr (RS == 8)
    dft8<S>(a);
  else
    dft16<S>(a);
}

// v 2^-SH rounded to nearest
template <int SH>
__device__ __forceinline__ cx shift_down(cx v) {
  if constexpr (SH == 0) return v;
  constexpr i64 r = SH > 0 ? 1ll << (SH > 0 ? SH - 1 : 0) : 0;
  return {(v.x + r) >> SH, (v.y + r) >> SH};
}

// ---- conversions.  The state's element: FP64 pairs, or hi + lo FP32 pairs (FF); a raw
// element is its two 8-byte halves.  Exponents are FP64's biased ones in both cases.
// the least biased exponent of a normal number; subnormal ones are below 2^(kMinExp - 1023)
template <bool FF>
constexpr int kMinExp = FF ? 897 : 1;
// biased exponent of a raw real (0 for zero and subnormals; 2047 when it is not finite)
template <bool FF>
__device__ __forceinline__ int raw_exp(i64 r) {
  if constexpr (!FF) return (int)((r >> 52) & 0x7ff);
  const int e = (int)((uint32_t)r >> 23) & 0xff;  // the hi word is the low half in memory
  return e == 255 ? 2047 : (e == 0 ? 0 : e + 896);
}
// |x| 2^(1023 - ref) of a raw real as FP32, cut to 20 significand bits or more (0 for
// subnormal x and below 2^-127)
template <bool FF>
__device__ __forceinline__ float raw_rel(i64 r, int ref) {
  if constexpr (!FF) {
    const int h = (int)(r >> 32) & 0x7fffffff;
    const int d = h - (ref - 127) * (1 << 20);  // the FP32 exponent field, from bit 20 on
    return h >= (1 << 20) && d > 0 ? __int_as_float(d << 3) : 0.0f;
  } else {
    const int b = (int)((uint32_t)r & 0x7fffffffu);
    const int d = b - (ref - 896 - 127) * (1 << 23);
    return b >= (1 << 23) && d > 0 ? __int_as_float(d) : 0.0f;
  }
}
// the bits of |x|, of hi and lo together for a pair: below kMinExp, |x| < 2^(their length - kSubnormal)
template <bool FF>
__device__ __forceinline__ unsigned long long raw_bits(i64 r) {
  if constexpr (!FF) return (unsigned long long)(r & 0x7fffffffffffffffll);
  return (uint32_t)(r | (r >> 32)) & 0x7fffffffu;
}
template <bool FF>
constexpr int kSubnormal = FF ? 149 : 1074;
// raw_rel at ref = kMinExp of a value that is not above that exponent, subnormal ones as well
template <bool FF>
__device__ __forceinline__ float raw_rel_least(i64 r) {
  if constexpr (!FF) return (float)(r & 0x1fffffffffffffll) * 0x1p-52f;
  return (float)((uint32_t)r & 0xffffffu) * 0x1p-23f;
}
// a significand with its top bit at 62, moved right by r >= 1 bits, rounded to nearest (from 64
// bits on it is below half a unit: zero)
__device__ __forceinline__ i64 shr_round(unsigned long long m, int r) {
  r = r > 64 ? 64 : (r < 1 ? 1 : r);
  return (i64)(((m >> (r - 1)) + 1ull) >> 1);
}
__device__ __forceinline__ i64 apply_sign(i64 v, int s) { return (v ^ (i64)s) - (i64)s; }  // s: 0 or -1
// raw real -> round(x 2^(60 - e)), |x| <= 2^e (e unbiased)
template <bool FF>
__device__ __forceinline__ i64 raw_to_fx(i64 r, int e) {
  if constexpr (!FF) {
    int E = (int)((r >> 52) & 0x7ff);
    unsigned long long m = (unsigned long long)r & 0xfffffffffffffull;
    m |= E ? 1ull << 52 : 0ull;
    E = E ? E : 1;
    return apply_sign(shr_round(m << 10, 1025 + e - E), (int)(r >> 63));
  } else {
    i64 v = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t b = (uint32_t)(r >> (32 * k));
      int E = (int)(b >> 23) & 0xff;
      unsigned long long m = b & 0x7fffffu;
      m |= E ? 1u << 23 : 0u;
      E = E ? E : 1;
      // m 2^(E - 150): as above with a 24-bit significand moved to bit 62
      v += apply_sign(shr_round(m << 39, 129 + e - E), (int)b >> 31);
    }
    return v;
  }
}
// |d| 2^(x + 1022), x < -1022 (out of line: lanes below 2^-962 come here)
static __device__ __noinline__ unsigned long long lower_f64(unsigned long long b, int x) {
  if (x < -2022) return 0ull;
  return (unsigned long long)__double_as_longlong(__longlong_as_double((i64)b) * __longlong_as_double((i64)(x + 2045) << 52));
}
// v 2^x -> FP64 bits, rounded to nearest.  From x = kLowExp on no result is subnormal; below (LOW), it is
// made at kLowExp and brought down by a multiplication.
constexpr int kLowExp = -1022;
template <bool LOW>
__device__ __forceinline__ i64 fx_to_f64(i64 v, int x) {
  const int s = (int)(v >> 63);
  const unsigned long long a = (unsigned long long)apply_sign(v, s);
  const int lz = __clzll((i64)a);
  const unsigned long long n = a << (lz & 63);               // top bit at 63
  const unsigned long long m = (n >> 11) + ((n >> 10) & 1);  // 53 bits (2^53 after a carry)
  const int E = 63 - lz + (LOW ? max(x, kLowExp) : x) + 1023;
  unsigned long long b = m + ((unsigned long long)(E - 1) << 52);  // the hidden bit adds 1 to E - 1
  if (E > 2046) b = 0x7ffull << 52;
  if (a == 0) b = 0;
  if (LOW && __builtin_expect(x < kLowExp, 0)) b = lower_f64(b, x);
  return (i64)(b | ((unsigned long long)(uint32_t)s << 63));
}
// v 2^x -> the hi + lo FP32 pair as a raw half
__device__ __forceinline__ i64 fx_to_ff(i64 v0, int x) {
  // moved up to 62 bits first: small values keep all of theirs
  const int s = __clzll(v0 ^ (v0 >> 63)) - 2;  // at least -1 (|v0| <= 2^63), 62 for zero
  const i64 v = s >= 0 ? v0 << s : v0 >> 1;
  const int h = (int)(v >> 32);
  float fh = __int2float_rn(h);
  const i64 rem = v - ((i64)__float2int_rn(fh) << 32);
  // fh counts 2^32 units; the remainder, below 2^38, in units of 2^8
  float fl = __int2float_rn((int)((rem + 128) >> 8)) * 0x1p-24f;
  const float t = __fadd_rn(fh, fl);
  fl = __fsub_rn(fl, __fsub_rn(t, fh));
  fh = t;
  // times 2^(x - s + 32) in two exact steps
  int q = x - s + 32;
  q = q < -250 ? -250 : (q > 250 ? 250 : q);
  const int q1 = q / 2, q2 = q - q1;
  const float f1 = __int_as_float((127 + q1) << 23), f2 = __int_as_float((127 + q2) << 23);
  fh = fh * f1 * f2;
  fl = fl * f1 * f2;
  return (i64)(((unsigned long long)__float_as_uint(fl) << 32) | __float_as_uint(fh));
}
template <bool FF, bool LOW = true>
__device__ __forceinline__ i64 fx_to_raw(i64 v, int x) {
  if constexpr (FF) return fx_to_ff(v, x);
  return fx_to_f64<LOW>(v, x);
}
template <bool FF>
__device__ __forceinline__ i64 raw_nan() {
  return FF ? (i64)0x7fc000007fc00000ll : (i64)0x7ff8000000000000ll;
}

#endif  // __CUDACC__

}  // namespace fx
}  // namespace so
