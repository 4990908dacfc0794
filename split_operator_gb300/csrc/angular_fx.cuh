// The lane-matrix pass of FP64 and float-float states on the tensor cores.
//
// Replaces, fused into one pass like the FP32 kernel of angular_tc.cu, MatrixTransformation and
// StateMatrixTransformation for real matrices (matrix_transformation.rs:60-75,
// state_matrix_transformation.rs:48-73) with the diagonal propagators, masks, scales and norm
// folds around them.  On the CUDA cores the products were bound by the FP64 pipe (two FMAs per
// matrix entry and complex value at 1.7 a clock and SM: 592 us for the two-matrix pass of a
// 4096 x 128 state).  Here they are exact integer products on the tensor cores and everything
// else is 64-bit fixed point (fx.cuh).
//
// Slices (the Ozaki scheme: K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59,
// 2012).  Every B column (a real or imaginary column of the tile) is scaled by a power of two
// above its largest magnitude and rounded to 55 bits, every A row (a matrix row, on the host)
// likewise; both are cut into seven signed 8-bit digits, held as FP16 integers of magnitude
// <= 128.  The digit products of one order r = i + j (A digit i, B digit j) share a weight, so
// they sum in one FP32 accumulator: (r + 1) K 2^14 <= 2^24 for K = 128 and every r <= 6, so
// the sums are exact (K = 256: r <= 3; the other orders weigh less than 2^-48).  The products of
// orders 7 .. 12 are left out: at most 2^-51 of (row maximum x column maximum) for random rows and
// columns of K = 128, 2^-47 for constant ones, whose sum is 2^7 times as large (2^-45.5 and 2^8 for K =
// 256).  Error of [T, phase, T^-1], relative L2 per column, against the same in FP64: Legendre pairs of
// 16 to 256 points 1.0e-16 - 5.2e-16 / 1.6e-16 - 9.4e-16 (columns random, constant, of few or the highest
// l, of one point), random orthogonal ones of 16 points 2.3e-16 / 2.1e-16, from 32 on below FP64's.
//
// A tile is BN complex columns of the inner axis for all n rows (n <= 256), N = 2 BN real
// columns.  One persistent CTA per SM (seven accumulators of 64 columns fill its tensor memory):
//   warps 0-15  load the tile, apply the point-wise ops, write the B digits, drain the
//               accumulators, store, and sum the norms per warp; thread = one matrix row (TMEM
//               lane) and NB neighbouring complex columns in every phase
//   warp 16     streams the A digit images (8 KB per 128 rows x 32 K values) through a 64 KB
//               ring by bulk TMA copies
//   warp 17     issues tcgen05.mma kind::f16 (48 clocks a product: the reads of both operands) and
//               publishes the tile's norms and ticket meanwhile (pass_end.cuh)
// The two-matrix pass of a 4096 x 128 state takes 62 us now: 13 in the products, the rest in the work
// warps' integer arithmetic (27 % of the issue slots; latency at four warps a scheduler).
// B digits lie N-major in shared memory (eight real columns of one K row are 16 bytes), so a
// thread writes its four complex columns of a digit with one 16-byte store.
// Every mbarrier wait is bounded (2 s), as in angular_tc.cu.
#pragma once
#include "common.cuh"
#include "fx.cuh"
#include "overlap.cuh"
#include "pass_end.cuh"
#include "tc_common.cuh"

namespace so {

using namespace fx;

struct FxTcParams {
  PassParams p;
  int32_t mat_op[2];  // op indices of the (one or two) lane matrices
  int32_t nmat;
  int32_t handover;   // see pass_handover
  int32_t kp;         // lane extent rounded up to 32: K of the products
  int32_t error_slot;
  int32_t slice_axis[2];      // state matrix: the logical axis whose coordinate picks the image (-1: one)
  const unsigned char* images[2];
  int64_t slice_stride[2];    // bytes between two coordinates' images
  uint32_t slice_pre[2], slice_div[2], slice_ext[2];  // the tile's coordinate, as in TcParams
};

namespace {

constexpr int kFxWork = 512;                 // work threads (warps 0-15)
constexpr int kFxThreads = kFxWork + 64;     // + warp 16 (TMA) + warp 17 (MMA)
constexpr int kDigits = 7;
constexpr uint32_t kChunkRowBytes = 8192;    // 128 rows x 32 K values of one digit
constexpr uint64_t kFxWait = 2000000000ull;  // 2 s per wait
constexpr int kFxTabSlots = 4;               // DIAG1D ops on a non-lane axis per pass
constexpr int kFxMaxCols = 32;
constexpr int kNoTerm = 1 << 20;             // exponent of a zero weight: below every other
constexpr int kFxPoison = 1 << 24;           // exponent of a column with a value that is not finite

__host__ __device__ constexpr uint32_t fx_b_bytes(int cols, int kp) { return (uint32_t)(2 * cols * kp * 2); }
constexpr uint32_t kRingBytes = 65536;
__host__ __device__ constexpr uint32_t fx_tc_smem(int cols, int kp) {
  return kRingBytes + kDigits * fx_b_bytes(cols, kp);
}

__device__ __forceinline__ void fx_work_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kFxWork) : "memory"); }
__device__ __forceinline__ bool fx_work_all(bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v), "n"(kFxWork)
      : "memory");
  return r != 0;
}

// kind::f16 with FP16 A (K-major) and B (N-major), D = F32
__host__ __device__ constexpr uint32_t idesc_f16_nmajor(uint32_t m, uint32_t n) {
  return (1u << 4) | (1u << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// columns c .. c + 3 of the seven accumulators (step columns apart), one wait
__device__ __forceinline__ void tmem_ld4x7(uint32_t taddr, uint32_t step, uint32_t (&r)[28]) {
#pragma unroll
  for (int k = 0; k < 7; ++k)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[4 * k]), "=r"(r[4 * k + 1]), "=r"(r[4 * k + 2]), "=r"(r[4 * k + 3])
                 : "r"(taddr + (uint32_t)k * step)
                 : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13])
               :
               : "memory");
  asm volatile(""
               : "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
                 "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27])
               :
               : "memory");
}

// The seven orders' sums of one value -> the product times 2^-sh of the last order's unit,
// rounded to nearest (sh = lg K + 1 keeps it below 2^61).  s0 .. s6 are integers below 2^24.
template <int MH>
__device__ __forceinline__ i64 combine(int s0, int s1, int s2, int s3, int s4, int s5, int s6, int sh) {
  i64 hi;
  if constexpr (MH == 1)
    hi = mw(s0 * 256 + s1, 65536, (i64)(s2 * 256 + s3));  // K <= 128: both fit 32 bits
  else
    hi = mw(s0, 1 << 24, mw(s1, 65536, mw(s2, 256, (i64)s3)));
  const i64 lo = mw(s4, 65536, mw(s5, 256, (i64)s6));
  return (hi << (24 - sh)) + (((lo >> (sh - 1)) + 1) >> 1);
}

// pair (a, b) of 56-bit values: digit j of both as packed FP16 integers
__device__ __forceinline__ uint32_t digit_pair(const uint32_t (&a)[2], const uint32_t (&b)[2], int j) {
  const int byte = 6 - j;
  uint32_t p;
  if (byte == 6)
    p = __byte_perm(a[1], b[1], 0x7632);  // the top digit (plus 128) may be 256: a half word
  else
    p = __byte_perm(a[byte >> 2], b[byte >> 2], 0x0400 | (byte & 3) | ((4 + (byte & 3)) << 8)) & 0x00ff00ffu;
  p |= 0x64006400u;  // FP16 1024 + (digit + 128)
  uint32_t r;
  asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(p), "r"(0x64806480u));
  return r;
}

// v 2^sh rounded to nearest (-63 <= sh; left shifts stay in range by the caller's bounds)
__device__ __forceinline__ i64 shift_by(i64 v, int sh) {
  if (sh >= 0) return v << sh;
  const int r = sh < -62 ? 62 : -sh;
  return (((v >> (r - 1)) + 1) >> 1);
}

__device__ __forceinline__ int bits_of(i64 x, i64 y) {  // |x|, |y| <= 2^bits (0: both zero)
  const unsigned long long a = (unsigned long long)(x ^ (x >> 63)) | (unsigned long long)(y ^ (y >> 63));
  return a == 0 ? ((x | y) != 0 ? 1 : 0) : 64 - __clzll((i64)a);
}

// d 2^k (d >= 0 or NaN), saturating to infinity
__device__ __forceinline__ double scale_pow2(double d, int k) {
  const i64 b = __double_as_longlong(d);
  const int e = (int)(b >> 52) & 0x7ff;
  if (e == 0 || e == 0x7ff) return d;
  if (e + k <= 0)  // subnormal
    return e + k < -60 ? 0.0 : __longlong_as_double(b + ((i64)(k + 64) << 52)) * 0x1p-64;
  if (e + k >= 0x7ff) return __longlong_as_double(0x7ff0000000000000ll);
  return __longlong_as_double(b + ((i64)k << 52));
}

// Two neighbouring 16-byte values in one access of 32 bytes: a warp's accesses, one row to a lane, then
// move whole sectors (16-byte ones fetched each twice; 4096 x 128 plane 85.4 -> 83.5 us a step).
// Rows whose address or width does not allow it take the 16-byte form.
__device__ __forceinline__ bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }
__device__ __forceinline__ void load_pair(const int4* p, int4& a, int4& b) {  // constant tables
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
      : "l"(p));
}
__device__ __forceinline__ void load_pair(const longlong2* p, cx& a, cx& b) {
  asm volatile("ld.global.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(a.x), "=l"(a.y), "=l"(b.x), "=l"(b.y) : "l"(p) : "memory");
}
__device__ __forceinline__ void store_pair(longlong2* p, cx a, cx b) {
  asm volatile("st.global.v4.b64 [%0], {%1,%2,%3,%4};" ::"l"(p), "l"(a.x), "l"(a.y), "l"(b.x), "l"(b.y) : "memory");
}

struct FxTabs {
  int4 colt[kFxTabSlots][kFxMaxCols];   // DIAG1D on a non-lane axis: its factor per tile column
  // NORM: product of the weights of every non-lane axis, as a RowWeight's digits and exponent
  int2 colwd[kMaxRed][kFxMaxCols];
  int colwx[kMaxRed][kFxMaxCols];
  int scale_x[kMaxOps];                 // SCALE: factor = digits x 2^scale_x
  int2 scale_d[kMaxOps];
  int colx[kFxMaxCols];                 // exponent of the column's values (before row exponents)
  int cole[2][kFxMaxCols];              // column maxima: biased exponents
  int coler[kFxMaxCols];                // the same at a ROUND
  int colb[kFxMaxCols];                 // exponent bound of the column's B operand
  int nonident[kFxTabSlots];            // the factors of this tile: 0 all are 1, 1 all real, else complex
  int16_t opk[kMaxOps][kFxMaxCols];     // tables with exponents: of the op's factors per column
  uint32_t kany;                        // bit i: op i has one in this tile
  int8_t slot[kMaxOps];
  double red[2][kMaxRed][kFxWork / 32];  // norms: the warps' sums (of every second tile)
};

__device__ __forceinline__ int64_t fx_coord(const Geometry& g, int a, int64_t o, int64_t i) {
  int64_t v = i;
  for (int q = g.ndim - 1; q > g.spos; --q) {
    if (g.perm[q] == a) return v % g.sshape[q];
    v /= g.sshape[q];
  }
  v = o;
  for (int q = g.spos - 1; q >= 0; --q) {
    if (g.perm[q] == a) return v % g.sshape[q];
    v /= g.sshape[q];
  }
  return 0;
}

// image block of matrix m for a tile (a state matrix: the one of the tile's coordinate)
__device__ __forceinline__ const unsigned char* fx_image(const FxTcParams& q, int m, int64_t tile) {
  const unsigned char* img = q.images[m];
  if (q.slice_axis[m] >= 0) {
    uint32_t t = (uint32_t)tile;
    if (q.slice_pre[m]) t %= q.slice_pre[m];
    img += (int64_t)((t / q.slice_div[m]) % q.slice_ext[m]) * q.slice_stride[m];
  }
  return img;
}

struct FxTile {
  const FxTcParams* prm;
  int64_t tile;
};
struct FxResolve {
  const FxTcParams* one;
  const FxTcParams* params;
  const uint2* owners;
  __device__ __forceinline__ FxTile operator()(int64_t b) const {
    if (params == nullptr) return {one, b};
    const uint2 o = __ldg(owners + b);
    return {params + o.x, (int64_t)o.y};
  }
};

// Warp 16, lane 0: the digit images of every tile's matrices through the ring, all digits of 32 K
// values, then the next 32: the last digits of a chunk take few products, and in this order the
// copies keep an even pace.
template <int MH>
__device__ __noinline__ void fx_producer(FxResolve resolve, int64_t total, uint32_t ring, uint64_t* full,
                                         uint64_t* empty, volatile int* fail) {
  using namespace tc;
  constexpr uint32_t bytes = kChunkRowBytes * MH;
  constexpr int ns = (int)(kRingBytes / bytes);
  int s = 0;
  uint32_t use = 0;
  int64_t cc = 0;
  bool ok = true;
  for (int64_t gt = blockIdx.x; gt < total && ok && !*fail; gt += gridDim.x) {
    const FxTile r = resolve(gt);
    const int nk = r.prm->kp / 32;
    for (int m = 0; m < r.prm->nmat && ok; ++m) {
      const unsigned char* img = fx_image(*r.prm, m, r.tile);
      for (int q = 0; q < kDigits * nk; ++q) {
        const int part = (q % kDigits) * nk + q / kDigits;  // stored digit by digit
        if (use > 0 && !mbar_poll(&empty[s], (use - 1) & 1u, kFxWait)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&full[s], bytes);
        bulk_g2s(sm_ptr(ring + (uint32_t)s * bytes), img + (size_t)part * bytes, bytes, &full[s]);
        ++cc;
        if (++s == ns) {
          s = 0;
          ++use;
        }
      }
    }
  }
  if (!ok) {
    *fail = 1;
    // let the copies in flight land before the CTA lets go of its shared memory
    for (int64_t c = cc - ns < 0 ? 0 : cc - ns; c < cc; ++c)
      mbar_poll(&full[(int)(c % ns)], (uint32_t)((c / ns) & 1), kFxWait);
  }
}

// One whole warp: lane k < nred gets the sum of reduction k's warp sums (a fixed tree).
__device__ __forceinline__ double fx_tile_sum(const double (&red)[kMaxRed][kFxWork / 32], int nred) {
  static_assert(kFxWork / 32 == 16, "two reductions per warp-wide add");
  const int lane = threadIdx.x & 31;
  double v = 0.0;
#pragma unroll 1
  for (int k = 0; k < nred; k += 2) {
    double a = red[k + (lane >> 4)][lane & 15];
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    const double a0 = __shfl_sync(0xffffffffu, a, 0), a1 = __shfl_sync(0xffffffffu, a, 16);
    if (lane == k) v = a0;
    if (lane == k + 1) v = a1;
  }
  return v;
}

// Warp 17: per matrix, once its B digits are written, the products of A digit i with the B digits
// j <= 6 - i into accumulator i + j, for 32 K values after the other.  The warp stays converged and
// its elected lane issues (elect_one).
template <int N, int MH>
__device__ __noinline__ void fx_issuer(FxResolve resolve, int64_t total, uint32_t ring, uint32_t b0, uint64_t* full,
                                       uint64_t* empty, uint64_t* dbar, uint64_t* bready, uint64_t* quiet,
                                       uint32_t tmem, volatile int* fail, const FxTabs* T, volatile int* handed) {
  using namespace tc;
  constexpr uint32_t bytes = kChunkRowBytes * MH;
  constexpr int ns = (int)(kRingBytes / bytes);
  constexpr uint32_t idesc = idesc_f16_nmajor(128, N);
  const uint64_t abits = smem_desc_bits(128, 512);
  const uint32_t el = elect_one();
  int s = 0;
  uint32_t phase = 0, nready = 0;
  bool ok = true;
  int ntile = 0, need = 0;  // tiles of this CTA, warps that have handed over by then
  for (int64_t gt = blockIdx.x; gt < total && ok; gt += gridDim.x, ++ntile) {
    const FxTile r = resolve(gt);
    const int kp = r.prm->kp, nk = kp / 32;
    // B: K rows of 16 bytes (eight columns), K groups of 8 rows 128 bytes apart, column groups
    // 16 kp apart, digits 2 N kp apart
    const uint64_t bbits = smem_desc_bits(128, (uint32_t)(16 * kp));
    const uint64_t bfirst = smem_desc_at(bbits, b0), bdig = (uint64_t)((2 * N * kp) >> 4);
    const int nmat = r.prm->nmat, handover = r.prm->handover;
    for (int m = 0; m <= nmat && ok; ++m) {
      if (m < nmat) {
        ok = __all_sync(0xffffffffu, mbar_poll(bready, nready & 1u, kFxWait));
        ++nready;
        tc_fence_after();
        uint64_t bk = bfirst;
        for (int q = 0; q < nk && ok; ++q) {
#pragma unroll
          for (int i = 0; i < kDigits; ++i) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_poll(&full[s], phase, kFxWait));
            if (!ok) break;
            tc_fence_after();
            const uint64_t a = smem_desc_at(abits, ring + (uint32_t)s * bytes);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
#pragma unroll
              for (int h = 0; h < MH; ++h)
#pragma unroll
                for (int j = 0; j < kDigits - i; ++j)
                  mma_f16_warp(tmem + (uint32_t)((i + j) * MH * N + h * N),
                               a + (uint64_t)(ks * (256 >> 4) + h * (kChunkRowBytes >> 4)),
                               bk + (uint64_t)(ks * (256 >> 4)) + (uint64_t)j * bdig, idesc,
                               (i | ks) != 0 || q != 0 ? 1u : 0u, el);
            if (el) mma_commit(&empty[s]);
            if (++s == ns) {
              s = 0;
              phase ^= 1u;
            }
          }
          bk += 512 >> 4;
        }
        if (ok && el) mma_commit(dbar);
      }
      if (ok && m == handover) {
        // the tile's norms, while the matrix just issued runs (m == nmat: after the tile)
        ok = await_handover(handed, need += kFxWork / 32, fail, kFxWait);
        if (ok) publish_tile(r.prm->p, r.tile, fx_tile_sum(T->red[ntile & 1], r.prm->p.nred));
      }
    }
  }
  if (!ok && el) {
    *fail = 1;
    // every MMA already issued completes before the tensor memory is released
    mma_commit(quiet);
    mbar_poll(quiet, 0u, kFxWait);
  }
}

// a b 2^-64 (b: digits), rounded
__device__ __forceinline__ i64 mulhi64(dig a, int2 b) {
  return mw(a.h, b.y, mw(a.h, b.x, mw(a.l, b.y, 1ll << 31)) >> 32);
}

// w = m 2^x, m in [1/2, 1): digits {l, h} of m 2^62; x is kFxPoison if w is not finite
struct RowWeight {
  int2 d;
  int x;
  __device__ __forceinline__ void set(double w) {
    int e = 0;
    const double m = frexp(w, &e);
    const dig q = split(isfinite(w) ? (i64)(m * 4611686018427387904.0) : 0);
    d = {q.l, q.h};
    x = isfinite(w) ? (w != 0.0 ? e : -kNoTerm) : kFxPoison;
  }
};

// v 2^e rounded as a store in FP64 would (fx_to_f64), in place; E: the biased exponent of the stored
// value (0 or less: zero or subnormal; 2047: infinite).  Subnormal values keep their 53 bits here: the check
// for them took 1 % of the pass, so among them a run in parts may differ by one unit of 2^-1074.
__device__ __forceinline__ i64 round_f64(i64 v, int e, int& E) {
  const i64 s = v >> 63;
  unsigned long long a = (unsigned long long)((v ^ s) - s);
  const int drop = 11 - __clzll((i64)a);
  if (drop > 0) a = ((a >> drop) + ((a >> (drop - 1)) & 1ull)) << drop;
  const int after = 63 - __clzll((i64)a) + e + 1023;  // one more after a carry
  E = a == 0 ? 0 : min(after, 2047);
  return ((i64)a ^ s) - s;
}
// ... and as the load of that value would scale it (raw_to_fx): v 2^-k
__device__ __forceinline__ i64 rescale_f64(i64 v, int k) {
  if (k <= 0) return v << (k < -63 ? 63 : -k);
  const i64 s = v >> 63;
  const unsigned long long a = (unsigned long long)((v ^ s) - s);
  const unsigned long long r = ((a >> (k > 64 ? 63 : k - 1)) + 1ull) >> 1;
  return ((i64)r ^ s) - s;
}

// (out of line: columns below 2^-962)
__device__ __noinline__ i64 cold_to_f64(i64 v, int e) { return fx_to_f64<true>(v, e); }

// The tile's tables of weights and factors (all but SCALE's); clears the column maxima.  All work threads.
template <bool EXPS>
__device__ __forceinline__ void fx_tables(FxTabs& T, const PassParams& p, int64_t o, int64_t i0, int ncols, int bn) {
  const Geometry& g = p.g;
  const int tid = threadIdx.x;
  if (tid < 2 * kFxMaxCols) T.cole[tid >> 5][tid & 31] = 0;
  if (tid < kFxTabSlots) T.nonident[tid] = 0;
  if (EXPS && tid == kFxWork - 1) T.kany = 0u;
  if (tid < p.nops) {
    int k = 0;
    for (int q = 0; q < tid; ++q) k += p.ops[q].kind == OP_DIAG1D && p.ops[q].axis != g.sweep_axis;
    T.slot[tid] = (int8_t)k;
  }
  fx_work_sync();
  for (int idx = tid; idx < p.nops * bn; idx += kFxWork) {
    const int oi = idx / bn, c = idx - oi * bn;
    const DevOp& op = p.ops[oi];
    const int64_t i = i0 + (c < ncols ? c : 0);
    if (op.kind == OP_NORM) {
      double wt = 1.0;
      for (int a = 0; a < g.ndim; ++a)
        if (a != g.sweep_axis) wt *= __ldg(op.w[a] + fx_coord(g, a, o, i));
      RowWeight cw;
      cw.set(wt);
      T.colwd[op.red][c] = cw.d;
      T.colwx[op.red][c] = cw.x;
    } else if (op.kind == OP_DIAG1D && op.axis != g.sweep_axis) {
      const int4 t = __ldg(reinterpret_cast<const int4*>(op.ptr) + fx_coord(g, op.axis, o, i));
      T.colt[T.slot[oi]][c] = t;
      const int kind = (t.x != 0 || t.y != (1 << 30) ? 1 : 0) | (t.z != 0 || t.w != 0 ? 3 : 0);
      if (kind) atomicOr(&T.nonident[T.slot[oi]], kind);
    }
    if (EXPS && (op.kind == OP_DIAGND || op.kind == OP_DIAG1D) && op.exps) {
      const int16_t k = c >= ncols ? 0 : __ldg(op.exps + (op.kind == OP_DIAGND ? o * g.inner + i : fx_coord(g, op.axis, o, i)));
      T.opk[oi][c] = k;
      if (k) atomicOr(&T.kany, 1u << oi);
    }
  }
}

// Op oi's factors are 2^opk too large: the columns' exponents go down.  All work threads.
__device__ __forceinline__ void lower_columns(FxTabs& T, int oi, int bn) {
  fx_work_sync();
  if ((int)threadIdx.x < bn && T.colx[threadIdx.x] != kFxPoison) T.colx[threadIdx.x] -= T.opk[oi][threadIdx.x];
  fx_work_sync();
}

// The work threads' view of a tile: row j, complex columns c0 .. c0 + NB - 1.
template <int NB, bool FF, bool EXPS>
struct FxWork {
  cx w[NB];
  int rowx;    // exponent of this row's values on top of their column's
  int xs;      // exponent from SCALE ops, of the whole tile
  int j, c0, ncols;
  int par;     // of the CTA's tiles: 0, 1, 0, ...
  bool row_ok;
  const double* roww_ptr;  // lane-axis weights of the pass's first norm, and this row's
  RowWeight roww;

  // this row's weight of the pass's first norm
  __device__ __forceinline__ void load_roww(const PassParams& p) {
    const int axis = p.g.sweep_axis;
    roww_ptr = nullptr;
    for (int oi = 0; oi < p.nops && roww_ptr == nullptr; ++oi)
      if (p.ops[oi].kind == OP_NORM) roww_ptr = p.ops[oi].w[axis];
    roww.set(roww_ptr && row_ok ? __ldg(roww_ptr + j) : 0.0);
  }

  // point-wise ops [ob, oe)
  __device__ __forceinline__ void apply(const PassParams& p, FxTabs& T, int ob, int oe, int64_t ix0, int bn) {
    const Geometry& g = p.g;
    for (int oi = ob; oi < oe; ++oi) {
      const DevOp& op = p.ops[oi];
      switch (op.kind) {
        case OP_DIAGND: {
          const int4* t = reinterpret_cast<const int4*>(op.ptr) + ix0;
          if (row_ok && c0 + NB <= ncols && aligned32(t)) {
#pragma unroll
            for (int u = 0; u < NB; u += 2) {
              int4 a, b;
              load_pair(t + u, a, b);
              w[u] = cmul<0>(w[u], a);
              w[u + 1] = cmul<0>(w[u + 1], b);
            }
          } else if (row_ok) {
#pragma unroll
            for (int u = 0; u < NB; ++u)
              if (c0 + u < ncols) w[u] = cmul<0>(w[u], __ldg(t + u));
          }
          if (EXPS && ((T.kany >> oi) & 1u)) lower_columns(T, oi, bn);
          break;
        }
        case OP_DIAG1D: {
          if (op.axis == g.sweep_axis) {
            if (row_ok) {
              const int4 t = __ldg(reinterpret_cast<const int4*>(op.ptr) + j);
#pragma unroll
              for (int u = 0; u < NB; ++u) w[u] = cmul<0>(w[u], t);
            }
          } else if (const int kind = T.nonident[T.slot[oi]]) {
            if (kind & 2) {
#pragma unroll
              for (int u = 0; u < NB; ++u) w[u] = cmul<0>(w[u], T.colt[T.slot[oi]][c0 + u]);
            } else {  // real factors (a mask)
#pragma unroll
              for (int u = 0; u < NB; ++u) {
                const int4 t = T.colt[T.slot[oi]][c0 + u];
                w[u] = cmul<0>(w[u], int4{t.x, t.y, 0, 0});
              }
            }
          }
          if (EXPS && ((T.kany >> oi) & 1u)) lower_columns(T, oi, bn);
          break;
        }
        case OP_SCALE: {
          const int2 d = T.scale_d[oi];
#pragma unroll
          for (int u = 0; u < NB; ++u) w[u] = cmul<0>(w[u], int4{d.x, d.y, 0, 0});
          xs += T.scale_x[oi];
          break;
        }
        case OP_NORM: {
          // Squares of the values moved up to 61 bits, in units of 2^64, times the column weights
          // (digits of m 2^62 and an exponent) over the largest column factor of the thread, times
          // the row's weight; the warp's sum over its largest row factor.  In integers throughout:
          // the FP64 pipe takes 1.7 operations a clock, so weights and sums in FP64 (three
          // operations a point, and their fold) took 5 us of a 32 x 128 tile.
          unsigned long long m = 0;
          int top = -kPoison;
#pragma unroll
          for (int u = 0; u < NB; ++u) {
            m |= (unsigned long long)(w[u].x ^ (w[u].x >> 63)) | (unsigned long long)(w[u].y ^ (w[u].y >> 63));
            top = max(top, T.colwx[op.red][c0 + u] + 2 * T.colx[c0 + u]);
          }
          const int lz = __clzll((i64)m), s = lz > 3 ? (lz < 60 ? lz - 3 : 57) : 0;
          i64 sum = 0;
#pragma unroll
          for (int u = 0; u < NB; ++u) {
            const dig a = split(w[u].x << s), b = split(w[u].y << s);
            const i64 q = mw(a.h, a.h, (mw(a.h, a.l, 1ll << 30)) >> 31) + mw(b.h, b.h, (mw(b.h, b.l, 1ll << 30)) >> 31);
            const int2 cw = T.colwd[op.red][c0 + u];
            sum += mulhi64(split(q << 2), cw) >> min(top - (T.colwx[op.red][c0 + u] + 2 * T.colx[c0 + u]), 63);
          }
          RowWeight rw = roww;
          if (op.w[g.sweep_axis] != roww_ptr) rw.set(row_ok ? __ldg(op.w[g.sweep_axis] + j) : 0.0);
          const bool bad = row_ok && max(top, rw.x) >= kPoison / 2;
          int e = -kPoison;  // the row's term is sum 2^e, |sum| < 2^60
          if (row_ok && sum != 0) {
            const int up = __clzll(sum ^ (sum >> 63)) - 2;  // |sum| <= 2^62
            sum = up >= 0 ? sum << up : sum >> 1;
            sum = mulhi64(split(sum), rw.d);
            if (sum != 0) e = 66 + 2 * (rowx + xs - s) + top + rw.x - max(up, -1);
          } else {
            sum = 0;
          }
          const int et = __reduce_max_sync(0xffffffffu, e);
          const bool any_bad = __any_sync(0xffffffffu, bad);
          i64 t = ((sum >> min(et - e, 60)) + 4) >> 3;  // 32 of them stay below 2^63
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
          if ((threadIdx.x & 31) == 0)
            T.red[par][op.red][threadIdx.x >> 5] =
                any_bad ? __longlong_as_double(0x7ff8000000000000ll) : scale_pow2((double)t, et + 3);
          break;
        }
        case OP_ROUND: {
          cx raw[NB];
          int mx[NB];
#pragma unroll
          for (int u = 0; u < NB; ++u) {
            const int x = T.colx[c0 + u];
            const bool ok = row_ok && c0 + u < ncols && x != kPoison;
            const int e = x + rowx + xs;
            int m;
            if constexpr (FF) {
              raw[u] = {ok ? fx_to_raw<FF>(w[u].x, e) : 0, ok ? fx_to_raw<FF>(w[u].y, e) : 0};
              m = max(raw_exp<FF>(raw[u].x), raw_exp<FF>(raw[u].y));
            } else {
              // FP64: rounded in place (packing and unpacking would only move the bits)
              const i64 re = ok ? w[u].x : 0, im = ok ? w[u].y : 0;
              int ex, ey;
              w[u] = {round_f64(re, e, ex), round_f64(im, e, ey)};
              m = max(ex, ey);
            }
            mx[u] = __reduce_max_sync(0xffffffffu, m);
          }
          if (threadIdx.x < 4 * NB) T.coler[threadIdx.x] = 0;
          int unit[NB];
#pragma unroll
          for (int u = 0; u < NB; ++u) unit[u] = T.colx[c0 + u] + rowx + xs;
          fx_work_sync();
#pragma unroll
          for (int u = 0; u < NB; ++u)
            if ((threadIdx.x & 31) == u) atomicMax(&T.coler[c0 + u], mx[u]);
          fx_work_sync();
          if (threadIdx.x < 4 * NB) {
            const int e = T.coler[threadIdx.x];
            if (e == 2047) T.colx[threadIdx.x] = kPoison;
            if (T.colx[threadIdx.x] != kPoison) T.colx[threadIdx.x] = max(e, kMinExp<FF>) - 1022 - 60;
          }
#pragma unroll
          for (int u = 0; u < NB; ++u) {
            const int e = max(T.coler[c0 + u], kMinExp<FF>);
            const bool live = e != 2047;
            if constexpr (FF) {
              w[u] = {live ? raw_to_fx<FF>(raw[u].x, e - 1022) : 0, live ? raw_to_fx<FF>(raw[u].y, e - 1022) : 0};
            } else {
              const int k = e - 1082 - unit[u];
              w[u] = {live ? rescale_f64(w[u].x, k) : 0, live ? rescale_f64(w[u].y, k) : 0};
            }
          }
          rowx = 0;
          xs = 0;
          fx_work_sync();
          break;
        }
        default:
          break;
      }
    }
  }
  static constexpr int kPoison = kFxPoison;

  // B digits of the values, K row j: v = value 2^(55 - colb) as seven digits
  __device__ __forceinline__ void write_operand(const FxTabs& T, unsigned char* B, int kp, uint32_t bbytes) {
    if (j >= kp) return;
#pragma unroll
    for (int u4 = 0; u4 < NB; u4 += 4) {
      constexpr int kU = NB < 4 ? NB : 4;
      uint32_t re[kU][2], im[kU][2];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int c = c0 + u4 + u;
        const int x = T.colx[c];
        const int sh = (x == kPoison ? 0 : x) + rowx + xs + 55 - T.colb[c];
        const i64 a = shift_by(w[u4 + u].x, sh) + 0x0080808080808080ll;
        const i64 b = shift_by(w[u4 + u].y, sh) + 0x0080808080808080ll;
        re[u][0] = (uint32_t)a;
        re[u][1] = (uint32_t)(a >> 32);
        im[u][0] = (uint32_t)b;
        im[u][1] = (uint32_t)(b >> 32);
      }
      // complex column c: real columns 2 c, 2 c + 1; column group (2 c) / 8
      unsigned char* dst = B + (uint32_t)((c0 + u4) >> 2) * (uint32_t)(16 * kp) + (uint32_t)(j >> 3) * 128u +
                           (uint32_t)(j & 7) * 16u + (uint32_t)((c0 + u4) & 3) * 4u;
#pragma unroll
      for (int d = 0; d < kDigits; ++d) {
        uint32_t v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) v[u] = digit_pair(re[u], im[u], d);
        if constexpr (kU == 4)
          *reinterpret_cast<uint4*>(dst + (uint32_t)d * bbytes) = make_uint4(v[0], v[1], v[2], v[3]);
        else
          *reinterpret_cast<uint2*>(dst + (uint32_t)d * bbytes) = make_uint2(v[0], v[1]);
      }
    }
  }
};

// EXPS: tables with an exponent per column (Engine::fx_table).  A kernel of its own: asking every op
// whether it has them took 1 us of a 25 us pass (256 x 64 points with a matrix per Omega).
template <int NB, int MH, bool FF, bool EXPS>
__global__ void __launch_bounds__(kFxThreads, 1)
    fx_angular_kernel(const __grid_constant__ FxTcParams one, const FxTcParams* __restrict__ params,
                      const uint2* __restrict__ owners, const int64_t total) {
  using namespace tc;
  constexpr int kGroups = MH == 1 ? 4 : 2;     // column groups of the work warps
  constexpr int BN = NB * kGroups, N = 2 * BN;
  constexpr int kRing = (int)(kRingBytes / (kChunkRowBytes * MH));
  using Work = FxWork<NB, FF, EXPS>;
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ __align__(16) FxTcParams tp;
  __shared__ __align__(16) FxTabs T;
  __shared__ __align__(8) uint64_t bars[2 * 8 + 3];
  __shared__ uint32_t tmem_s;
  __shared__ volatile int s_fail, s_handed;
  __shared__ int s_bad;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (blockIdx.x >= total) {
    wait_for_previous();
    return;
  }
  const FxResolve resolve{&one, params, owners};
  uint64_t *full = bars, *empty = bars + kRing, *dbar = bars + 2 * kRing, *bready = dbar + 1, *quiet = dbar + 2;
  if (tid == 0) {
    for (int k = 0; k < 2 * kRing; ++k) mbar_init(bars + k, 1);
    mbar_init(dbar, 1);
    mbar_init(bready, kFxWork);
    mbar_init(quiet, 1);
    fence_mbar_init();
    s_fail = 0;
    s_handed = 0;
    s_bad = 0;
  }
  if (warp == 0) tmem_alloc(&tmem_s, 512);
  // (ahead of the wait below: the parameters are no memory of the kernel before)
  if (params == nullptr)
    for (int k = tid; k < (int)(sizeof(FxTcParams) / 4); k += kFxThreads)
      reinterpret_cast<uint32_t*>(&tp)[k] = reinterpret_cast<const uint32_t*>(&one)[k];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s;
  const uint32_t ring = smem_u32(sm);
  unsigned char* B = sm + kRingBytes;

  if (warp == kFxWork / 32) {
    wait_for_previous();
    if (lane == 0) fx_producer<MH>(resolve, total, ring, full, empty, &s_fail);
  } else if (warp == kFxWork / 32 + 1) {
    wait_for_previous();
    fx_issuer<N, MH>(resolve, total, ring, ring + kRingBytes, full, empty, dbar, bready, quiet, tmem, &s_fail, &T,
                     &s_handed);
  } else {
    const int quad = warp & 3, grp = warp >> 2;
    Work W;
    W.j = (MH == 2 ? 128 * (grp >> 1) : 0) + 32 * quad + lane;
    W.c0 = NB * (MH == 2 ? (grp & 1) : grp);
    // this thread's accumulator columns: half (MH = 2) grp >> 1, real columns 2 c0 ..
    const uint32_t tcol = tmem + ((uint32_t)(32 * quad) << 16) + (uint32_t)((MH == 2 ? (grp >> 1) * N : 0) + 2 * W.c0);
    uint32_t drains = 0;
    const FxTcParams* cur = params == nullptr ? &one : nullptr;
    W.par = 1;
    // A single pass makes its first tile's tables while the launch ahead drains: they are constants,
    // complete before this launch was made (the host waits for every upload of one).  That takes a
    // block that fits beside the launch ahead (half of an SM's shared memory, one_block_per_sm); one
    // that starts behind it overlaps them with the loads of the tile instead.  us per step, tables
    // with the loads / ahead: 2048 x 64 61.2 / 59.3, state matrix 256 x 64 x 4 33.5 / 31.8 (both fit),
    // 4096 x 128 83.5 / 85.8 (does not).
    // (The widest tiles, 8 columns a thread, fit for 32 rows alone and always take the second way.)
    bool tabled = NB < 8 && params == nullptr && fx_tc_smem(BN, tp.kp) <= 100 * 1024;
    if (tabled) {
      const Geometry& g = tp.p.g;
      const int64_t o = blockIdx.x / g.tiles_per_outer, i0 = (blockIdx.x - o * g.tiles_per_outer) * BN;
      W.row_ok = W.j < (int)g.n;
      W.load_roww(tp.p);
      fx_tables<EXPS>(T, tp.p, o, i0, (int)min((int64_t)BN, g.inner - i0), BN);
    }
    wait_for_previous();
    for (int64_t gt = blockIdx.x; gt < total; gt += gridDim.x) {
      W.par ^= 1;
      const FxTile r = resolve(gt);
      if (r.prm != cur) {
        for (int k = tid; k < (int)(sizeof(FxTcParams) / 4); k += kFxWork)
          reinterpret_cast<uint32_t*>(&tp)[k] = reinterpret_cast<const uint32_t*>(r.prm)[k];
        cur = r.prm;
        fx_work_sync();
      }
      const PassParams& p = tp.p;
      const Geometry& g = p.g;
      const int n = (int)g.n, kp = tp.kp;
      const uint32_t bbytes = fx_b_bytes(BN, kp);
      // products are drained with 2^-sh of their last bit: |product| <= 2^61
      const int sh = kp <= 32 ? 6 : (kp <= 64 ? 7 : (kp <= 128 ? 8 : 9));
      const int64_t o = r.tile / g.tiles_per_outer;
      const int64_t i0 = (r.tile - o * g.tiles_per_outer) * BN;
      const int64_t left = g.inner - i0;
      W.ncols = left < BN ? (int)left : BN;
      W.row_ok = W.j < n;
      W.xs = 0;
      W.rowx = 0;
      const int64_t ix0 = o * g.n * g.inner + (int64_t)W.j * g.inner + i0 + W.c0;
      longlong2* psi = reinterpret_cast<longlong2*>(p.psi) + ix0;

      // the tile's values
      cx raw[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) raw[u] = {0, 0};
      const bool whole = W.row_ok && W.c0 + NB <= W.ncols && aligned32(psi);
      if (whole) {
#pragma unroll
        for (int u = 0; u < NB; u += 2) load_pair(psi + u, raw[u], raw[u + 1]);
      } else if (W.row_ok) {
#pragma unroll
        for (int u = 0; u < NB; ++u)
          if (W.c0 + u < W.ncols) {
            const longlong2 x = psi[u];
            raw[u] = {x.x, x.y};
          }
      }
      if (!tabled) W.load_roww(p);
      if (!tabled) fx_tables<EXPS>(T, p, o, i0, W.ncols, BN);
      tabled = false;
      if (tid < p.nops && p.ops[tid].kind == OP_SCALE) {
        // sqrt(target / norm) = m 2^x, m in [1/2, 1): digits of m 2^62
        const double f = sqrt(__ldcg(p.slots + p.ops[tid].b) / __ldcg(p.slots + p.ops[tid].c));
        int x = 0;
        const double m = frexp(f, &x);
        i64 v = isfinite(f) ? __double2ll_rn(ldexp(m, 62)) : 0;
        if ((int)v == (int)0x80000000) ++v;
        const dig d = split(v);
        T.scale_d[tid] = {d.l, d.h};
        T.scale_x[tid] = x;
        if (!isfinite(f)) s_bad = 1;  // the whole tile becomes NaN
      }
      // column exponents
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int m = __reduce_max_sync(0xffffffffu, max(raw_exp<FF>(raw[u].x), raw_exp<FF>(raw[u].y)));
        if (lane == u) atomicMax(&T.cole[0][W.c0 + u], m);
      }
      fx_work_sync();
      if (tid < BN) {
        const int e = T.cole[0][tid];
        T.colx[tid] = e == 2047 || s_bad ? Work::kPoison : max(e, kMinExp<FF>) - 1022 - 60;
        T.colb[tid] = max(e, kMinExp<FF>) - 1022;
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int e = max(T.cole[0][W.c0 + u], kMinExp<FF>);
        const bool live = e != 2047 && !s_bad;
        W.w[u] = {live ? raw_to_fx<FF>(raw[u].x, e - 1022) : 0, live ? raw_to_fx<FF>(raw[u].y, e - 1022) : 0};
      }
      fx_work_sync();  // the exponents and tables are complete
      bool ok = true;
      for (int m = -1; m < tp.nmat && ok; ++m) {
        if (m >= 0) {
          // drain matrix m
          ok = fx_work_all(mbar_wait(dbar, drains & 1u, kFxWait));
          if (!ok) break;
          ++drains;
          tc_fence_after();
          const unsigned char* img = fx_image(tp, m, r.tile);
          W.rowx = __ldg(reinterpret_cast<const int*>(img + (size_t)kDigits * (kp / 32) * kChunkRowBytes * MH) + W.j);
          W.xs = 0;
          if (tid < BN) {
            T.colx[tid] = T.colx[tid] == Work::kPoison ? Work::kPoison : T.colb[tid] + sh - 62;
            T.cole[0][tid] = 0;
          }
#pragma unroll
          for (int u = 0; u < NB; u += 2) {
            uint32_t rg[28];
            tmem_ld4x7(tcol + 2u * u, (uint32_t)(MH * N), rg);
            float mx = 0.0f;
#pragma unroll
            for (int k = 0; k < 28; ++k) mx = fmaxf(mx, fabsf(__uint_as_float(rg[k])));
            int v[28];
            if (mx <= 4194304.0f) {
              // |sum| <= 2^22: the FP32 addition of 1.5 2^23 leaves the integer in the low bits
#pragma unroll
              for (int k = 0; k < 28; ++k)
                v[k] = __float_as_int(__fadd_rn(__uint_as_float(rg[k]), 12582912.0f)) - 0x4B400000;
            } else {
#pragma unroll
              for (int k = 0; k < 28; ++k) v[k] = __float2int_rn(__uint_as_float(rg[k]));
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              W.w[u + q].x = combine<MH>(v[2 * q], v[4 + 2 * q], v[8 + 2 * q], v[12 + 2 * q], v[16 + 2 * q],
                                         v[20 + 2 * q], v[24 + 2 * q], sh);
              W.w[u + q].y = combine<MH>(v[2 * q + 1], v[5 + 2 * q], v[9 + 2 * q], v[13 + 2 * q], v[17 + 2 * q],
                                         v[21 + 2 * q], v[25 + 2 * q], sh);
            }
          }
          tc_fence_before();
          fx_work_sync();  // colx is complete
        }
        const int ob = m < 0 ? 0 : tp.mat_op[m] + 1;
        const int oe = m + 1 < tp.nmat ? tp.mat_op[m + 1] : p.nops;
        W.apply(p, T, ob, oe, ix0, BN);
        if (m + 1 < tp.nmat) {
          if (m >= 0 || oe > 0) {
            // the operand's column maxima
            int* ce = T.cole[m < 0 ? 1 : 0];  // set 0 was cleared with the drain
#pragma unroll
            for (int u = 0; u < NB; ++u) {
              const int b = W.row_ok ? bits_of(W.w[u].x, W.w[u].y) : 0;
              const int e = b ? b + W.rowx + 8192 : 0;
              const int mx = __reduce_max_sync(0xffffffffu, e);
              if (lane == u) atomicMax(ce + W.c0 + u, mx);
            }
            fx_work_sync();
            if (tid < BN) {
              const int e = ce[tid], x = T.colx[tid];
              T.colb[tid] = (e ? e - 8192 : 0) + (x == Work::kPoison ? 0 : x) + W.xs;
            }
            fx_work_sync();
          }
          W.write_operand(T, B, kp, bbytes);
          fence_proxy_async();
          mbar_arrive(bready);
        }
        // the tile's norms are complete: the issuing warp publishes them
        if (m + 1 == tp.handover && lane == 0) hand_over(&s_handed);
      }
      if (!ok) {
        if (tid == 0) s_fail = 1;
        break;
      }
      // store
      bool low = false;
      if constexpr (!FF) {
#pragma unroll
        for (int u = 0; u < NB; ++u) low = low || T.colx[W.c0 + u] + W.rowx + W.xs < kLowExp;
      }
      auto packed = [&](auto&& f) {
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const int x = T.colx[W.c0 + u], e = x + W.rowx + W.xs;
          W.w[u] = {f(W.w[u].x, e), f(W.w[u].y, e)};
          if (x == Work::kPoison) W.w[u] = {raw_nan<FF>(), raw_nan<FF>()};
        }
      };
      if (!FF && __builtin_expect(low, 0))
        packed([](i64 v, int e) { return cold_to_f64(v, e); });
      else
        packed([](i64 v, int e) { return fx_to_raw<FF, false>(v, e); });
      if (whole) {
#pragma unroll
        for (int u = 0; u < NB; u += 2) store_pair(psi + u, W.w[u], W.w[u + 1]);
      } else if (W.row_ok) {
#pragma unroll
        for (int u = 0; u < NB; ++u)
          if (W.c0 + u < W.ncols) psi[u] = longlong2{W.w[u].x, W.w[u].y};
      }
      if (tid == 0) s_bad = 0;
      fx_work_sync();  // the tables and the pass copy are free for the next tile
    }
  }
  __syncthreads();
  if (tid == 0 && s_fail) {
    const FxTcParams* f0 = resolve(blockIdx.x).prm;  // the pass of the first tile records the failure
    if (f0->error_slot >= 0) f0->p.slots[f0->error_slot] = 1.0;
  }
  // teardown: every MMA has completed (drained, or waited on by the MMA warp)
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace
}  // namespace so
