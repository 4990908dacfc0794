// Fixed-point lane-matrix pass (angular_fx.cuh): digit images, planning, and the FP64 kernels.
#include <cmath>
#include <cstring>
#include <vector>

#include "angular_fx.cuh"
#include "angular_fx_launch.cuh"

namespace so {

static int fx_halves(int n) { return n > 128 ? 2 : 1; }
static int fx_kp(int n) { return (n + 31) / 32 * 32; }
static size_t fx_digit_bytes(int n) { return (size_t)kDigits * (fx_kp(n) / 32) * kChunkRowBytes * fx_halves(n); }

size_t fx_angular_image_bytes(int n) { return fx_digit_bytes(n) + sizeof(int32_t) * 128 * fx_halves(n); }

// FP16 bits of an integer of magnitude <= 128
static uint16_t half_of(int v) {
  if (v == 0) return 0;
  const unsigned a = v < 0 ? -v : v;
  int e = 0;
  while (a >> (e + 1)) ++e;  // a in [2^e, 2^(e + 1))
  return (uint16_t)((v < 0 ? 0x8000u : 0u) | ((unsigned)(e + 15) << 10) | ((a << (10 - e)) & 0x3ffu));
}

// Digit images of one real n x n matrix (row-major, out[r] = sum_k m[r][k] in[k]): digit by
// digit, chunk by chunk (32 K values), rows in the K-major core-matrix order (8 rows x 16
// bytes, K groups 128 bytes apart, row groups 512 bytes apart); then the rows' exponents e,
// |m[r][k]| < 2^e.  False when a value is not finite, or when the matrix is sparse (a row with
// values, more than half of them zero): the products are accurate relative to a column's
// largest value, as FP64's are where every value enters every sum, but an identity or
// block-diagonal matrix keeps small values beside large ones exact in FP64.
bool fx_angular_image(const double* m, int n, unsigned char* out) {
  const int mh = fx_halves(n), rows = 128 * mh, kp = fx_kp(n), nk = kp / 32;
  std::memset(out, 0, fx_angular_image_bytes(n));
  int32_t* ex = reinterpret_cast<int32_t*>(out + fx_digit_bytes(n));
  (void)rows;
  for (int r = 0; r < n; ++r) {
    double amax = 0.0;
    for (int k = 0; k < n; ++k) {
      const double a = std::fabs(m[(size_t)r * n + k]);
      if (!std::isfinite(a)) return false;
      amax = a > amax ? a : amax;
    }
    int e = 0, nonzero = 0;
    if (amax > 0.0) std::frexp(amax, &e);
    ex[r] = e;
    for (int k = 0; k < n; ++k) nonzero += std::fabs(m[(size_t)r * n + k]) > std::ldexp(amax, -53);
    if (amax > 0.0 && 2 * nonzero <= n) return false;
    for (int k = 0; k < n; ++k) {
      const int64_t v = (int64_t)std::llround(std::ldexp(m[(size_t)r * n + k], 55 - e)) + 0x0080808080808080ll;
      const size_t off = (size_t)(r >> 3) * 512 + (size_t)((k % 32) / 8) * 128 + (size_t)(r & 7) * 16 + (size_t)(k % 8) * 2;
      for (int d = 0; d < kDigits; ++d) {
        const int digit = (int)(d == 0 ? v >> 48 : (v >> (8 * (6 - d))) & 0xff) - 128;
        const uint16_t h = half_of(digit);
        std::memcpy(out + ((size_t)d * nk + k / 32) * kChunkRowBytes * mh + off, &h, 2);
      }
    }
  }
  return true;
}

// Columns per tile: the widest tile reads the digit images least often, but a pass of few tiles
// is done soonest when every SM has one.  Relative tile times 1, 0.65, 0.45 (a 32-, 16- and
// 8-column tile of 128 rows: the products take 51, 40 and 36 clocks each, the rest is per column).
static int fx_columns(const Geometry& g, int64_t stride, int sms) {
  const int most = g.n > 128 ? 16 : 32;
  int best = 0;
  double cost = 0.0;
  for (int bn = most; bn >= 8; bn /= 2) {
    if (stride % bn != 0) continue;
    const int64_t tiles = g.outer * ((g.inner + bn - 1) / bn);
    const double t = (double)((tiles + sms - 1) / sms) * (bn == most ? 1.0 : (2 * bn == most ? 0.65 : 0.45));
    if (best == 0 || t < cost) {
      best = bn;
      cost = t;
    }
  }
  return best;
}

bool fx_angular_plan(PassParams& p, const DevOp* ops, int nops, const double* table_max, int* cols) {
  Geometry& g = p.g;
  if (g.n < 16 || g.n > 256) return false;
  int mats = 0, across = 0;
  int64_t stride = 0;  // columns that share a state matrix (0: any tile width)
  double prod = 1.0;
  for (int i = 0; i < nops; ++i) {
    const DevOp& op = ops[i];
    switch (op.kind) {
      case OP_MAT_SLICE: {
        // the dependent coordinate is constant over a tile when it is an outer axis, or an inner
        // one whose stride is a multiple of the tile's columns
        int q = -1;
        for (int a = 0; a < g.ndim; ++a)
          if (g.perm[a] == op.axis) q = a;
        if (q < 0 || q == g.spos || op.count < g.sshape[q]) return false;
        if (q > g.spos) {
          int64_t s = 1;
          for (int a = q + 1; a < g.ndim; ++a) s *= g.sshape[a];
          stride = s;
        }
        ++mats;
        break;
      }
      case OP_MAT: ++mats; break;
      case OP_DIAG1D: across += op.axis != g.sweep_axis; [[fallthrough]];
      case OP_DIAGND:
        // (a table that is not finite has the maximum infinity)
        if (!(table_max[i] >= kMinTable && table_max[i] <= kMaxTable)) return false;
        prod *= table_max[i] > 1.0 ? table_max[i] : 1.0;
        break;
      case OP_FFT: case OP_MAT_LANE: case OP_DOT: return false;
      default: break;
    }
  }
  if (mats < 1 || mats > 2 || across > kFxTabSlots || !(prod <= kMaxProduct)) return false;
  const int bn = fx_columns(g, stride, sm_count());
  if (bn == 0) return false;
  g.lanes_per_tile = bn;
  g.tiles_per_outer = (int32_t)((g.inner + bn - 1) / bn);
  g.tiles = g.outer * g.tiles_per_outer;
  if (g.tiles >= (int64_t)0xffffffff) return false;
  *cols = bn;
  return true;
}

size_t fx_angular_params_bytes() { return sizeof(FxTcParams); }

void fx_angular_params(const PassParams& p, const int* mat_op, int nmat, const unsigned char* const* images,
                       const int* slice_axis, int error_slot, void* out) {
  FxTcParams t{};
  t.p = p;
  t.nmat = nmat;
  t.handover = pass_handover(p, mat_op, nmat);
  t.kp = fx_kp((int)p.g.n);
  t.error_slot = error_slot;
  const Geometry& g = p.g;
  for (int m = 0; m < 2; ++m) {
    t.slice_axis[m] = -1;
    if (m >= nmat) continue;
    t.mat_op[m] = mat_op[m];
    t.images[m] = images[m];
    if (slice_axis[m] < 0) continue;
    int q = 0;
    for (int a = 0; a < g.ndim; ++a)
      if (g.perm[a] == slice_axis[m]) q = a;
    int64_t div = 1;
    if (q < g.spos) {
      for (int a = q + 1; a < g.spos; ++a) div *= g.sshape[a];
      t.slice_pre[m] = 0;
      t.slice_div[m] = (uint32_t)(div * g.tiles_per_outer);
    } else {
      for (int a = q + 1; a < g.ndim; ++a) div *= g.sshape[a];
      t.slice_pre[m] = (uint32_t)g.tiles_per_outer;
      t.slice_div[m] = (uint32_t)(div / g.lanes_per_tile);
    }
    t.slice_ext[m] = (uint32_t)g.sshape[q];
    t.slice_axis[m] = slice_axis[m];
    t.slice_stride[m] = (int64_t)fx_angular_image_bytes((int)g.n);
  }
  std::memcpy(out, &t, sizeof(t));
}

cudaError_t launch_fx_angular(int real, int n, int cols, bool exps, const void* one, const void* params_dev,
                              const void* owners_dev, int64_t tiles, cudaStream_t s) {
  const unsigned grid = (unsigned)(tiles < sm_count() ? tiles : sm_count());
  const FxTcParams* prm = reinterpret_cast<const FxTcParams*>(params_dev);
  const uint2* own = reinterpret_cast<const uint2*>(owners_dev);
  FxAngularLaunch* const launch = real == kRealFF ? (exps ? launch_fx_angular_ff_exps : launch_fx_angular_ff)
                                                  : (exps ? launch_fx_angular_exps : fx_angular_launch<false, false>);
  return launch(fx_halves(n), fx_kp(n), cols, one, prm, own, tiles, grid, s);
}

int64_t fx_angular_grid(int64_t tiles) { return tiles < sm_count() ? tiles : sm_count(); }

}  // namespace so
