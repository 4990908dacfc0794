// The end of a pass: the CTA that draws its last ticket folds the norm partials of all tiles and
// runs the pass's scalar bookkeeping (norm slots, loss accumulation, slot copies).
//
// Every pass waits for this, and it is all latency: one lane that walks the ops and the slots in
// global memory makes a dependent round trip (0.4 - 0.7 us) of nearly every access.  Here one warp
// takes it: lane i holds op i and the slots that op reads, loaded while the ticket is under way;
// the partials come all at once; the program then runs in registers, each op's result handed by
// shuffles to the lanes whose op reads that slot, and the stores are not waited for.
#pragma once
#include "common.cuh"

namespace so {

// The first lane matrix (0 .. nmat; nmat: the end of the tile) by whose product a tile's norms are
// complete and its factors from slots taken: there the tile hands its partials over, and the
// chain below runs beside the rest of the tile.
inline int pass_handover(const PassParams& p, const int* mat_op, int nmat) {
  int last = -1;
  for (int i = 0; i < p.nops; ++i)
    if (p.ops[i].kind == OP_NORM || p.ops[i].kind == OP_SCALE) last = i;
  int m = 0;
  while (m < nmat && last > mat_op[m]) ++m;
  return m;
}

namespace {

static_assert(kMaxOps <= 32 && kMaxRed == 8, "one lane per op; three halving levels");

// The program: lane i holds op i (kind -1: nothing to do) and the slots it reads.
struct EndOp {
  int kind, sa, sb, sc, red;
  double va, vb, vc, value;
  int64_t count;
  // p may lie in any memory.  Nobody writes the pass's slots before its last ticket is drawn, so
  // this runs ahead of the caller's own ticket and overlaps its round trip.
  __device__ __forceinline__ void load(const PassParams& p) {
    const int lane = threadIdx.x & 31;
    kind = -1;
    sa = sb = sc = -1;
    red = 0;
    count = 0;
    va = vb = vc = value = 0.0;
    if (lane < p.nops) {
      const DevOp& o = p.ops[lane];
      const int k = o.kind;
      if (k == OP_NORM || k == OP_DOT || k == OP_COPY || k == OP_LOSS || k == OP_SETC || k == OP_RECORD) {
        kind = k;
        sa = o.a;
        sb = o.b;
        sc = o.c;
        red = o.red;
        count = o.count;
        value = o.value;
      }
    }
    if (kind == OP_LOSS || kind == OP_RECORD) va = __ldcg(p.slots + sa);
    if (kind == OP_LOSS || kind == OP_COPY) vb = __ldcg(p.slots + sb);
    if (kind == OP_LOSS) vc = __ldcg(p.slots + sc);
  }
};

// One whole warp, after its last ticket: sums over the tiles of the pass's reductions (fixed
// order: lane l adds tiles l, l + 32, ...; then a fixed tree), then the scalar program.
__device__ __forceinline__ void finish_pass(const PassParams& p, EndOp& op, const double* part, int64_t tiles) {
  const int lane = threadIdx.x & 31;
  const int nred = p.nred;
  double* const slots = p.slots;
  double* const record = p.record;
  const int nonfinite = p.nonfinite_slot;
  unsigned int* const counter = p.counter;
  const int kind = op.kind, sa = op.sa, sb = op.sb, sc = op.sc, red = op.red;
  const double value = op.value;
  const int64_t count = op.count;
  double &va = op.va, &vb = op.vb, &vc = op.vc;
  double t[kMaxRed];
#pragma unroll
  for (int k = 0; k < kMaxRed; ++k) t[k] = 0.0;
  for (int64_t b0 = lane; b0 < tiles; b0 += 128) {
    // four tiles of four reductions in flight
#pragma unroll
    for (int k4 = 0; k4 < kMaxRed; k4 += 4) {
      if (k4 >= nred) break;
      double v[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          v[k][u] = 0.0;
          if (k4 + k < nred && b0 + 32 * u < tiles) v[k][u] = __ldcg(part + (int64_t)(k4 + k) * tiles + b0 + 32 * u);
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (b0 - lane + 32 * u < tiles) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k4 + k < nred) t[k4 + k] += v[k][u];
        }
    }
  }
  // The trees of all reductions at once: at each of the first three levels a lane keeps half of
  // its reductions (the adds of a whole warp take some 70 clocks on the FP64 pipe: 9 instead
  // of 5 per reduction).  Lane l ends with reduction 4 bit4(l) + 2 bit3(l) + bit2(l).
  const int h4 = (lane >> 4) & 1, h3 = (lane >> 3) & 1, h2 = (lane >> 2) & 1;
  double t4[4], t2[2];
#pragma unroll
  for (int k = 0; k < 4; ++k) t4[k] = (h4 ? t[4 + k] : t[k]) + __shfl_xor_sync(0xffffffffu, h4 ? t[k] : t[4 + k], 16);
#pragma unroll
  for (int k = 0; k < 2; ++k) t2[k] = (h3 ? t4[2 + k] : t4[k]) + __shfl_xor_sync(0xffffffffu, h3 ? t4[k] : t4[2 + k], 8);
  double tr = (h2 ? t2[1] : t2[0]) + __shfl_xor_sync(0xffffffffu, h2 ? t2[0] : t2[1], 4);
  tr += __shfl_xor_sync(0xffffffffu, tr, 2);
  tr += __shfl_xor_sync(0xffffffffu, tr, 1);
  // this lane's reductions
  const int r1 = red + 1;
  const double t0 = __shfl_sync(0xffffffffu, tr, ((red & 4) << 2) | ((red & 2) << 2) | ((red & 1) << 2));
  const double t1 = __shfl_sync(0xffffffffu, tr, ((r1 & 4) << 2) | ((r1 & 2) << 2) | ((r1 & 1) << 2));
  for (unsigned left = __ballot_sync(0xffffffffu, kind >= 0); left; left &= left - 1) {
    // op i: the value of its slot a (a DOT also sets its slot b)
    const int i = __ffs(left) - 1;
    const int k_i = __shfl_sync(0xffffffffu, kind, i);
    if (k_i == OP_RECORD) {
      if (lane == i && record) record[count] = va;
      continue;
    }
    double v = t0;
    if (k_i == OP_COPY) v = vb;
    if (k_i == OP_SETC) v = value;
    if (k_i == OP_LOSS) v = va + (vb - vc);
    if (lane == i) {
      slots[sa] = v;
      if (k_i == OP_DOT) slots[sb] = t1;
      if (k_i == OP_NORM && !isfinite(v) && nonfinite >= 0) slots[nonfinite] = 1.0;
    }
    const int a_i = __shfl_sync(0xffffffffu, sa, i);
    const double v_i = __shfl_sync(0xffffffffu, v, i);
    if (sa == a_i) va = v_i;
    if (sb == a_i) vb = v_i;
    if (sc == a_i) vc = v_i;
    if (k_i == OP_DOT) {
      const int b_i = __shfl_sync(0xffffffffu, sb, i);
      const double w_i = __shfl_sync(0xffffffffu, t1, i);
      if (sa == b_i) va = w_i;
      if (sb == b_i) vb = w_i;
      if (sc == b_i) vc = w_i;
    }
    __syncwarp();  // stores of one slot by two lanes stay in program order
  }
  if (lane == 0) *counter = 0u;
}

// The tensor-core kernels' warps that issue products are idle between two of them, and take a
// tile's partials from there: the work warps leave their warp sums in shared memory, count
// themselves in, and go on with the tile.  On the work warps' own path the ticket took 3 us of
// every pass, and the last CTA's fold another 5.
__device__ __forceinline__ void hand_over(volatile int* handed) {  // lane 0 of a work warp
  __threadfence_block();
  atomicAdd(const_cast<int*>(handed), 1);
}
// One whole warp: waits until `need` warps have handed over (false after limit_ns, or on *fail).
__device__ __forceinline__ bool await_handover(volatile int* handed, int need, volatile int* fail,
                                               unsigned long long limit_ns) {
  unsigned long long t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  while (__any_sync(0xffffffffu, *handed < need)) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (__any_sync(0xffffffffu, *fail != 0 || t1 - t0 > limit_ns)) return false;
    __nanosleep(40);
  }
  __threadfence_block();
  return true;
}
// One whole warp: the tile's partials (lane k: reduction k) and its ticket; the last one finishes
// the pass.  p may lie in any memory.
__device__ __noinline__ void publish_tile(const PassParams& p, int64_t tile, double v) {
  const int lane = threadIdx.x & 31;
  double* const part = p.partials;
  const int64_t tiles = p.g.tiles;
  EndOp end;
  end.load(p);
  if (lane < p.nred) part[(int64_t)lane * tiles + tile] = v;
  __syncwarp();
  unsigned int last = 0u;
  if (lane == 0) {
    __threadfence();
    last = atomicAdd(p.counter, 1u) == (unsigned int)(tiles - 1) ? 1u : 0u;
  }
  last = __shfl_sync(0xffffffffu, last, 0);
  if (!last) return;
  __threadfence();
  finish_pass(p, end, part, tiles);
}

}  // namespace
}  // namespace so
