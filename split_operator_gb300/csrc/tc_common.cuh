// Inline-PTX helpers for sm_103a tensor-core passes: mbarriers with bounded
// waits, bulk (TMA) copies, TMEM allocation, tcgen05.mma / commit / ld, and the
// shared-memory / instruction descriptors of kind::tf32 with K-major operands in
// the no-swizzle "core matrix" layout (8 rows x 16 bytes per core matrix; LBO =
// byte step between core matrices along K, SBO = byte step between 8-row groups).
#pragma once
#include <cstdint>

#include <cuda_bf16.h>

namespace so {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// generic pointer of a shared-memory address (inverse of smem_u32)
__device__ __forceinline__ void* sm_ptr(uint32_t a) { return __cvta_shared_to_generic(a); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One bounded try: the thread may be suspended (not spinning, so it takes no issue slots
// from the warps doing work) until the phase completes or about 20 us pass.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase), "r"(20000u)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// try_wait without a suspend hint: returns promptly (the single issuing lanes poll with it,
// so they see a completed phase without a wake-up delay)
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}

// Bounded polling wait for a single lane: false after `limit_ns` without completion.
__device__ __forceinline__ bool mbar_poll(uint64_t* bar, uint32_t phase, uint64_t limit_ns) {
  if (mbar_test(bar, phase)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (true) {
    if (mbar_test(bar, phase)) return true;
    if (globaltimer_ns() - t0 > limit_ns) return false;
  }
}

// Bounded wait: false when `limit_ns` nanoseconds passed without the phase completing.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t phase, uint64_t limit_ns) {
  if (mbar_try_wait(bar, phase)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (true) {
    if (mbar_try_wait(bar, phase)) return true;
    if (globaltimer_ns() - t0 > limit_ns) return false;
  }
}

// 1-D bulk copy global -> shared completing on `bar` (byte count multiple of 16, both 16-byte aligned)
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// whole warp
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// K-major, no swizzle: start address, LBO (K direction), SBO (M/N direction), version 1
__device__ __forceinline__ uint64_t smem_desc(const void* p, uint32_t lbo, uint32_t sbo) {
  const uint64_t a = (smem_u32(p) & 0x3FFFFu) >> 4;
  return a | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// the same descriptor split into its constant part and the address field
__device__ __forceinline__ uint64_t smem_desc_bits(uint32_t lbo, uint32_t sbo) {
  return ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
__device__ __forceinline__ uint64_t smem_desc_at(uint64_t bits, uint32_t smem_addr) {
  return bits | (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
}

// kind::tf32, D = F32, A = B = TF32, both K-major
__host__ __device__ constexpr uint32_t idesc_tf32(uint32_t m, uint32_t n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// kind::f16 with BF16 A and B, D = F32, both K-major (K = 16 per instruction)
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t m, uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// One lane of a converged warp (the same one at every call).  A whole warp that runs the issue
// loop with only this lane's instructions taking effect keeps descriptors and loop state in
// uniform registers: products then issue at the tensor core's own rate (M = 128: 32 + N / 4
// clocks, the operands' shared-memory reads), where a single lane's loop, moving every
// descriptor to uniform registers first, took 45 to 180 clocks each.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r));
  return r;
}
// kind::f16 product issued by the elected lane of the warp
__device__ __forceinline__ void mma_f16_warp(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}

// the same for kind::tf32
__device__ __forceinline__ void mma_tf32_warp(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}

// arrives on `bar` when every tcgen05.mma issued so far by this thread has completed
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 32 columns of 32-bit: thread t of the warp gets lane (base lane + t), 32 consecutive columns
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 lanes x 16 columns of 32-bit: thread t of the warp gets lane (base lane + t), 16 consecutive columns
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// three 32 x 16 loads at column offsets 0, step, 2 step from taddr (the regions R0, R1, R2 of
// one accumulator layout), one wait for all of them
__device__ __forceinline__ void tmem_ld16x3(uint32_t taddr, uint32_t step, float* v0, float* v1, float* v2) {
  uint32_t r[48];
#pragma unroll
  for (int k = 0; k < 3; ++k)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[16 * k + 0]), "=r"(r[16 * k + 1]), "=r"(r[16 * k + 2]), "=r"(r[16 * k + 3]), "=r"(r[16 * k + 4]),
          "=r"(r[16 * k + 5]), "=r"(r[16 * k + 6]), "=r"(r[16 * k + 7]), "=r"(r[16 * k + 8]), "=r"(r[16 * k + 9]),
          "=r"(r[16 * k + 10]), "=r"(r[16 * k + 11]), "=r"(r[16 * k + 12]), "=r"(r[16 * k + 13]),
          "=r"(r[16 * k + 14]), "=r"(r[16 * k + 15])
        : "r"(taddr + (uint32_t)k * step)
        : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v0[i] = __uint_as_float(r[i]);
    v1[i] = __uint_as_float(r[16 + i]);
    v2[i] = __uint_as_float(r[32 + i]);
  }
}

// the same with 8 columns per region
__device__ __forceinline__ void tmem_ld8x3(uint32_t taddr, uint32_t step, float* v0, float* v1, float* v2) {
  uint32_t r[24];
#pragma unroll
  for (int k = 0; k < 3; ++k)
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[8 * k + 0]), "=r"(r[8 * k + 1]), "=r"(r[8 * k + 2]), "=r"(r[8 * k + 3]), "=r"(r[8 * k + 4]),
          "=r"(r[8 * k + 5]), "=r"(r[8 * k + 6]), "=r"(r[8 * k + 7])
        : "r"(taddr + (uint32_t)k * step)
        : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v0[i] = __uint_as_float(r[i]);
    v1[i] = __uint_as_float(r[8 + i]);
    v2[i] = __uint_as_float(r[16 + i]);
  }
}

__device__ __forceinline__ float round_tf32(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}

// fp32 -> hi + lo with both parts exact in tf32 (each rounded to nearest).  The
// tensor core reads only the top 19 bits of an fp32 operand; an unrounded
// remainder would be truncated there, which biases every product toward zero.
__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
  hi = round_tf32(x);
  lo = round_tf32(x - hi);
}

// fp32 -> hi + lo, both BF16 rounded to nearest (16 significant bits together), as raw bits
__device__ __forceinline__ void split_bf16(float x, uint16_t& hi, uint16_t& lo) {
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
  hi = __bfloat16_as_ushort(h);
  lo = __bfloat16_as_ushort(l);
}

// bring [p, p + bytes) into L2 without waiting (p 16-byte aligned, bytes a multiple of 16)
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// the same through the load/store path, one 128-byte line per instruction: the bulk form
// takes a slot of the SM's bulk-copy unit per row, which the A-chunk copies also use
__device__ __forceinline__ void prefetch_lines_l2(const void* p, uint32_t bytes) {
  const char* c = static_cast<const char*>(p);
  for (uint32_t o = 0; o < bytes; o += 128u) asm volatile("prefetch.global.L2 [%0];" ::"l"(c + o));
}

}  // namespace tc
}  // namespace so
