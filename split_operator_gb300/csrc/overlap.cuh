// Launches that begin while the kernel ahead of them in the stream drains (programmatic stream
// serialization).  A kernel launched with launch_overlapped does its set-up (barriers, tensor
// memory), then wait_for_previous(), and only after that reads or writes global memory: the wait
// returns when the kernels before it have completed and their writes are visible.  It then lets
// the next launch begin; so at most two kernels of a stream are on the GPU at a time.  Every thread
// of every block passes through the wait, or the kernel behind could overtake the one ahead.
//
// A step of the 2-D plane is two launches of 10 to 80 us; starting a launch, setting it up and
// draining the one ahead took 3 to 5 us of each.  us per step without / with: FP32 BF16x6 plane of
// 4096 x 128 46.8 / 39.2 (with the earlier hand-over of the norms, pass_end.cuh), 512 x 32 40.0 / 37.2.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <utility>

namespace so {

constexpr size_t kHalfSmem = 115 * 1024;  // more than half of an SM's shared memory

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// SMs of the current device at the first call (1 if it cannot be asked)
inline int sm_count() {
  static const int sms = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      n = 1;
    return n;
  }();
  return sms;
}

// Dynamic shared memory of an overlapped launch: where its blocks do not outnumber the SMs, enough
// that an SM holds only one.  Blocks that begin while the kernel ahead still runs would otherwise
// crowd on the SMs that it left idle (measured: 41.5 us a step instead of 39.2, and 71.7 instead of
// 61.0 for 45 x 1000 points in FP64).
inline size_t one_block_per_sm(int64_t blocks, size_t smem) {
  return blocks <= sm_count() && smem < kHalfSmem ? kHalfSmem : smem;
}

template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, std::forward<A>(args)...);
}

}  // namespace so
