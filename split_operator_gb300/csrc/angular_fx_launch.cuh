// Launchers of the fixed-point lane-matrix kernels, one instantiation per translation unit.
#pragma once
#include <cstring>

#include "angular_fx.cuh"

namespace so {

// angular_fx_ff.cu, angular_fx_exps.cu, angular_fx_ff_exps.cu
using FxAngularLaunch = cudaError_t(int halves, int kp, int cols, const void* one, const FxTcParams* params,
                                    const uint2* owners, int64_t tiles, unsigned grid, cudaStream_t s);
FxAngularLaunch launch_fx_angular_ff, launch_fx_angular_exps, launch_fx_angular_ff_exps;

namespace {

template <int NB, int MH, bool FF, bool EXPS>
cudaError_t fx_angular_one(int kp, const void* one, const FxTcParams* params, const uint2* owners, int64_t tiles,
                           unsigned grid, cudaStream_t s) {
  static bool done = false;
  auto kern = fx_angular_kernel<NB, MH, FF, EXPS>;
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 180 * 1024);
    if (e != cudaSuccess) return e;
    done = true;
  }
  const uint32_t smem = fx_tc_smem(NB * (MH == 1 ? 4 : 2), kp);
  if (smem > 180 * 1024) return cudaErrorInvalidValue;
  FxTcParams p{};
  if (one) std::memcpy(&p, one, sizeof(p));
  count_launch();
  return launch_overlapped(kern, grid, kFxThreads, smem, s, p, params, owners, tiles);
}

template <bool FF, bool EXPS>
cudaError_t fx_angular_launch(int halves, int kp, int cols, const void* one, const FxTcParams* params,
                              const uint2* owners, int64_t tiles, unsigned grid, cudaStream_t s) {
  if (halves == 1 && cols == 32) return fx_angular_one<8, 1, FF, EXPS>(kp, one, params, owners, tiles, grid, s);
  if (halves == 1 && cols == 16) return fx_angular_one<4, 1, FF, EXPS>(kp, one, params, owners, tiles, grid, s);
  if (halves == 1 && cols == 8) return fx_angular_one<2, 1, FF, EXPS>(kp, one, params, owners, tiles, grid, s);
  if (halves == 2 && cols == 16) return fx_angular_one<8, 2, FF, EXPS>(kp, one, params, owners, tiles, grid, s);
  if (halves == 2 && cols == 8) return fx_angular_one<4, 2, FF, EXPS>(kp, one, params, owners, tiles, grid, s);
  return cudaErrorInvalidValue;
}

}  // namespace
}  // namespace so
